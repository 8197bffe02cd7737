// fr_batch_merged.cuh -- one launch per stage kernel for a whole batch.
//
// A batch holds one merged mesh per (order, scheme) group.  Run group by
// group, a viscous RK stage launches the gradient kernel, the interface-flux
// kernel (orders 2 and 4) and the update kernel of every group: 2-3 launches
// per group and stage.  The merged launches
// below run each of those kernels once for all groups of hexahedra of orders
// 2, 3 and 4: the grid is the concatenation of the groups' element blocks,
// and each block runs the body of its group's order on that group's buffers
// (one body per block, chosen by the block index, so every barrier of a body
// is reached by the whole block).  All groups use blocks of 192 threads with
// as many elements as give each flux point a thread; order 3 takes the fused
// interface/update body, orders 2 and 4 the interface-flux and update bodies.
// No norms are formed (the batch reports none).
#pragma once

#include "fr_b200.h"
#include "fr_update.cuh"

namespace frb {

// Threads per block and elements per block: 162, 192 and 150 of 192 threads
// have a flux point.  The cap for four CTAs per SM spills (FP64 gradient kernel,
// 80 registers: 1.6 kB of stores), yet is the fastest: a step of 12 boxes of
// 6^3 to 14^3, us, caps for 4 / 3 / 1 CTAs: 1545 / 1649 / 1771, FP32 1041 / 1128 /
// 1357; of 6 boxes of 4^3 to 6^3 130 / 139 / 145.  Blocks of 128 threads (2, 1 and
// 1 elements) spill a fifth of that and take 1570 / 1703 / 1688, FP32 1057 / 1142 /
// 1143; 133 / 158 / 157.  Per-group launches: 1370, 1030; 203.
constexpr int kMergedNT = 192;
template <int P> struct MergedTile { static constexpr int epb = P == 2 ? 3 : P == 3 ? 2 : 1; };

template <typename TC>
struct MergedGrad {
  const double* U; const TC* UF; const int* mate; const unsigned char* side; const TC* JG; const TC* detj;
  const TC* nL; TC* VF; TC* ND; TC* DV; TC* BV;
  long long E, nblk;
  Line<TC> L;
  PhysT<TC> ph;
};

template <typename TC>
struct MergedFace {
  const int2* face; const unsigned char* fsign; long long nint; const TC* UF; const TC* VF; const TC* nL;
  const TC* tdA; TC* CF; long long NFE, nbdy; const int* bf; const unsigned char* bt; const TC* BV;
  long long nblk;
  PhysT<TC> ph;
};

template <typename TC>
struct MergedUpd {
  double* U; double* REG; TC* UFn; const TC* UF; const TC* CF; const int* mate; const unsigned char* side;
  const TC* VF; const TC* ND; const TC* DV; const TC* JG; const TC* nL; const TC* tdA;
  const double* idetj; const TC* BV; double* DIV;
  long long E, nblk;
  Line<TC> L;
  PhysT<TC> ph;
  double rk_a, rk_b, dt;
  int first_stage;
};

// Slot k of each launch holds the group of order k + 2 (nblk 0: no such group).
template <typename TC> struct MergedGrads { MergedGrad<TC> s[3]; };
template <typename TC> struct MergedFaces { MergedFace<TC> s[3]; };
template <typename TC> struct MergedUpds { MergedUpd<TC> s[3]; };

// Host: launch the three merged kernels of one stage (faces only when some
// group needs the separate interface kernel).  minb: CTAs per SM the
// registers are capped for (0: no cap).
fr_status merged_stage_launch(bool fp32, const void* grads, const void* faces, bool any_face, const void* upds,
                              int minb, cudaStream_t s);

}  // namespace frb
