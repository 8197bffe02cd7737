// fr_tiles.hpp -- tile variants of the element kernels behind fr_solver, and
// the one a mesh starts with.  Host code without CUDA, so that the rule can be
// checked where there is no GPU.
#pragma once

namespace frb {

struct Tile {
  int epb, nt, minb;   // elements per CTA, threads per CTA, CTAs per SM the registers are sized for (0: any)
  int pers = 0;        // gradient kernel only: 1 = persistent blocks that walk over element blocks
};

// Compiled tile variants (elements per CTA, threads per CTA) of the gradient
// and update kernels per (dims, order); the autotuner may pick any.  The first
// entry is the default of large meshes (hexes of P = 2 apart, see
// default_grad_tile), the last of those with the fewest elements per CTA that of
// small ones.  A gradient tile has a thread for each
// of its F EPB NU / (P+1) line tasks, an update tile one for each of its flux
// points, in as few idle lanes as whole warps allow.
template <int DIM, int P> struct Tiles;
#define FR_TILES(D_, P_, G, U) \
  template <> struct Tiles<D_, P_> { static constexpr Tile grad[] = G; static constexpr Tile upd[] = U; };
#define T_(...) {__VA_ARGS__}
FR_TILES(2, 1, T_({16, 128, 5}, {4, 32}), T_({16, 128, 4}, {4, 32}))
FR_TILES(2, 2, T_({10, 128, 5}, {2, 32}), T_({10, 128, 4}, {2, 32}))
FR_TILES(2, 3, T_({8, 128, 5}, {16, 256, 3}, {2, 32}), T_({8, 128, 4}, {16, 256, 2}, {2, 32}))
FR_TILES(2, 4, T_({6, 160, 4}, {3, 96, 6}, {1, 32}), T_({5, 128, 5}, {10, 256, 2}, {1, 32}))
FR_TILES(2, 5, T_({3, 128, 5}, {5, 192, 3}, {1, 64}), T_({3, 128, 5}, {7, 256, 2}, {1, 64}))
FR_TILES(3, 1, T_({8, 192, 4}, {5, 128, 5}, {1, 32}), T_({8, 192, 3}, {5, 128, 4}, {1, 32}))
FR_TILES(3, 2, T_({4, 224, 2}, {2, 128, 5}, {1, 64, 10}), T_({4, 224, 3}, {2, 128, 4}, {1, 64, 8}))
FR_TILES(3, 3, T_({1, 96, 6}, {1, 96, 8}, {1, 96, 5}, {2, 192, 3}, {2, 192, 3, 1}, {1, 96, 7}),
         T_({1, 96, 6}, {1, 96, 8}, {1, 96, 5}, {2, 192, 3}))
FR_TILES(3, 4, T_({1, 160, 3}, {1, 160, 4}, {1, 128, 4}), T_({1, 160, 5}, {1, 160, 4}))
#undef T_
#undef FR_TILES

// The tile of a mesh before any autotuning: the first, or the last of those
// with the fewest elements where the first would leave the GPU with fewer than
// two blocks per SM (148 SMs).
template <int N>
constexpr int default_tile(const Tile (&t)[N], long long E)
{
  if ((E + t[0].epb - 1) / t[0].epb >= 296) return 0;
  int m = 0;
  for (int i = 1; i < N; i++)
    if (t[i].epb <= t[m].epb) m = i;
  return m;
}

// The gradient tile likewise, but for large meshes of hexes of P = 2 without LES
// the second one, 2 elements on 128 threads: a stage of 21840 hexes takes 199 us
// with it against 208 with 4 elements on 224 threads, in FP32 148 against 166.
// The LES kernel spills more at its 96 registers than at the 128 of the first
// (6188 walled hexes, Smagorinsky: 102.8 against 101.2 us).
template <int DIM, int P>
constexpr int default_grad_tile(long long E, bool les)
{
  const int i = default_tile(Tiles<DIM, P>::grad, E);
  return DIM == 3 && P == 2 && i == 0 && !les ? 1 : i;
}

}  // namespace frb
