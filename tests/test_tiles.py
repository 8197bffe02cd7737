"""The tile a solver starts with (csrc/fr_tiles.hpp, host code): the first of
its list on a mesh that gives the GPU two blocks per SM, one with the fewest
elements per block on a smaller mesh, so that a small mesh has as many blocks as
it can."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hifiles-solver_b200", "csrc")
SHAPES = [(2, P) for P in range(1, 6)] + [(3, P) for P in range(1, 5)]
SMALL, LARGE = (1, 8, 216, 295), (296 * 16, 32 ** 3)

PROGRAM = """
#include <cstdio>
#include <initializer_list>
#include "fr_tiles.hpp"
template <int N> void show(const char* kind, int d, int p, const frb::Tile (&t)[N])
{
  int least = t[0].epb;
  for (const frb::Tile& q : t) least = q.epb < least ? q.epb : least;
  for (long long e : {%s}) {
    const int i = frb::default_tile(t, e);
    std::printf("%%s %%d %%d %%lld %%d %%d %%d\\n", kind, d, p, e, i, t[i].epb, least);
  }
}
int main()
{
%s
  for (int les : {0, 1})
    for (long long e : {8LL, 1200LL, 30000LL}) {
      const frb::Tile t = frb::Tiles<3, 2>::grad[frb::default_grad_tile<3, 2>(e, les)];
      std::printf("p2 %%d %%lld %%d %%d\\n", les, e, t.epb, t.nt);
      if (frb::default_grad_tile<3, 3>(e, les) != frb::default_tile(frb::Tiles<3, 3>::grad, e)) return 1;
    }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_default_tiles(tmp_path):
    calls = "\n".join('show("%s", %d, %d, frb::Tiles<%d, %d>::%s);' % (k, d, p, d, p, k)
                      for d, p in SHAPES for k in ("grad", "upd"))
    src = tmp_path / "tiles.cpp"
    src.write_text(PROGRAM % (", ".join("%dLL" % e for e in SMALL + LARGE), calls))
    exe = str(tmp_path / "tiles")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    rows = [r.split() for r in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    hexes_p2 = [tuple(int(v) for v in r[1:]) for r in rows if r[0] == "p2"]
    assert hexes_p2 == [(0, 8, 1, 64), (0, 1200, 2, 128), (0, 30000, 2, 128),
                        (1, 8, 1, 64), (1, 1200, 4, 224), (1, 30000, 4, 224)]
    rows = [r for r in rows if r[0] != "p2"]
    assert len(rows) == len(SHAPES) * 2 * len(SMALL + LARGE)
    for kind, d, p, e, i, epb, least in rows:
        if int(e) in SMALL:
            assert epb == least, (kind, d, p, e, i, epb, least)
        if int(e) in LARGE:
            assert int(i) == 0, (kind, d, p, e, i)
