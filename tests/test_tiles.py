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
    assert len(rows) == len(SHAPES) * 2 * len(SMALL + LARGE)
    for kind, d, p, e, i, epb, least in rows:
        if int(e) in SMALL:
            assert epb == least, (kind, d, p, e, i, epb, least)
        if int(e) in LARGE:
            assert int(i) == 0, (kind, d, p, e, i)
