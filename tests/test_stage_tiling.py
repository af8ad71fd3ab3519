"""The host rules of the stage kernels' tiling, compiled from the header that the
library uses: the buffer of per-block CFL maxima holds every launch's blocks, and
a launch's grid holds every plane."""
import subprocess

import pytest

from lsmlib_b200 import build

PROGRAM = r"""
#include <cstdio>
#include "stage_launch.h"
using namespace lsmgpu;

static FillBox box(int nx, int ny, int nz, int ghost) {
  FillBox f;
  const int n[3] = {nx, ny, nz};
  for (int d = 0; d < 3; d++) {
    f.lo[d] = -ghost;
    f.hi[d] = n[d] - 1 + ghost;
  }
  return f;
}

int main() {
  const int wide[] = {1,    8,    31,   33,   64,   129,  257,  512,  1023, 1448, 1536,
                      2000, 2056, 2305, 2560, 3000, 4096, 8192, 20000};
  long bad = 0;
  for (int nx : wide)
    for (int ny : wide)
      for (int nz = 1; nz <= 400; nz++) {
        const FillBox f = box(nx, ny, nz, 0);
        const int room = stage_blocks_max(box(nx, ny, nz, 3), kHostSlabs);
        int zlo[kHostSlabs + 1];
        const int ns = stage_slabs(f, zlo);
        long sum = 0;
        bool cover = ns >= 1 && ns <= kHostSlabs && zlo[0] == 0 && zlo[ns] == nz;
        for (int q = 0; q < ns; q++) {
          FillBox s = f;
          s.lo[2] = zlo[q];
          s.hi[2] = zlo[q + 1] - 1;
          cover = cover && s.n(2) >= 1;
          sum += stage_blocks(s);
        }
        if (!cover || sum > room || stage_blocks(f) > room) {
          if (bad++ < 5)
            std::printf("%dx%dx%d: %d slabs, %ld blocks in all, %d whole, room for %d\n", nx, ny,
                        nz, ns, sum, stage_blocks(f), room);
        }
      }
  return bad != 0;
}
"""


# grid extents of fill boxes with many planes (1,048,560 is what 16 planes a block
# reach) and what a block marches
TALL = r"""
#include <cstdio>
#include "stage_launch.h"
using namespace lsmgpu;

int main() {
  long bad = 0;
  const int planes[] = {1,      720884,  720885,  720886,  851955,   851956,
                        900001, 1048559, 1048560, 1048561, 16000000, 2000000000};
  for (int nx : {1, 8, 33, 64, 300})
    for (int nz : planes) {
      FillBox f;
      const int n[3] = {nx, 1 + nx % 7, nz};
      for (int d = 0; d < 3; d++) {
        f.lo[d] = 0;
        f.hi[d] = n[d] - 1;
      }
      for (int tz : {stage_tz(f), one_cell_tz(f)}) {
        const long blocks = ((long)nz + tz - 1) / tz;
        if (tz < 1 || blocks > 65535) {
          bad++;
          std::printf("%d planes: %d a block, %ld blocks\n", nz, tz, blocks);
        }
      }
    }
  return bad != 0;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    def go(program):
        d = tmp_path_factory.mktemp("tiling")
        src, exe = str(d / "t.cu"), str(d / "t")
        with open(src, "w") as f:
            f.write(program)
        subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "-O1", "-I", build.CSRC, "-I",
                                                    build.INCLUDE, src, "-o", exe],
                       check=True, capture_output=True)
        return subprocess.run([exe], capture_output=True, text=True)
    return go


def test_tall_boxes_fit_a_grid(run):
    r = run(TALL)
    assert r.returncode == 0, r.stdout


def test_partials_hold_every_slab(run):
    r = run(PROGRAM)
    assert r.returncode == 0, r.stdout
