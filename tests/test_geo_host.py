"""The grid columns of geo.cuh on the host: every slot's column against the colour
order itself, and whether two blocks of a colour phase can meet in 32 bytes of a
vector (rows of two colours, or rows and the zero sink), which is what the kernels
leave out a fence by. The header is compiled as plain C++."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "geo.cuh"
using namespace hb;
int main(int argc, char** argv) {
  const int n[3] = {std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3])};
  ColourGrid g;
  g.init(n[0], n[1], n[2], kSweepDefault);
  const GeoGrid G = geo_grid(g);
  const int rows = n[0] * n[1] * n[2];
  long wrong = 0;
  std::vector<int> owner(rows + 1, kColours);  // of each entry: its sweep position, or the sink
  for (int s = 0; s < kColours; ++s)
    for (int q = g.start[s]; q < g.start[s + 1]; ++q) {
      owner[q] = s;
      const GeoRow r(G.block[s], q);
      int ix, iy, iz;
      g.coords(q, ix, iy, iz);
      for (int k = 0; k < kSlots; ++k) {
        const int x = ix + k % 3 - 1, y = iy + k / 3 % 3 - 1, z = iz + k / 9 - 1;
        const bool in = x >= 0 && x < n[0] && y >= 0 && y < n[1] && z >= 0 && z < n[2];
        wrong += r.col(G.block[s], k, rows) != (in ? g.old2new(x, y, z) : rows);
      }
    }
  int meet = 0;  // FP32: eight entries to 32 bytes
  for (int i = 1; i <= rows; ++i) meet |= i % 8 != 0 && owner[i] != owner[i - 1];
  for (int s = 0; s < kColours; ++s) wrong += (G.block[s].shared != 0) != (meet != 0);
  std::printf("%ld %d\n", wrong, meet);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("geo")
    src, exe = d / "geo.cpp", d / "geo"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "hpcg_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-I", include, str(src), "-o", str(exe)], check=True)
    return str(exe)


# whole sectors throughout; the sink beside the last rows (16k + 1); colours that
# meet; a last level of a batch member; flat, thin, single
@pytest.mark.parametrize("dims,meet", [((32, 16, 48), 0), ((33, 33, 33), 1), ((17, 33, 65), 1), ((6, 6, 6), 1),
                                       ((82, 82, 2), 1), ((74, 74, 2), 1), ((33, 31, 29), 1), ((4, 4, 4), 0),
                                       ((75, 6, 13), 1), ((17, 1, 9), 1), ((2, 3, 1), 1), ((1, 1, 1), 1)])
def test_grid_columns_and_shared_sectors(program, dims, meet):
    out = subprocess.run([program, *map(str, dims)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", str(meet)]
