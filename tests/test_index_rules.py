"""Index arithmetic of the kernels at sizes that no test allocates, compiled
for the host from the kernels' own headers."""

import os
import shutil
import subprocess

import pytest

from wakis_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _host_program(tmp_path, main):
    if shutil.which(build.nvcc()) is None:
        pytest.skip("nvcc not available")
    src = tmp_path / "main.cu"
    src.write_text('#include <cstdio>\n#include "wakis_b200.h"\n#include "abi_internal.h"\n'
                   '#include "fit_common.cuh"\n#include "fit_kernels.cuh"\n' + main)
    exe = tmp_path / "main"
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "--expt-relaxed-constexpr", "--extended-lambda", "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "wakis_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    subprocess.run([str(exe)], check=True)


def test_neighbour_guard_of_the_largest_grids(tmp_path):
    """A neighbour index n + off past the last cell is refused on every grid
    below 2^31 cells, also where the sum passes 2^31."""
    _host_program(tmp_path, """
int main() {
  const int dims[][3] = {{1289, 1289, 1289}, {1290, 1290, 1290}, {5, 5, 85899345}, {20724, 20724, 5},
                         {5, 429496, 1000}, {7, 5, 9}};
  for (auto& s : dims) {
    const long long N = (long long)s[0] * s[1] * s[2], plane = (long long)s[0] * s[1];
    if (N >= (1LL << 31)) return 2;
    const int offs[] = {1, s[0], (int)plane};
    for (int off : offs)
      for (long long back = 0; back < 3 * plane; back += back < 4 ? 1 : plane / 7 + 1) {
        const long long n = N - 1 - back;
        const bool want = n + off < N;
        if (n >= 0 && wk::inside_after((int)n, off, (int)N) != want) return 1;
        const long long e = N - off - 1 + (back & 3);   // the two sides of the line
        if (e >= 0 && e < N && wk::inside_after((int)e, off, (int)N) != (e + off < N)) return 1;
      }
  }
  return 0;
}
""")


def test_barrier_count_of_a_call_with_very_many_steps(tmp_path):
    """The arrivals of a grid barrier against their target where both pass 2^32."""
    _host_program(tmp_path, """
#include "fit_loop.cuh"
int main() {
  for (unsigned blocks : {1u, 7u, 148u, 160u})
    for (long long step : {1LL, 2LL, 29020049LL, 29020050LL, 29020051LL, 2147483647LL}) {
      const long long target = step * blocks;
      for (long long behind = -(long long)blocks; behind <= (long long)blocks; behind++) {
        const long long count = target - behind;
        if (wk::loop_arrived((unsigned)count, (unsigned)target) != (count >= target)) return 1;
      }
    }
  return 0;
}
""")
