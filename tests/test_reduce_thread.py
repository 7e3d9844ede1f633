"""One thread's share of a reduction (reduce_thread of reduce.cuh) on the host,
compiled with bounds checks: every element is taken once by one lane of one
warp, and no accumulator outside its array is touched. The kernel runs the same
function (CPU only)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "reduce.cuh"
using namespace psb;

// Sum, maximum and minimum of distinct whole numbers in padded rows and planes.
template <typename T>
static int check(int rx, int ry, int rz, int nwarps) {
  const int64_t sy = rx + 3, sz = sy * (ry + 1);
  std::vector<T> v(sz * rz, (T)-1000000);  // the padding
  int64_t n = 0;
  for (int z = 0; z < rz; z++)
    for (int y = 0; y < ry; y++)
      for (int x = 0; x < rx; x++) v[x + y * sy + z * sz] = (T)(++n);
  RAcc sum = racc_init(PS_SUM), hi = racc_init(PS_MAX), lo = racc_init(PS_MIN);
  for (int w = 0; w < nwarps; w++)
    for (int lane = 0; lane < 32; lane++) {
      sum = racc_merge(PS_SUM, sum, reduce_thread<T, PS_SUM>(v.data(), sy, sz, rx, ry, rz, w, nwarps, lane));
      hi = racc_merge(PS_MAX, hi, reduce_thread<T, PS_MAX>(v.data(), sy, sz, rx, ry, rz, w, nwarps, lane));
      lo = racc_merge(PS_MIN, lo, reduce_thread<T, PS_MIN>(v.data(), sy, sz, rx, ry, rz, w, nwarps, lane));
    }
  const bool ok = sum.s + sum.c == (double)n * (n + 1) / 2 && hi.s == n && lo.s == 1;
  if (!ok) printf("%zu bytes, %d x %d x %d, %d warps: %g %g %g\n", sizeof(T), rx, ry, rz, nwarps,
                  sum.s + sum.c, hi.s, lo.s);
  return ok ? 0 : 1;
}

int main() {
  int bad = 0;
  const int shapes[][3] = {{1, 1, 1}, {31, 3, 2}, {256, 2, 3}, {257, 5, 1}, {600, 1, 4}};
  for (auto &s : shapes)
    for (int nwarps : {1, 8, 24}) {
      bad += check<float>(s[0], s[1], s[2], nwarps);
      bad += check<int32_t>(s[0], s[1], s[2], nwarps);
      bad += check<double>(s[0], s[1], s[2], nwarps);
      bad += check<int64_t>(s[0], s[1], s[2], nwarps);
    }
  return bad;
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="no nvcc")
def test_each_element_once_and_nothing_out_of_bounds(tmp_path):
    src, exe = tmp_path / "reduce.cu", tmp_path / "reduce"
    src.write_text(PROGRAM)
    r = subprocess.run(
        [NVCC, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "physis_b200", "csrc"),
         "-I" + os.path.join(ROOT, "include"), "-Xcompiler",
         "-fsanitize=bounds,-fno-sanitize-recover=all", str(src), "-o", str(exe),
         "-Xlinker", "-lubsan"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
