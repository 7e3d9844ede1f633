"""The x column of a thread of the thread-per-point kernel (gen_point) on the host:
the threads of the last block past the domain must get its end, also where lo plus
their index lies beyond the largest int (CPU only)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PROGRAM = r"""
#include <climits>
#include <cstdio>
#include "internal.h"
#include "k_generic.cuh"

int main() {
  int bad = 0;
  const int doms[][2] = {{0, 1}, {0, 256}, {3, 300}, {0, INT_MAX}, {1, INT_MAX},
                         {INT_MAX - 5, INT_MAX}};
  for (auto &d : doms) {
    const long long lo = d[0], hi = d[1], ext = hi - lo, end = (ext + 255) / 256 * 256;
    for (long long i = end > 1024 ? end - 1024 : 0; i < end; i++) {
      const long long want = lo + i < hi ? lo + i : hi;
      const int got = psb::gen_point(d[0], d[1], (unsigned)i);
      if (got != want && bad++ < 5) printf("[%lld, %lld) %lld: %d\n", lo, hi, i, got);
    }
  }
  return bad != 0;
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="no nvcc")
def test_threads_past_the_domain_get_its_end(tmp_path):
    src, exe = tmp_path / "columns.cu", tmp_path / "columns"
    src.write_text(PROGRAM)
    r = subprocess.run(
        [NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "physis_b200", "csrc"),
         "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe)],
        capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
