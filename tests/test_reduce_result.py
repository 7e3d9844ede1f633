"""PSReduce's result pointer when its set-up fails once: k_reduce.cu linked to a
stand-in for the CUDA runtime whose cudaHostGetDevicePointer fails on its first
call. That call reports the error; the next one must not launch the kernel with
a null result (CPU only, no GPU and no CUDA runtime)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "physis_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

STUB = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cuda_runtime_api.h>
#include "internal.h"

namespace psb {
psb_status set_status(psb_status s) { return s; }
psb_status cuda_status(cudaError_t, const char *) { return PSB_ERR_CUDA; }
cudaError_t device_malloc(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
}  // namespace psb

namespace psb {
struct Scratch {  // ReduceScratch
  void *partials;
  unsigned *ticket;
  double *result;
};
}  // namespace psb

static int g_failures = 1, g_launches = 0, g_null = 0;

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorUnknown; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **p, void *h, unsigned) {
  if (g_failures > 0) {
    g_failures--;
    return cudaErrorUnknown;
  }
  *p = h;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **args, size_t, cudaStream_t) {
  double *result = ((psb::Scratch *)args[2])->result;
  g_launches++;
  if (result) *result = 42.0;
  else g_null++;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *,
                            void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 0; }
}

int main() {
  psb::GridView v;
  memset(&v, 0, sizeof(v));
  float x = 0;
  v.origin = &x;
  psb::Dom3 d;
  for (int i = 0; i < 3; i++) d.lo[i] = 0, d.hi[i] = 1;
  double r = 0;
  const int first = psb::reduce_view(v, PS_FLOAT, PS_SUM, d, &r, nullptr);
  const int after = g_launches;
  const int second = psb::reduce_view(v, PS_FLOAT, PS_SUM, d, &r, nullptr);
  printf("%d %d %d %d %d %g\n", first != PSB_OK, after, second, g_launches, g_null, r);
  return 0;
}
"""


@pytest.mark.skipif(not shutil.which(NVCC), reason="no nvcc")
def test_failed_setup_is_repeated(tmp_path):
    src, obj, exe = tmp_path / "stub.cpp", tmp_path / "k_reduce.o", tmp_path / "stub"
    src.write_text(STUB)
    inc = ["-I" + CSRC, "-I" + os.path.join(ROOT, "include")]
    cuda = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    for cmd in ([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-gencode",
                 "arch=compute_100a,code=sm_100a"] + inc +
                ["-c", os.path.join(CSRC, "k_reduce.cu"), "-o", str(obj)],
                ["g++", "-std=c++17", "-I" + cuda] + inc + [str(src), str(obj), "-o", str(exe),
                                                            "-lpthread"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    # The failure is reported without a launch; then one launch with a result.
    assert out == ["1", "0", "0", "1", "0", "42"], out
