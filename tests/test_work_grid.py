"""The runtime's work grid (Himeno runs keep one between runs) on a stand-in for
the CUDA runtime with little memory: any device allocation of the library that
fails gets the work grid's memory and succeeds, a run that is queueing its
launches keeps it, the last grid takes it along, and it is not taken where
little is left (CPU only: the library's objects linked to the stand-in)."""
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "physis_b200", "csrc")
OBJ = os.path.join(ROOT, "physis_b200", "lib", "obj")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

STUB = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <cuda_runtime_api.h>
#include "internal.h"

static size_t g_limit = (size_t)1 << 30, g_used = 0;
static std::map<void *, size_t> g_blocks;

static cudaError_t take(void **p, size_t n) {
  if (g_used + n > g_limit) return cudaErrorMemoryAllocation;
  *p = calloc(1, n + 256);
  g_blocks[*p] = n;
  g_used += n;
  return cudaSuccess;
}
static cudaError_t give(void *p) {
  auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return cudaSuccess;
  g_used -= it->second;
  free(p);
  g_blocks.erase(it);
  return cudaSuccess;
}

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
  return take(p, n);
}
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = g_limit - g_used;
  *t = g_limit;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
#undef cudaGetDeviceProperties
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
  memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  p->sharedMemPerBlockOptin = 227 << 10;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "?"; }
}

static int failures = 0;
#define EXPECT(x) \
  do { \
    if (!(x)) { \
      printf("line %d: %s\n", __LINE__, #x); \
      failures++; \
    } \
  } while (0)

int main() {
  using namespace psb;
  const PSIndex dims[3] = {64, 48, 32};
  __PSGrid *g = nullptr;
  EXPECT(psb_grid_new(PS_FLOAT, 3, dims, PSB_LAYOUT_PITCHED, &g) == PSB_OK);
  GridImpl *gi = as_impl(g);
  const size_t bytes = gi->alloc_bytes, before = g_used;
  GridImpl *first = nullptr;
  auto acquire = [&] {
    g_limit = (size_t)1 << 30;
    const WorkGrid w(gi);
    EXPECT(w.grid && w.grid != gi && w.grid->alloc_bytes == bytes);
    EXPECT(g_used == before + bytes);
    first = w.grid;
    g_limit = g_used;  // full
  };

  acquire();
  {
    const WorkGrid again(gi);
    EXPECT(again.grid == first && g_used == before + bytes);  // kept between runs
    void *p = nullptr;
    EXPECT(device_malloc(&p, 64) == cudaErrorMemoryAllocation);  // not while it is used
    EXPECT(g_used == before + bytes);
  }
  psb_generic_stencil d;
  memset(&d, 0, sizeof(d));
  d.ndims = 1;
  d.ngrids = 1;
  d.nterms = 1;
  d.accum_type = PS_FLOAT;
  d.grid_type[0] = PS_FLOAT;
  d.grid_axes[0][1] = d.grid_axes[0][2] = -1;
  int id = 0;
  EXPECT(psb_generic_register(&d, &id) == PSB_OK);  // a table of the library's own
  EXPECT(g_used > before && g_used < before + bytes);
  const size_t table = g_used - before;

  g_limit = (size_t)1 << 30;
  {
    const WorkGrid w(gi);
    EXPECT(w.grid);
  }
  g_limit = g_used;
  const int id3[3] = {32, 32, 32};
  GridImpl *pooled = nullptr;
  EXPECT(grid_alloc_pool(PS_FLOAT, id3, (cudaMemPool_t)1, nullptr, &pooled) == PSB_OK);
  EXPECT(pooled && g_used < before + table + bytes);
  grid_free_pool(pooled, nullptr);
  EXPECT(g_used == before + table);

  // Another grid of the user's.
  g_limit = (size_t)1 << 30;
  {
    const WorkGrid w(gi);
    EXPECT(w.grid);
  }
  g_limit = g_used;
  __PSGrid *h = nullptr;
  EXPECT(psb_grid_new(PS_FLOAT, 3, dims, PSB_LAYOUT_PITCHED, &h) == PSB_OK);
  EXPECT(g_used == before + table + bytes);

  // Less than eight times its size is left: not taken.
  g_limit = g_used + 8 * bytes - 1;
  {
    const WorkGrid w(gi);
    EXPECT(!w.grid);
  }
  // The last grid takes it along.
  g_limit = (size_t)1 << 30;
  {
    const WorkGrid w(gi);
    EXPECT(w.grid);
  }
  PSGridFree(h);
  EXPECT(g_used == before + table + bytes);
  PSGridFree(g);
  EXPECT(g_used == before + table - bytes);
  printf("%d failures\n", failures);
  fflush(stdout);
  _Exit(failures ? 1 : 0);
}
"""


def test_failed_allocations_get_the_work_grid_back(tmp_path):
    objs = sorted(glob.glob(os.path.join(OBJ, "*.o")))
    if not objs:
        pytest.skip("the library's objects are not here")
    und = subprocess.run(["nm", "-u"] + objs, capture_output=True, text=True, check=True).stdout
    names = sorted(set(re.findall(r" U ((?:__)?cuda\w+)", und)))
    own = set(re.findall(r"\b(cuda\w+)\(", STUB))
    others = "\n".join("long %s() { return 0; }" % n for n in names if n not in own)
    # The default answers go into a C file of their own, without the header's types.
    stub, rest, exe = tmp_path / "stub.cpp", tmp_path / "rest.c", tmp_path / "stub"
    stub.write_text(STUB)
    rest.write_text(others + "\n")
    cuda = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    for cmd in (["gcc", "-w", "-c", str(rest), "-o", str(tmp_path / "rest.o")],
                ["g++", "-std=c++17", "-I" + cuda, "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                 str(stub), str(tmp_path / "rest.o")] + objs +
                ["-o", str(exe), "-ldl", "-lpthread"]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60,
                       env={k: v for k, v in os.environ.items() if not k.startswith("PHYSIS_")})
    assert r.returncode == 0, r.stdout + r.stderr
