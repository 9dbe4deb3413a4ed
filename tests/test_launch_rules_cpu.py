"""The launches of the float64 kernels, by the library's own host code against a
stand-in for the CUDA runtime (no GPU): a launch that asks for more dynamic shared
memory than its kernel may use on the current device, or for a grid beyond the
hardware's, is refused as the runtime refuses it."""
import os
import shutil
import subprocess

import pytest

from bilby_gb300 import _build
from tests.conftest import ROOT

RUNTIME = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <utility>
#include "gwl_internal.h"
static int device = 0;
static cudaError_t last = cudaSuccess;
static std::map<std::pair<int, const void*>, int> limit;  // by device and kernel
static struct { dim3 grid, block; } config;
static cudaError_t launched(const void* k, dim3 g, size_t smem) {
  const auto it = limit.find({device, k});
  const size_t most = it == limit.end() ? 48 * 1024 : it->second;
  if (smem > most || g.x > 2147483647u || g.y > 65535u || g.z > 65535u || !g.x || !g.y) last = cudaErrorInvalidValue;
  return last;
}
extern "C" {
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int bytes) {
  limit[{device, f}] = bytes;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launched(f, c->gridDim, c->dynamicSmemBytes);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void*);
static size_t config_smem;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void*) {
  config.grid = g;
  config.block = b;
  config_smem = smem;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = config.grid;
  *b = config.block;
  *smem = config_smem;
  *static_cast<void**>(s) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void**, size_t smem, cudaStream_t) {
  return launched((const void*)k, g, smem);
}
cudaError_t cudaLaunchKernel(const void* k, dim3 g, dim3, void**, size_t smem, cudaStream_t) { return launched(k, g, smem); }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
int main(int argc, char** argv) {
  // detectors, complex sums, chunks, points, device: one launch of each kind per five
  for (int q = 1; q + 4 < argc; q += 5) {
    gwl::LaunchArgs a = {};
    a.n_det = std::atoi(argv[q]);
    a.cplx = std::atoi(argv[q + 1]);
    a.n_chunks = a.wide_chunks = std::atoll(argv[q + 2]);
    a.B = std::atoll(argv[q + 3]);
    device = std::atoi(argv[q + 4]);
    std::printf("%d %d\n", (int)gwl::launch_wide(a, nullptr), (int)gwl::launch_wide_sg(a, nullptr));
  }
}
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    gxx = shutil.which("g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    if gxx is None or not os.path.isdir(cuda):
        pytest.skip("no host compiler or CUDA headers")
    objects = [os.path.join(_build.OBJ_DIR, f) for f in ("gwl_wide.o", "gwl_wide_sg.o")]
    _build.build(force=not all(os.path.exists(f) for f in objects))
    tmp = tmp_path_factory.mktemp("runtime")
    (tmp / "probe.cpp").write_text(RUNTIME)
    exe = tmp / "probe"
    subprocess.run([gxx, "-std=c++17", "-w", "-I", os.path.join(ROOT, "bilby_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", cuda, str(tmp / "probe.cpp"), *objects, "-o", str(exe)], check=True)

    def run(*launches):
        args = [str(x) for q in launches for x in q]
        res = subprocess.run([str(exe), *args], capture_output=True, text=True, check=True)
        return [int(x) for x in res.stdout.split()]
    return run


@pytest.mark.parametrize("cplx", [0, 1])
@pytest.mark.parametrize("detectors", [1, 2, 3, 4])
def test_batches_on_a_second_device(runtime, detectors, cplx):
    one = (detectors, cplx, 17, 600)
    assert runtime(one + (0,), one + (0,), one + (1,), one + (2,)) == [0] * 8


# 65,535 CTAs of eight tiles of 32 points, one point more, and many more
@pytest.mark.parametrize("points", [65535 * 256, 65535 * 256 + 1, 20_000_000, 400_000_000])
@pytest.mark.parametrize("chunks", [1, 17])
def test_batches_beyond_the_grid_of_eight_tiles(runtime, points, chunks):
    assert runtime((2, 0, chunks, points, 0), (1, 1, chunks, points, 0)) == [0] * 4
