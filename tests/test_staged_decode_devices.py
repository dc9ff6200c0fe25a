"""The staged decode sweep asks for its shared memory on every device it runs on
(CPU only: its host code against a stand-in for the CUDA runtime, which refuses a
launch with more than 48 KB that the current device was not asked for)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "grass_b200", "csrc")

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")

# The runtime: compiled by itself, since the CUDA headers define some of it for device code.
RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <map>
#include <utility>
int device, refuse, launched, refused;
static std::map<std::pair<int, const void *>, int> opted;
static dim3 grid, block;
static size_t shared;
static cudaStream_t stream;
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v) {
  if (refuse) return cudaErrorInvalidValue;
  opted[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) {
  const bool ok = smem <= 48 * 1024 || (size_t)opted[{device, f}] >= smem;
  ok ? launched++ : refused++;
  return ok ? cudaSuccess : cudaErrorInvalidValue;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
  grid = g, block = b, shared = s, stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
  *g = grid, *b = block, *s = shared, *(cudaStream_t *)st = stream;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
cudaError_t cudaMalloc(void **, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
}
"""

MAIN = r"""
#include "graph.h"
extern int device, refuse, launched, refused;
namespace grass {
std::atomic<uint64_t> g_launches{0};
int sm_count(int) { return 148; }
int cuda_fail(cudaError_t, const char *) { return GRASS_E_CUDA; }
}
int main() {
  for (uint32_t depth : {4u, 2u, 1u}) {
    for (device = 0; device < 3; device++) {
      grass_graph g;
      g.device = device;
      g.info.n = g.info.num_edges = g.plan_nbig = 1;
      g.tuning.decode_stage_depth = depth;
      g.plan_ok = true;
      refuse = device == 2;  // no launch where the device does not grant it
      launched = refused = 0;
      grass::launch_decode_if_planned(&g, nullptr, nullptr, nullptr, 0);
      if (refused || launched != (device < 2)) {
        printf("depth %u, device %d: launched %d, refused %d\n", depth, device, launched, refused);
        return 1;
      }
    }
  }
}
"""


def test_shared_memory_is_asked_for_on_every_device(tmp_path):
    (tmp_path / "main.cu").write_text(MAIN)
    (tmp_path / "runtime.cpp").write_text(RUNTIME)
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-w",
             "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-cudart", "none"]
    out = subprocess.run(["nvcc", *flags, "-o", str(tmp_path / "main"), str(tmp_path / "main.cu"), str(tmp_path / "runtime.cpp"),
                          os.path.join(CSRC, "kernels_decode.cu")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
    run = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
