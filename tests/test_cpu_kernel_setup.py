"""The per-device setup of a kernel, against a CUDA runtime of stand-ins: what one call did not ask for, a later one gets."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "kernel_setup.h"
#include <cstdio>
static int queries = 0, device = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { ++queries; *n = 70; return cudaSuccess; }
}
int main() {
  static char first, second;
  using penny::kernel_setup;
  std::printf("%d ", kernel_setup(&first, 1000).pairs);
  std::printf("%d ", kernel_setup(&first, 1000, 320).pairs);
  std::printf("%d ", kernel_setup(&first, 1000, 320).pairs);
  std::printf("%d ", kernel_setup(&first, 1000).pairs);
  std::printf("%d ", kernel_setup(&second, 1000, 320).pairs);
  device = 1;
  std::printf("%d ", kernel_setup(&second, 1000, 320).pairs);
  std::printf("queries %d", queries);
}
"""


def test_pairs_are_asked_for_when_first_wanted(tmp_path):
    (tmp_path / "setup.cpp").write_text(SOURCE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(cuda, "include"), "-I", os.path.join(ROOT, "csrc"), "-o", "setup", "setup.cpp"],
                   cwd=tmp_path, check=True, timeout=300)
    out = subprocess.run(["./setup"], cwd=tmp_path, check=True, timeout=60, capture_output=True, text=True).stdout
    assert out == "0 70 70 70 70 70 queries 3"
