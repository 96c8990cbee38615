"""Host code of the kernel launches, compiled against a runtime of the test's own (no GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))

# two devices, on which a kernel may have 48 KB of dynamic shared memory until its limit has been raised there
_RUNTIME = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <map>
#include <utility>
static int device = 0, refused = 0, raised = 0;
static std::map<std::pair<int, const void*>, int> limits;
template <typename F> cudaError_t fake_set(F* f, cudaFuncAttribute, int bytes) {
  limits[{device, (const void*)f}] = bytes; ++raised; return cudaSuccess;
}
inline cudaError_t fake_device(int* d) { *d = device; return cudaSuccess; }
inline cudaError_t fake_attribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
inline cudaError_t fake_error() { return cudaSuccess; }
template <typename F, typename... A> cudaError_t fake_launch(const cudaLaunchConfig_t* c, F* f, A&&...) {
  auto it = limits.find({device, (const void*)f});
  if ((int)c->dynamicSmemBytes > (it == limits.end() ? 48 * 1024 : it->second)) ++refused;
  return cudaSuccess;
}
#define cudaFuncSetAttribute fake_set
#define cudaGetDevice fake_device
#define cudaDeviceGetAttribute fake_attribute
#define cudaGetLastError fake_error
#define cudaPeekAtLastError fake_error
#define cudaLaunchKernelEx fake_launch
"""

_STREAM = _RUNTIME + r"""
#include "gemm_stream.cu"
namespace xrt { const Tuning& tuning() { static const Tuning t; return t; } }
int main() {
  for (int turn = 0; turn < 2; ++turn)
    for (device = 0; device < 2; ++device)
      for (int mode = 0; mode < 3; ++mode)
        if (xrt::dispatch_stream<1>(nullptr, nullptr, nullptr, 1, 2048, 8192, 8192, 2048, XRT_F32, mode, 2048ll * 8192, {}, {}, nullptr)) return 1;
  printf("%d %d", refused, raised);
  return 0;
}
"""


def test_products_of_few_rows_raise_their_limit_on_every_device(tmp_path):
    """A process that launches on two devices: no launch asks for more shared memory than was allowed there, and a limit is raised
    once a kernel and device."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    (tmp_path / "main.cu").write_text(_STREAM)
    csrc = os.path.join(os.path.dirname(HERE), "xeno-rt_b200", "csrc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17", "-I", csrc,
                    "-o", str(tmp_path / "main"), str(tmp_path / "main.cu")], check=True, capture_output=True, text=True)
    refused, raised = map(int, subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout.split())
    assert refused == 0 and raised == 2 * 2  # (stored products have rings of three stages, which need none)
