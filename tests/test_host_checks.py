"""Host-side checks of the launch helpers, compiled with the host compiler against a fake of the CUDA runtime."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FAKE = r"""
#include "tpf_host.cuh"
static int g_reserved, g_sets;
static size_t g_static;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrReservedSharedMemoryPerBlock ? g_reserved : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { *a = {}; a->sharedSizeBytes = g_static; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++g_sets; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
namespace tpf { char* last_error_buffer() { static char b[512]; return b; } }
static const void* const kernel = &g_sets;  // handles of kernels are opaque to the host compiler
// prints code of the call, number of attribute calls, code of a second call
static void run(int reserved, size_t stat, int align) {
  static tpf::PerDeviceOnce* keep[64];
  static int n;
  tpf::PerDeviceOnce& once = *(keep[n++] = new tpf::PerDeviceOnce());
  g_reserved = reserved;
  g_static = stat;
  g_sets = 0;
  const int a = tpf::ensure_dynamic_smem(kernel, 200000, once, align), sets = g_sets;
  printf("%d %d %d\n", a, sets, tpf::ensure_dynamic_smem(kernel, 200000, once, align));
}
int main() {
  run(1024, 0, 1024);     // what the device has
  run(1024, 1024, 1024);  // padded static variables
  run(1024, 16, 1024);    // static variables in front of the array
  run(512, 0, 1024);      // a device that keeps another amount
  run(512, 16, 1);        // a kernel that aligns by hand
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                    reason="needs the host compiler and the CUDA headers")
def test_unaligned_shared_memory_base_is_an_error_before_the_launch(tmp_path):
    src, exe = tmp_path / "fake.cpp", tmp_path / "fake"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(CUDA, "include"),
                    "-I" + os.path.join(ROOT, "openfold3_triangle_kernel_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    # TPF_ERR_UNSUPPORTED (2) before any attribute is set, and again on the next call
    assert lines[:5] == ["0 1 0", "0 1 0", "2 0 2", "2 0 2", "0 1 0"]


def test_a_warp_comes_together_again_after_every_wait():
    """Kernels wait by warp_wait*, which end in a warp barrier: what follows (TMEM loads and stores, UMMAs, copies) is for whole
    warps, and lanes may leave a bare mbar_wait one by one.  The bounded-wait self-test waits with one thread."""
    csrc = os.path.join(ROOT, "openfold3_triangle_kernel_b200", "csrc")
    bare = []
    for name in sorted(set(os.listdir(csrc)) - {"tpf_ptx.cuh", "tpf_selftest.cu"}):
        with open(os.path.join(csrc, name)) as f:
            bare += [f"{name}:{i}" for i, line in enumerate(f, 1) if re.search(r"\bmbar_(try_)?wait\d?\s*\(", line)]
    assert bare == []
