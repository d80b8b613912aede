"""The allocation-free entry point loads everything it can launch on its first call.

Where modules load lazily, the first launch of a kernel loads it, which may allocate and synchronise. A caller that
makes one call before it starts a stream capture must not meet that inside the capture, whatever the number of ranges
of the later calls. No GPU needed: the entry point is built against a CUDA runtime that records what it is asked."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")

RECORDING_RUNTIME = r"""
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>
#include <tpb/noalloc.h>
struct Dim { unsigned x = 1, y = 1, z = 1; };
static std::vector<const void*>& kernels() { static std::vector<const void*> v; return v; }
static std::map<const void*, int> loaded, launched;
static unsigned char scratch[4096];
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char*, int, void*, void*, void*, void*, int*) { kernels().push_back(host); }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 1; }
unsigned __cudaPushCallConfiguration(Dim, Dim, size_t, void*) { return 0; }
int __cudaPopCallConfiguration(Dim*, Dim*, size_t*, void*) { return 0; }
int cudaLaunchKernel(const void* f, Dim, Dim, void**, size_t, void*) { ++launched[f]; return 0; }
int __cudaLaunchKernel(const void* f, Dim, Dim, void**, size_t, void*) { ++launched[f]; return 0; }
int cudaFuncGetAttributes(void* out, const void* f) { std::memset(out, 0, 8); ++loaded[f]; return 0; }
int cudaGetSymbolAddress(void** out, const void*) { *out = scratch; return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 148; return 0; }
int cudaGetLastError() { return 0; }
const char* cudaGetErrorString(int) { return ""; }
}
int main() {
  static unsigned char bytes[64];
  tpb_noalloc_item one{bytes, bytes + 32, 16};
  if (tpb_noalloc_push(&one, 1, nullptr, 0, nullptr) != 0) return 2;
  int launches = 0, missing = 0;
  for (auto& l : launched) launches += l.second;
  for (const void* k : kernels()) missing += loaded[k] == 0 && launched[k] == 0;
  std::printf("kernels %zu launches %d not loaded %d\n", kernels().size(), launches, missing);
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC) and shutil.which("nvcc") is None, reason="no nvcc")
def test_first_call_loads_every_kernel(tmp_path):
    source, binary = tmp_path / "runtime.cc", tmp_path / "first_call"
    source.write_text(RECORDING_RUNTIME)
    subprocess.check_call([NVCC if os.path.exists(NVCC) else "nvcc", "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-cudart", "none", "-I", os.path.join(REPO, "include"),
                           "-I", os.path.join(REPO, "src"), os.path.join(REPO, "src", "kernels", "noalloc.cu"),
                           str(source), "-o", str(binary)])
    out = subprocess.run([str(binary)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.split() == ["kernels", "2", "launches", "1", "not", "loaded", "0"]
