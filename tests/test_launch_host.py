"""Host side of the kernel launches (csrc/launch.cuh) with a fake of the runtime, without a GPU."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "makani_b200", "csrc")
CUDA = next((d for d in (os.environ.get("CUDA_HOME"), os.environ.get("CUDA_PATH"), "/usr/local/cuda")
             if d and os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <set>
#include "launch.cuh"
static int device = 0, calls = 0;
static bool refuse = false;
static std::set<std::pair<const void*, int>> allowed;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
  ++calls;
  if (refuse) return cudaErrorInvalidValue;
  allowed.insert({f, device});
  return cudaSuccess;
}
#define EXPECT(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
  static std::atomic<uint64_t> first, second;
  const char f = 0, g = 0;
  refuse = true;
  EXPECT(mk::allow_shared_memory(first, &f, 100000) != cudaSuccess);
  refuse = false;      // a refusal is not kept
  EXPECT(mk::allow_shared_memory(first, &f, 100000) == cudaSuccess && allowed.count({&f, 0}));
  const int before = calls;
  EXPECT(mk::allow_shared_memory(first, &f, 100000) == cudaSuccess && calls == before);
  device = 1;      // a second device of the process, another kernel, devices that no bit stands for
  EXPECT(mk::allow_shared_memory(first, &f, 100000) == cudaSuccess && allowed.count({&f, 1}));
  EXPECT(mk::allow_shared_memory(second, &g, 100000) == cudaSuccess && allowed.count({&g, 1}) && !allowed.count({&g, 0}));
  for (device = 62; device < 70; ++device)
    for (int k = 0; k < 2; ++k) EXPECT(mk::allow_shared_memory(second, &g, 100000) == cudaSuccess && allowed.count({&g, device}));
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or CUDA is None, reason="no host compiler or CUDA headers")
def test_shared_memory_is_allowed_on_every_device(tmp_path):
    src, exe = tmp_path / "launch.cpp", tmp_path / "launch"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-isystem", os.path.join(CUDA, "include"), "-o", str(exe), "-x", "c++", str(src)], check=True)
    run = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert run.returncode == 0, run.stdout
