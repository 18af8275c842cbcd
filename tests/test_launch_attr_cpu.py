"""Kernel attributes are set once per device, not once per process: csrc/launch_attr.cuh compiled on the host against counting
stand-ins for the two runtime calls it makes."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "x_algorithm_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
MAIN = r"""
#include "launch_attr.cuh"
#include <assert.h>
#include <thread>
#include <vector>
static thread_local int current = 0;
static std::atomic<int> asked[80];
static std::atomic<bool> refuse{false};
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int bytes) {
  assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize && bytes == 98304);
  asked[current]++;
  return refuse ? cudaErrorInvalidValue : cudaSuccess;
}
void kernel(int) {}
int main() {
  static phx::SmemLimit limit;
  for (int rep = 0; rep < 3; ++rep)
    for (int d : {0, 3, 1, 63}) { current = d; assert(limit.raise(kernel, 98304) == cudaSuccess); }
  assert(asked[0] == 1 && asked[1] == 1 && asked[3] == 1 && asked[63] == 1 && asked[2] == 0);
  current = 70;                                  // beyond the table: every time
  for (int rep = 0; rep < 3; ++rep) assert(limit.raise(kernel, 98304) == cudaSuccess);
  assert(asked[70] == 3);
  current = 2; refuse = true;                    // a refusal is reported and asked again
  assert(limit.raise(kernel, 98304) != cudaSuccess);
  refuse = false;
  assert(limit.raise(kernel, 98304) == cudaSuccess && asked[2] == 2);
  std::vector<std::thread> t;
  for (int i = 0; i < 16; ++i) t.emplace_back([i] { current = 10 + i % 4; for (int r = 0; r < 100; ++r) assert(limit.raise(kernel, 98304) == cudaSuccess); });
  for (auto& x : t) x.join();
  for (int d = 10; d < 14; ++d) assert(asked[d] >= 1 && asked[d] <= 4);
  return 0;
}
"""


def test_limit_is_raised_on_every_device(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", CUDA_INCLUDE, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_no_launcher_keeps_a_flag_of_its_own():
    """Every raised limit goes through the helper, or is set on each launch."""
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        assert not re.search(r"static\s+bool\s+\w*attr\w*", text), f
