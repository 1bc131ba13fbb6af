"""The shared-memory limit of a kernel is set for every device that launches it: the host code that remembers it, compiled
against a stand-in for the CUDA runtime that writes the calls down, and the launches, none of which remembers it otherwise."""
import ctypes
import os
import re
import subprocess

from rllm_b200.kernels import build

RUNTIME = """
#pragma once
#include <stddef.h>
typedef int cudaError_t;
enum { cudaSuccess = 0 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern int device, answer, set_calls, last_device, last_bytes;
static inline cudaError_t cudaGetDevice(int* d) { *d = device; return 0; }
template <typename K> static inline cudaError_t cudaFuncSetAttribute(K, int, int bytes) {
  ++set_calls; last_device = device; last_bytes = bytes;
  return answer;
}
"""
CALLER = """
#include "smem_limit.h"
int device, answer, set_calls, last_device, last_bytes;
static void kernel(int) {}
extern "C" int allow(int d, int bytes, int a, int* out) {
  static SmemLimit limit;
  device = d; answer = a; set_calls = 0;
  const int rc = limit.allow(kernel, bytes);
  out[0] = set_calls; out[1] = last_device; out[2] = last_bytes;
  return rc;
}
"""


def test_the_limit_is_set_on_every_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "caller.cpp").write_text(CALLER)
    so = tmp_path / "caller.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(tmp_path), "-I", build.CSRC, "-o", str(so),
                    str(tmp_path / "caller.cpp")], check=True)
    lib, out = ctypes.CDLL(str(so)), (ctypes.c_int * 3)()

    def allow(dev, size, answer=0):
        return lib.allow(dev, size, answer, out), list(out)

    assert allow(0, 60000) == (0, [1, 0, 60000])
    assert allow(0, 60000)[1][0] == 0 and allow(0, 50000)[1][0] == 0
    assert allow(1, 60000) == (0, [1, 1, 60000])           # another device: set there too
    assert allow(0, 70000) == (0, [1, 0, 70000])           # more than was allowed
    assert allow(1, 70000) == (0, [1, 1, 70000]) and allow(0, 70000)[1][0] == 0
    assert allow(2, 60000, answer=1) == (1, [1, 2, 60000])  # refused: nothing is remembered
    assert allow(2, 60000) == (0, [1, 2, 60000])
    assert [allow(64, 60000)[1][0] for _ in range(2)] == [1, 1]      # beyond the table: set each time


def test_no_launch_remembers_the_limit_for_all_devices():
    for name in sorted(os.listdir(build.CSRC)):
        with open(os.path.join(build.CSRC, name)) as f:
            text = f.read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            before = text[max(0, m.start() - 300): m.start()]
            assert not re.search(r"static (bool|size_t|int) \w+ = (false|0);", before), (name, before)
