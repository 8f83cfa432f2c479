"""Kernels that need more dynamic shared memory than the default have their limit
raised on every device they are launched on: a limit belongs to the device that
is current when it is set, and contexts may sit on several devices.  Run against
stand-ins for the two runtime calls (no device needed)."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fermi.jl_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "fcc_common.cuh"
static int current = 0, calls[4] = {0, 0, 0, 0}, refuse = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "refused"; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int bytes) {
  if (refuse) return cudaErrorInvalidValue;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && bytes == 200000) ++calls[current];
  return cudaSuccess;
}
static void kernel(int) {}
int main() {
  fcc::SmemLimit a, b;
  a.raise(kernel, 200000);
  a.raise(kernel, 200000);
  current = 1;
  refuse = 1;
  int code = 0;
  try { a.raise(kernel, 200000); } catch (const fcc::Error& e) { code = e.code; }
  refuse = 0;
  a.raise(kernel, 200000);
  a.raise(kernel, 200000);
  current = 0;
  a.raise(kernel, 200000);
  b.raise(kernel, 200000);
  std::printf("%d %d %d\n", calls[0], calls[1], code);
}
"""


def test_limits_are_raised_once_on_each_device(tmp_path):
    cxx = shutil.which("g++")
    inc = "/usr/local/cuda/include"
    if cxx is None or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "p.cpp", str(tmp_path / "p")
    src.write_text(PROGRAM)
    r = subprocess.run([cxx, "-std=c++17", "-I", CSRC, "-I", inc, str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    # a: once on each device (a refused call is reported and made again), b: its own kernel's
    assert r.returncode == 0 and r.stdout.split() == ["2", "1", "-3"], r.stdout + r.stderr


def test_every_limit_goes_through_it():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = open(path).read()
        if os.path.basename(path) == "fcc_common.cuh":
            assert len(re.findall(r"cudaFuncSetAttribute\(", text)) == 1
        else:
            assert "cudaFuncSetAttribute" not in text, path
