"""The shared-memory opt-in of a kernel (csrc/fr_launch.hpp) against a fake CUDA
runtime of two devices: set on each device that launches the kernel, once, not at
all below 48 KB, and tried again after a failure."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hifiles-solver_b200", "csrc")

FAKE = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
inline int device = 0, calls[2] = {0, 0}, bytes_of[2] = {0, 0}, failures = 0;
inline cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
inline cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int b)
{
  calls[device]++;
  if (failures > 0) { failures--; return cudaErrorUnknown; }
  bytes_of[device] = b;
  return cudaSuccess;
}
"""

PROGRAM = """
#include <cstdio>
#include "fr_launch.hpp"
int main()
{
  frb::SmemLimit small, large;
  for (device = 0; device < 2; device++) small(nullptr, 48 * 1024);
  if (calls[0] || calls[1]) return 1;
  for (int k = 0; k < 3; k++) { device = 0; large(nullptr, 50000); }
  if (calls[0] != 1 || calls[1] != 0 || bytes_of[0] != 50000) return 2;
  failures = 1;
  for (int k = 0; k < 3; k++) { device = 1; large(nullptr, 50000); device = 0; large(nullptr, 50000); }
  if (calls[0] != 1 || calls[1] != 2 || bytes_of[1] != 50000) return 3;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_limit_is_set_once_on_each_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    src, exe = tmp_path / "limit.cpp", str(tmp_path / "limit")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", CSRC, str(src), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
