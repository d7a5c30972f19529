"""Shared-memory limits and SM counts are kept per device (a stand-in for the CUDA runtime; no GPU).

A kernel's limit belongs to a device: a process that raises it once, on its first device, has its
launches on the next one refused."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pulsesuite_gb300" / "csrc"

RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
enum cudaDeviceAttr { cudaDevAttrMultiProcessorCount = 16 };
inline int dev = 0, limit[128] = {}, sets = 0, refuse = 0;
inline cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { *v = 100 + d; return cudaSuccess; }
template <class T> cudaError_t cudaFuncSetAttribute(T*, cudaFuncAttribute, int b) {
  ++sets;
  if (refuse) return cudaErrorInvalidValue;
  limit[dev] = b;
  return cudaSuccess;
}
"""

PROGRAM = """
#include <cstdio>
#include <initializer_list>
#include "per_device.cuh"
void kernel(int) {}
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\\n", __LINE__, #x); return 1; }
int main() {
  using sbe::raise_smem;
  refuse = 1;
  CHECK(raise_smem<kernel>(1000) == cudaErrorInvalidValue);
  refuse = 0;
  CHECK(raise_smem<kernel>(1000) == cudaSuccess && limit[0] == 1000);   // not remembered
  const int n = sets;
  CHECK(raise_smem<kernel>(1000) == cudaSuccess && sets == n);          // once a device
  for (int d : {1, 63, 64, 100}) {
    dev = d;
    CHECK(raise_smem<kernel>(1000) == cudaSuccess && limit[d] == 1000);
    CHECK(sbe::sm_count() == 100 + d && sbe::sm_count() == 100 + d);
  }
  dev = 0;
  CHECK(sbe::sm_count() == 100);
  return 0;
}
"""


def test_each_device_has_its_own(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-x", "c++", "-I", tmp_path, "-I", CSRC, tmp_path / "main.cpp",
                    "-o", tmp_path / "main"], check=True)
    p = subprocess.run([tmp_path / "main"], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout


def test_no_limit_is_raised_once_a_process():
    for path in CSRC.glob("*.cu"):
        assert not re.search(r"static\s+(?:const\s+)?(?:bool|cudaError_t)\s+\w+\s*=[^;]*cudaFuncSetAttribute",
                             path.read_text()), path.name
