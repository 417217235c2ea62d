"""CPU: what has to be set up once per device is not set up once per process."""

import pathlib
import re
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "sage_b200" / "csrc"

OPT_IN = r"""
#include "shared_opt_in.h"
#include <cstdio>
#include <vector>

// the runtime's calls, on any number of devices
static int current = 0, clears = 0, refuse = -1;
static std::vector<int> raised;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int *device) { *device = current; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaGetLastError(void) { ++clears; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *, cudaFuncAttribute attribute, int bytes) {
  if (attribute != cudaFuncAttributeMaxDynamicSharedMemorySize || bytes != 77824) return cudaErrorInvalidValue;
  if (current == refuse) return cudaErrorInvalidDevice;
  raised.push_back(current);
  return cudaSuccess;
}

int main() {
  static sageb200::SharedOptIn kernel, other;
  const int order[] = {0, 1, 0, 1, 63, 64, 64, 0};
  for (int device : order) {
    current = device;
    if (kernel("kernel", 77824) != cudaSuccess) return 1;
  }
  current = 2;
  refuse = 2;
  if (kernel("kernel", 77824) != cudaErrorInvalidDevice || clears != 1) return 2;  // reported, and cleared
  refuse = -1;
  if (kernel("kernel", 77824) != cudaSuccess) return 3;  // a refusal is not remembered
  current = 0;
  if (other("other", 77824) != cudaSuccess) return 4;  // each kernel for itself
  for (int device : raised) std::printf("%d ", device);
  return 0;
}
"""


def test_shared_memory_limit_is_raised_on_every_device(tmp_path):
    from sage_b200.build import _nvcc

    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    (tmp_path / "main.cpp").write_text(OPT_IN)
    include = pathlib.Path(_nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-isystem", str(include), "main.cpp", "-o", "main"], cwd=tmp_path,
                   check=True)
    done = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert done.returncode == 0
    # devices past the table of 64 are asked every time
    assert done.stdout.split() == ["0", "1", "63", "64", "64", "2", "0"]


def test_no_kernel_attribute_hangs_on_a_flag_of_the_process():
    for source in sorted(CSRC.glob("*.cu")):
        flags = re.findall(r"static bool \w+\s*(?:=|;)", source.read_text())
        assert not flags, f"{source.name}: {flags}"
