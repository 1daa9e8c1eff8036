"""A kernel's limit of shared memory holds for one device; a process may use several. The helper that raises it, compiled
against stand-ins for the two runtime calls it makes (no GPU)."""

import ctypes
import re
import subprocess

import pytest

from paged_attention_engine_b200.kernels import build

STAND_IN = r"""
#include <cuda_runtime.h>
namespace fake {
int device = 0, calls[128] = {}, refuse = 0;
inline cudaError_t get(int* d) { *d = device; return cudaSuccess; }
template <typename K> cudaError_t set(K*, cudaFuncAttribute, int) {
  if (refuse) return cudaErrorInvalidValue;
  ++calls[device];
  return cudaSuccess;
}
}
#define cudaGetDevice fake::get
#define cudaFuncSetAttribute fake::set
#include "common.cuh"
void kernel() {}
extern "C" int raise_on(int device, int refuse) {
  static pae::DevicesSet raised;
  fake::device = device;
  fake::refuse = refuse;
  return pae::raise_shared_memory(raised, kernel, 100000, "test");
}
extern "C" int calls_on(int device) { return fake::calls[device]; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    folder = tmp_path_factory.mktemp("limits")
    (folder / "limits.cu").write_text(STAND_IN)
    target = folder / "limits.so"
    subprocess.run([build.find_nvcc(), "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", str(build.CSRC), "-o", str(target), str(folder / "limits.cu")],
                   check=True, capture_output=True, timeout=300)
    return ctypes.CDLL(str(target))


def test_the_limit_is_raised_once_on_every_device(lib):
    for device in (0, 1, 0, 1, 7, 63, 0):
        assert lib.raise_on(device, 0) == 0
    assert [lib.calls_on(d) for d in (0, 1, 2, 7, 63)] == [1, 1, 0, 1, 1]
    assert lib.raise_on(100, 0) == lib.raise_on(100, 0) == 0 and lib.calls_on(100) == 2      # beyond those remembered: every time
    assert lib.raise_on(5, 1) != 0 and lib.raise_on(5, 0) == 0 and lib.calls_on(5) == 1       # a failure is not remembered


def test_no_kernel_remembers_one_device_for_all():
    for path in sorted(build.CSRC.glob("*.cu*")):
        for static in re.findall(r"static [^;{]*(?:bool|cudaError_t|size_t) \w+ =[^;]*;(?:(?!\n}).)*", path.read_text(), re.S):
            assert "cudaFuncSetAttribute" not in static, (path.name, static[:200])
