"""The arrays that the adjoint's calls take (CPU): kernels copy only memory of
the adjoint's own device, and Python refuses arrays that are too short or of
another type before any call."""
import ctypes as C
import os
import subprocess

import pytest

from nbody_b200 import adjoint

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
BUILD = os.path.join(HERE, "_build")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SHIM = r"""
#include "devptr.h"
static int g_type, g_device, g_error, g_cleared;
extern "C" cudaError_t cudaGetLastError() { ++g_cleared; return cudaSuccess; }
extern "C" int local(int type, int device, int error, int on) {
  g_type = type; g_device = device; g_error = error; g_cleared = 0;
  const int r = nbody::local_to(&g_type, on, [](cudaPointerAttributes* a, const void*) {
    if (g_error) return cudaErrorInvalidValue;
    a->type = static_cast<cudaMemoryType>(g_type);
    a->device = g_device;
    return cudaSuccess;
  });
  return r + 10 * g_cleared;
}
"""
UNREGISTERED, HOST, DEVICE, MANAGED = range(4)  # cudaMemoryType


@pytest.fixture(scope="module")
def local():
    os.makedirs(BUILD, exist_ok=True)
    src, so = os.path.join(BUILD, "devptr_check.cpp"), os.path.join(BUILD, "devptr_check.so")
    with open(src, "w") as f:
        f.write(SHIM)
    # -Bsymbolic: its own cudaGetLastError, not that of a CUDA runtime already loaded
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", os.path.join(CUDA, "include"),
                    "-I", os.path.join(ROOT, "n-body-code_b200", "csrc"), "-o", so, src], check=True)
    return C.CDLL(so).local


def test_only_memory_of_the_own_device_goes_to_the_copy_kernel(local):
    assert local(DEVICE, 0, 0, 0) == 1 and local(DEVICE, 1, 0, 1) == 1
    assert local(DEVICE, 1, 0, 0) == 0  # a peer's
    assert local(MANAGED, 1, 0, 0) == 1
    assert local(HOST, 0, 0, 0) == 0 and local(UNREGISTERED, 0, 0, 0) == 0
    assert local(DEVICE, 0, 1, 0) == 10  # a failed query leaves no error behind


class Array:
    """What the wrapper asks of a tensor."""

    def __init__(self, n, size=8, cuda=True, floating=True, contiguous=True):
        self.n, self.size, self.is_cuda, self.c = n, size, cuda, contiguous
        self.dtype = type("dtype", (), {"is_floating_point": floating})

    def is_contiguous(self):
        return self.c

    def element_size(self):
        return self.size

    def numel(self):
        return self.n

    def data_ptr(self):
        return 4096


def test_arrays_are_checked_before_a_call():
    assert adjoint._p(Array(10), 10).value == 4096
    assert adjoint._p(Array(11), 10).value == 4096
    for bad in (Array(9), Array(10, size=4), Array(10, cuda=False), Array(10, floating=False),
                Array(10, contiguous=False)):
        with pytest.raises(AssertionError):
            adjoint._p(bad, 10)


class Matrix(Array):
    """Three rows of n values, `row` apart."""

    def __init__(self, n, row=None, column=1, rows=3, **kw):
        super().__init__(n, **kw)
        self.shape, self.strides = (rows, n), (row or n, column)

    def stride(self):
        return self.strides


def test_rows_are_checked_before_a_call():
    def at(t, n):
        return [p.value for p in adjoint._rows(t, n)]
    assert at(Matrix(10), 10) == [4096, 4096 + 80, 4096 + 160]
    assert at(Matrix(10, row=16), 10) == [4096, 4096 + 128, 4096 + 256]  # columns of a wider matrix
    assert at(Matrix(12), 10) == [4096, 4096 + 96, 4096 + 192]
    assert at(Matrix(1, row=3, column=3), 1) == [4096, 4096 + 24, 4096 + 48]
    for bad in (Matrix(9), Matrix(10, size=4), Matrix(10, cuda=False), Matrix(10, floating=False),
                Matrix(10, column=3, row=1), Matrix(10, rows=2)):
        with pytest.raises(AssertionError):
            adjoint._rows(bad, 10)
