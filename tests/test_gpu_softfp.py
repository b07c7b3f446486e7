"""The device branches of tlq_softfp.cuh (FP64 division, square root and
multiplication on the integer pipe, with the GPU's own seeds) against NumPy's
IEEE operations, bit for bit, on the operands of the host test; and the
sigmoid's reciprocal (recip_ge1 of tlq_mlp.cuh) against the rounded 1/x."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from tests.test_softfp import SPECIAL, operands
from tlaloque_gb300 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "tlq_mlp.cuh"
#include "tlq_softfp.cuh"
__global__ void k_op(int op, const double* a, const double* b, double* o, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = op == 0 ? tlq::sf::div(a[i], b[i]) : op == 1 ? tlq::sf::sqrt_rn(a[i]) : tlq::sf::mul(a[i], b[i]);
}
__global__ void k_recip(const float* x, float* o, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) o[i] = tlq::mlp::recip_ge1(x[i]);
}
extern "C" int run_op(int op, const double* a, const double* b, double* o, long n) {
  double* d = nullptr;
  if (cudaMalloc(&d, 3 * n * sizeof(double))) return 1;
  int rc = cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice) ||
           cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  k_op<<<(unsigned)((n + 255) / 256), 256>>>(op, d, d + n, d + 2 * n, n);
  rc = rc || cudaMemcpy(o, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  return cudaFree(d) || rc;
}
extern "C" int run_recip(const float* x, float* o, long n) {
  float* d = nullptr;
  if (cudaMalloc(&d, 2 * n * sizeof(float))) return 1;
  int rc = cudaMemcpy(d, x, n * sizeof(float), cudaMemcpyHostToDevice);
  k_recip<<<(unsigned)((n + 255) / 256), 256>>>(d, d + n, n);
  rc = rc || cudaMemcpy(o, d + n, n * sizeof(float), cudaMemcpyDeviceToHost);
  return cudaFree(d) || rc;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    d = tmp_path_factory.mktemp("gpusoftfp")
    src, lib = d / "softfp.cu", d / "softfp.so"
    src.write_text(SRC)
    # (the flags of the unit that holds the plain stages)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-O3", "-fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    f"-I{build.CSRC}", str(src), "-o", str(lib)], check=True)
    L = C.CDLL(str(lib))
    D, F = C.POINTER(C.c_double), C.POINTER(C.c_float)
    L.run_op.argtypes = [C.c_int, D, D, D, C.c_long]
    L.run_recip.argtypes = [F, F, C.c_long]
    return L


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double if a.dtype == np.float64 else C.c_float))


@pytest.mark.parametrize("op", [0, 1, 2], ids=["div", "sqrt", "mul"])
def test_device_bits(device, op):
    s, t = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    a = np.concatenate([s, operands(1_000_000, 1, False), operands(1_000_000, 2, True)])
    b = np.concatenate([t, operands(1_000_000, 3, False), operands(1_000_000, 4, True)])
    if op == 1:
        near = (np.float64(1.0).view(np.uint64) + np.arange(1_000_000, dtype=np.uint64)).view(np.float64)
        a = np.concatenate([np.abs(a), SPECIAL, near, 2.0 * near, 4.0 - near])
        b = np.ones_like(a)
    with np.errstate(all="ignore"):
        want = a / b if op == 0 else np.sqrt(a) if op == 1 else a * b
    got = np.empty_like(a)
    assert device.run_op(op, ptr(a), ptr(b), ptr(got), len(a)) == 0
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


def recip(device, x):
    o = np.empty_like(x)
    assert device.run_recip(ptr(x), ptr(o), len(x)) == 0
    return o


def test_reciprocal(device):
    """Every x of a binade.  The approximation is within 1 ulp (2^-23); one
    fused Newton step squares that (2^-46) and adds its own rounding's 2^-47,
    2^-22.4 of an ulp: a result is off, by one ulp, only where 1/x lies that
    close to the middle of two numbers, 3 of 2^23 by chance; 16 allowed."""
    m = np.arange(1 << 23, dtype=np.uint32)
    for e in (0, 1, 7, 64, 125):
        x = (m | np.uint32((127 + e) << 23)).view(np.float32)
        want = (np.float32(1.0) / x).view(np.int32).astype(np.int64)
        off = recip(device, x).view(np.int32).astype(np.int64) - want
        assert np.abs(off).max() <= 1 and np.count_nonzero(off) <= 16


def test_reciprocal_ends(device):
    x = np.array([1.0, 2.0, 2.0**125, 2.0**126, 1.5 * 2.0**126, 2.0**127, 3.4028235e38, np.inf, np.nan], np.float32)
    o = recip(device, x)
    assert o[0] == 1.0 and o[1] == 0.5 and o[2] == np.float32(2.0**-125)
    # subnormal quotients and infinity: 0 (the smallest normal number is 2^-126)
    assert o[3] in (0.0, np.float32(2.0**-126)) and (o[4:8] == 0.0).all() and np.isnan(o[8])
