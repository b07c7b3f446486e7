"""The integer-pipe FP64 operations (tlq_softfp.cuh) against the host's IEEE
operations, bit for bit: the header compiles as plain C++, its FP32 seeds
moved by up to the error the GPU's approximations may have (reciprocal 1 ulp,
reciprocal square root 2^-22.9)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include <cstdint>
static int g_ulp = 0;
static float nudge(float y) {
  for (int q = 0; q < (g_ulp < 0 ? -g_ulp : g_ulp); ++q) y = std::nextafterf(y, g_ulp < 0 ? 0.0f : 4.0f);
  return y;
}
#define TLQ_SF_HOST_SEED(y) nudge(y)
#include "tlq_softfp.cuh"
extern "C" void run(int op, int ulp, const double* a, const double* b, double* o, long n) {
  g_ulp = ulp;
  for (long i = 0; i < n; ++i)
    o[i] = op == 0 ? tlq::sf::div(a[i], b[i]) : op == 1 ? tlq::sf::sqrt_rn(a[i]) : tlq::sf::mul(a[i], b[i]);
}
"""


@pytest.fixture(scope="module")
def soft(tmp_path_factory):
    d = tmp_path_factory.mktemp("softfp")
    src, lib = d / "softfp.cpp", d / "softfp.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{ROOT}/tlaloque_gb300/csrc",
                    str(src), "-o", str(lib)], check=True)
    L = C.CDLL(str(lib))
    D = C.POINTER(C.c_double)
    L.run.argtypes = [C.c_int, C.c_int, D, D, D, C.c_long]

    def run(op, ulp, a, b):
        o = np.empty_like(a)
        L.run(op, ulp, *(v.ctypes.data_as(D) for v in (a, b, o)), len(a))
        return o

    return run


def operands(n, seed, spread):
    """Significands at their edges (0, all ones, few low or high bits) and random ones."""
    g = np.random.default_rng(seed)
    m = g.integers(0, 1 << 52, n, dtype=np.uint64)
    k = g.integers(0, 8, n)
    full = np.uint64((1 << 52) - 1)
    m = np.select([k == 0, k == 1, k == 2, k == 3, k == 4], [np.uint64(0), full, m & np.uint64(15), m | (full ^ np.uint64(15)),
                                                            m & ~np.uint64(0xFFFFFFFF)], m)
    e = g.integers(1, 2047, n, dtype=np.uint64) if spread else g.integers(1003, 1043, n, dtype=np.uint64)
    return ((g.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072009e-308, 2.2250738585072014e-308,
                    1.7976931348623157e308, 1e-200, 1e200, 3.0, 0.1])


@pytest.mark.parametrize("ulp", [-2, -1, 0, 1, 2])
@pytest.mark.parametrize("op", [0, 1, 2], ids=["div", "sqrt", "mul"])
def test_same_bits_as_ieee(soft, op, ulp):
    s, t = (v.ravel() for v in np.meshgrid(SPECIAL, SPECIAL))
    a = np.concatenate([s, operands(300_000, 1, False), operands(300_000, 2, True)])
    b = np.concatenate([t, operands(300_000, 3, False), operands(300_000, 4, True)])
    if op == 1:
        a = np.concatenate([np.abs(a), SPECIAL])
        b = np.ones_like(a)
    with np.errstate(all="ignore"):
        want = a / b if op == 0 else np.sqrt(a) if op == 1 else a * b
    got = soft(op, ulp, a, b)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))
