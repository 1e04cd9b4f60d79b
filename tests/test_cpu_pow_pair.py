"""The tonemap's w^(1/gamma) / w in pairs of FP32 numbers, built for the host: its
error against FP64 over densities and gammas, and that every product whose rounding
the pair settles is the float that FP64 arithmetic gives. Divisions are moved by up to
2 ulp, as the GPU's approximate one may be."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

KERNELS = Path(__file__).resolve().parent.parent / "refraktor_gb300" / "csrc" / "kernels"
SOURCE = r"""
#include "pow_pair.h"
#include <cstdint>
static uint64_t state = 1;
namespace rfk_tm {
float pp_div(float a, float b) {
    float q = a / b;
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    if (std::fabs(q) > 1e-37f) q = pp_float(pp_bits(q) + (unsigned)((int)(state >> 33) % 5 - 2));
    return q;
}
}
// worst: relative error; returns the wrongly rounded products among those settled
extern "C" long check(const float* w, const float* col, long n, float gamma, double* worst, long* open, long* refused) {
    const rfk_tm::pow_table t = rfk_tm::make_pow_table(gamma);
    const double inv = 1.0 / (double)gamma;
    long wrong = 0;
    *worst = 0.0;
    *open = *refused = 0;
    for (long i = 0; i < n; i++) {
        float hi, lo, out;
        if (!rfk_tm::pow_pair(w[i], t.t, t.q, hi, lo)) {
            ++*refused;
            continue;
        }
        const double f = std::pow((double)w[i], inv) / (double)w[i];
        *worst = std::fmax(*worst, std::fabs(((double)hi + (double)lo) / f - 1.0));
        if (!rfk_tm::scale_pair(col[i], hi, lo, out)) ++*open;
        else if (rfk_tm::pp_bits(out) != rfk_tm::pp_bits((float)(col[i] * f))) wrong++;
    }
    return wrong;
}
extern "C" float limit() { return rfk_tm::kPowPairError; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pow_pair")
    (d / "t.cpp").write_text(SOURCE)
    # no contraction: the products that CUDA rounds by itself are plain ones here
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", f"-I{KERNELS}", str(d / "t.cpp"), "-o",
                    str(d / "t.so")], check=True)
    L = C.CDLL(str(d / "t.so"))
    L.check.restype, L.limit.restype = C.c_long, C.c_float
    L.check.argtypes = [C.c_void_p, C.c_void_p, C.c_long, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p]
    return L


def _check(L, w, col, gamma):
    worst, opened, refused = C.c_double(), C.c_long(), C.c_long()
    wrong = L.check(w.ctypes.data, col.ctypes.data, w.size, gamma, C.byref(worst), C.byref(opened), C.byref(refused))
    return wrong, worst.value, opened.value / w.size, refused.value


@pytest.mark.parametrize("gamma", [0.5, 0.8, 1.0, 1.3, 2.2, 4.0, 5.0, 1e6])
def test_settled_products_are_those_of_fp64(lib, gamma):
    rng = np.random.default_rng(int(gamma * 10) % 1000)
    n = 1 << 17
    w = np.exp2(rng.uniform(-40.0, 40.0, n)).astype(np.float32)
    w[:64] = np.exp2(np.arange(-32, 32)).astype(np.float32)
    w[64:128] = np.nextafter(w[:64], np.float32(0))
    w[128:192] = np.float32(np.sqrt(0.5)) * w[:64]  # where the exponent is split
    col = (w * rng.uniform(0, 1, n)).astype(np.float32)
    col[::1000] = 0.0
    wrong, worst, opened, refused = _check(lib, w, col, gamma)
    assert wrong == 0 and refused == 0
    # kPowPairError is stated with its measured margin: 2^-34.4 of 2^-33
    assert worst < 2.0 ** -34.3 < 0.5 * lib.limit()
    # of the floats' spacing 2^-24 .. 2^-23 of the product 2 * 2^-33 is open: 1 in 512 to 1 in 256
    assert gamma == 1.0 or opened < 1.0 / 200


def test_what_the_pair_leaves_to_fp64(lib):
    w = np.array([0.0, -1.0, 1e-40, np.inf, np.nan, 3e38, 1e-38], np.float32)
    col = np.ones_like(w)
    # zero, negative, subnormal and non-finite densities, and powers past 2^120
    assert _check(lib, w[:5], col[:5], 2.2)[3] == 5
    assert _check(lib, w[5:], col[5:], 0.5)[3] == 2
    # channels whose product is not a normal number stay open
    one = np.full(4, 2.0, np.float32)
    odd = np.array([1e-38, np.inf, np.nan, 3e38], np.float32)
    assert _check(lib, one, odd, 2.2)[2] == 1.0
