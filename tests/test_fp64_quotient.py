"""The shared-reciprocal quotients of the FP64 weights (quotient.h), compiled
for the host: each is the IEEE quotient or asks for the division, for random
operands, for quotients next to the middle of two doubles, and for every size
of the approximation's error up to the 2^-18 it may have."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "reef3d_b200", "csrc")
SOURCE = r"""
#include "quotient.h"
using namespace r3d::f64;
// an approximation of 1/b, err of it off, cut to its upper 32 bits where cut
static double approx(double b, double err, int cut) {
    double y = (1.0 / b) * (1.0 + err);
    if (cut) {
        uint64_t u;
        std::memcpy(&u, &y, 8);
        u &= 0xffffffff00000000ull;
        std::memcpy(&y, &u, 8);
    }
    return y;
}
// out[i]: the quotient a/b, and with c the quotient a/(b c) from the bounds of
// 1/b and 1/c; wrong: neither flagged nor IEEE's; flagged: asked for a division
extern "C" void check(const double* a, const double* b, const double* c, long n, double err, int cut, long* wrong,
                      long* flagged) {
    *wrong = *flagged = 0;
    for (long i = 0; i < n; ++i) {
        const double y = reciprocal_below(b[i], approx(b[i], err, cut));
        const double z = y * reciprocal_below(c[i], approx(c[i], err, cut));
        const double d[2] = {b[i], b[i] * c[i]}, r[2] = {y, z};
        for (int q = 0; q < 2; ++q) {
            uint32_t apart = 0;
            const double v = bracket_div(a[i], d[q], r[q], apart);
            if (apart) ++*flagged;
            else if (v != a[i] / d[q]) ++*wrong;
        }
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I" + CSRC, "-o",
                    str(d / "q.so"), str(d / "q.cpp")], check=True)
    return ctypes.CDLL(str(d / "q.so"))


def check(lib, a, b, c, err, cut):
    p = [np.ascontiguousarray(x, dtype=np.float64) for x in (a, b, c)]
    ptr = [x.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for x in p]
    wrong, flagged = ctypes.c_long(), ctypes.c_long()
    lib.check(*ptr, ctypes.c_long(len(p[0])), ctypes.c_double(err), ctypes.c_int(cut), ctypes.byref(wrong),
              ctypes.byref(flagged))
    return wrong.value, flagged.value


def spread(rng, n, lo, hi):
    """Random mantissas over the exponents lo .. hi."""
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi + 1, n)


ERRORS = [0.0, 2.0 ** -53, -2.0 ** -50, 2.0 ** -40, 2.0 ** -21, -2.0 ** -20, 0.99 * 2.0 ** -18, -0.99 * 2.0 ** -18]


@pytest.mark.parametrize("err", ERRORS)
def test_random_quotients(lib, err):
    """Ideal weights over squared indicators of 1e-12 .. 2^499, and sums."""
    rng = np.random.default_rng(1)
    n = 200000
    for lo, hi in ((-40, -30), (-40, 40), (-40, 498)):
        a, b, c = rng.uniform(0.05, 0.9, n), spread(rng, n, lo, hi), spread(rng, n, -40, 40)
        wrong, flagged = check(lib, a, b, c, err, 0)
        assert wrong == 0
        # the bracket's width, 2^-34 of a distance of at most 2^18 ulp
        assert flagged <= 8 + 2 * n * 2.0 ** -14


def next_to_middles(rng, n, product):
    """a, b, c with a/(b c) as close as j / (2 b c) ulp to the middle of two
    doubles: M odd with M d = j mod 2^54 makes a = (M d - j) / 2^54 an integer,
    d = b c of 53 bits (c = 1 unless `product`)."""
    a, b, c = [], [], []
    for _ in range(n):
        x = int(rng.integers(2 ** 25, 2 ** 26)) | 1 if product else int(rng.integers(2 ** 52, 2 ** 53)) | 1
        y = int(rng.integers(2 ** 26, 2 ** 27)) | 1 if product else 1
        j = int(rng.integers(-20, 21)) * 2 + 1
        m = j * pow(x * y, -1, 2 ** 54) % 2 ** 54
        if m < 2 ** 53 or not 2 ** 52 < x * y < 2 ** 53:
            continue
        a.append((m * x * y - j) >> 54)
        b.append(x)
        c.append(y)
    a, b, c = (np.array(v, dtype=np.float64) for v in (a, b, c))
    return a * 2.0 ** -53, b * 2.0 ** (-25 if product else -52), c


@pytest.mark.parametrize("product", [False, True])
@pytest.mark.parametrize("err", ERRORS)
def test_quotients_next_to_a_middle(lib, err, product):
    """Where one residual correction with an approximate reciprocal rounds the
    wrong way (a product of two reciprocals: one in forty of these)."""
    a, b, c = next_to_middles(np.random.default_rng(2), 40000, product)
    assert len(a) > 5000
    for cut in (0, 1) if abs(err) < 2.0 ** -19 else (0,):
        wrong, _ = check(lib, a, b, c, err, cut)
        assert wrong == 0


def test_divisors_next_to_powers_of_two(lib):
    """Mantissas of all ones and all zeros, whose reciprocals lie next to a
    double's neighbours."""
    rng = np.random.default_rng(3)
    near = np.array([1.0 + k * 2.0 ** -52 for k in range(64)] + [2.0 - k * 2.0 ** -52 for k in range(1, 65)])
    a = np.concatenate([near, rng.uniform(0.05, 0.9, 896)])
    aa, bb = (x.ravel() for x in np.meshgrid(a, near))
    for err in ERRORS:
        wrong, _ = check(lib, aa, bb, np.ones_like(bb), err, 0)
        assert wrong == 0
