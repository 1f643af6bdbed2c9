"""The integer forms of FP64 operations (csrc/soft64.cuh) over the operands the
collision passes them: sums and differences of numbers close in size,
reciprocals up to the largest density, and the check of a range."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_soft64_cpu import CSRC, CUDA, numbers, ptr, same_bits

SRC = r"""
#include "soft64.cuh"
using namespace jlb::soft64;
extern "C" {
void s_add_sub(const double *e, const double *o, double *p, double *m, int *least, int *close, long n) {
    for (long i = 0; i < n; ++i) {
        int32_t l = 1 << 30, c = 1 << 30;
        add_sub(e[i], o[i], p[i], m[i], l, &c);
        least[i] = l;
        close[i] = c;
    }
}
void s_recip(const double *x, const double *y, double *s, double *o, long n) {
    uint32_t range = 0;
    for (long i = 0; i < n; ++i) {
        const uint64_t a = add(fix(x[i], range), fix(y[i], range));
        s[i] = to_double(a);
        o[i] = recip(a);
    }
}
void s_within(const double *x, double lo, double hi, int *r, long n) {
    for (long i = 0; i < n; ++i) r[i] = within(x[i], lo, hi);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("soft64e")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(CUDA, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


def test_sums_and_differences_of_close_numbers(lib):
    rng = np.random.default_rng(18)
    n = 2_000_000
    e = numbers(rng, n, -40, 9)
    o = np.ldexp(numbers(rng, n, 0, 0, True), np.frexp(e)[1] - 1 - rng.integers(-1, 13, n))
    k = n // 10
    o[:k] = e[:k]                                               # no difference
    o[k: 2 * k] = np.nextafter(e[k: 2 * k], 0)                  # the smallest
    o[2 * k: 3 * k] = -e[2 * k: 3 * k] * (1 - 2.0 ** -rng.integers(1, 12, k).astype(float))
    p, m, least, close = np.empty(n), np.empty(n), np.empty(n, np.int32), np.empty(n, np.int32)
    lib.s_add_sub(ptr(e), ptr(o), ptr(p), ptr(m), ptr(least), ptr(close), ctypes.c_long(n))
    fine = (least >= 0) & (close >= 1 << 21)
    binade = np.ldexp(1.0, np.frexp(e)[1] - 1)
    with np.errstate(over="ignore"):
        assert np.array_equal(fine, (np.frexp(o)[1] <= np.frexp(e)[1]) & (e - np.abs(o) >= binade * 2.0 ** -8))
    assert same_bits(p[fine], (e + o)[fine]) and same_bits(m[fine], (e - o)[fine])


def test_reciprocals_of_large_densities(lib):
    rng = np.random.default_rng(19)
    n = 1_000_000
    x, y = numbers(rng, n, -9, 1), numbers(rng, n, -9, 1)
    s, o = np.empty(n), np.empty(n)
    lib.s_recip(ptr(x), ptr(y), ptr(s), ptr(o), ctypes.c_long(n))
    assert same_bits(s, x + y) and same_bits(o, 1.0 / (x + y))
    # nineteen populations: the sum of the largest that are accepted
    assert 18 * np.nextafter(0.25, 0) + 1.5 < 8.0


@pytest.mark.parametrize("lo,hi", [(0.125, 0.5), (2.0 ** -5, 1.5), (2.0 ** -9, 0.25)])
def test_within(lib, lo, hi):
    x = np.array([lo, np.nextafter(hi, 0), 0.2, np.nextafter(lo, 0), hi, -0.2, -lo, 0.0, -0.0, 5e-324, 1e300, np.inf,
                  -np.inf, np.nan])
    r = np.empty(len(x), np.int32)
    lib.s_within(ptr(x), ctypes.c_double(lo), ctypes.c_double(hi), ptr(r), ctypes.c_long(len(x)))
    assert (r != 0).tolist() == [True] * 3 + [False] * 11
