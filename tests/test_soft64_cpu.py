"""The integer forms of FP64 operations (csrc/soft64.cuh) against the
hardware's, bit for bit, on the CPU."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jyu-lb_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r"""
#include "soft64.cuh"
using namespace jlb::soft64;
extern "C" {
void s_mul(const double *x, const double *k, double *o, long n) {
    for (long i = 0; i < n; ++i) o[i] = mul(x[i], make_mulc(k[i]));
}
void s_mulz(const double *x, const double *k, double *o, long n) {
    for (long i = 0; i < n; ++i) o[i] = mulz(x[i], make_mulc(k[i]));
}
void s_recip(const double *x, double *o, long n) {
    for (long i = 0; i < n; ++i) {
        uint32_t range = 0;
        o[i] = recip(fix(x[i], range));
    }
}
void s_add_sub(const double *e, const double *o, double *p, double *m, int *least, long n) {
    for (long i = 0; i < n; ++i) {
        int32_t l = 1 << 30;
        add_sub(e[i], o[i], p[i], m[i], l);
        least[i] = l;
    }
}
// o0 = (x + y) + z, o1 = (x + y) - z, o2 = x - y; r, p as the callers check them
void s_chain(const double *x, const double *y, const double *z, double *o0, double *o1, double *o2,
             unsigned *r, unsigned *p, long n) {
    for (long i = 0; i < n; ++i) {
        uint32_t range = 0, least = 0;
        const uint64_t a = fix(x[i], range), b = fix(y[i], range), c = fix(z[i], range), s = add(a, b);
        o0[i] = to_double(add(s, c));
        o1[i] = to_double(sub(s, c, least));
        o2[i] = diff_to_double(a, b);
        r[i] = range;
        p[i] = least;
    }
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("soft64")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(CUDA, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


def numbers(rng, n, e0, e1, signed=False):
    """Random doubles with exponents in [e0, e1] whose significands are random,
    or end in runs of zeros or ones (ties and carries)."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    cut = rng.integers(0, 53, n).astype(np.uint64)
    kind = rng.integers(0, 3, n)
    low = (np.uint64(1) << cut) - np.uint64(1)
    m = np.where(kind == 1, m & ~low, np.where(kind == 2, m | low, m)) & np.uint64((1 << 52) - 1)
    e = rng.integers(1023 + e0, 1024 + e1, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64) if signed else np.zeros(n, np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def same_bits(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("e0,e1,k0,k1", [(-9, -2, -2, 1), (-40, 9, -7, -5), (-200, 200, -200, 9)])
def test_product_with_a_constant(lib, e0, e1, k0, k1):
    rng = np.random.default_rng(e0 + 1000)
    n = 1_000_000
    x, k = numbers(rng, n, e0, e1, True), numbers(rng, n, k0, k1, True)
    # short significands: exact products and exact ties
    x[: n // 4] = np.ldexp(rng.integers(1 << 26, 1 << 27, n // 4) | 1, e0)
    k[: n // 4] = np.ldexp(rng.integers(1 << 26, 1 << 27, n // 4) | 1, k0)
    o = np.empty(n)
    lib.s_mul(ptr(x), ptr(k), ptr(o), ctypes.c_long(n))
    assert same_bits(o, x * k)


def test_fixed_point_chains(lib):
    rng = np.random.default_rng(5)
    n = 2_000_000
    x, y, z = (numbers(rng, n, -9, -2) for _ in range(3))
    y[: n // 8] = x[: n // 8]                                   # exact zero difference
    y[n // 8: n // 4] = np.nextafter(x[n // 8: n // 4], 1)      # smallest differences
    o = [np.empty(n) for _ in range(3)]
    r, p = np.empty(n, np.uint32), np.empty(n, np.uint32)
    lib.s_chain(ptr(x), ptr(y), ptr(z), *(ptr(v) for v in o), ptr(r), ptr(p), ctypes.c_long(n))
    assert np.array_equal(r <= 7, np.max([x, y, z], axis=0) < 0.5)
    assert same_bits(o[0], (x + y) + z)
    d = (x + y) - z
    fine = p < (1 << 31) - (1 << 21)
    assert np.array_equal(fine, d >= 2.0 ** -8)
    assert same_bits(o[1][fine], d[fine])
    assert same_bits(o[2], x - y)


@pytest.mark.parametrize("bad", [-0.1, 0.0, -0.0, 2.0 ** -9 * (1 - 2.0 ** -53), 0.5, 1e-310, np.inf, -np.inf, np.nan])
def test_range_check_sees_other_numbers(lib, bad):
    x, y, z = np.array([bad]), np.array([0.1]), np.array([0.1])
    o = [np.empty(1) for _ in range(3)]
    r, p = np.empty(1, np.uint32), np.empty(1, np.uint32)
    lib.s_chain(ptr(x), ptr(y), ptr(z), *(ptr(v) for v in o), ptr(r), ptr(p), ctypes.c_long(1))
    assert r[0] > 7


def test_product_of_zeros(lib):
    x = np.array([0.0, -0.0, 1.5, -1.5] * 3)
    k = np.repeat([3.0, 18.0, 1 / 72], 4)
    o = np.empty(12)
    lib.s_mulz(ptr(x), ptr(k), ptr(o), ctypes.c_long(12))
    assert same_bits(o, x * k)


def test_reciprocals(lib):
    rng = np.random.default_rng(7)
    n = 2_000_000
    x = numbers(rng, n, -8, 1)
    # the ends of a binade, where the quotient's own binade changes
    x[:6] = [1.0, 0.5, 2.0, np.nextafter(1, 2), np.nextafter(1, 0), np.nextafter(2, 1)]
    o = np.empty(n)
    lib.s_recip(ptr(x), ptr(o), ctypes.c_long(n))
    assert same_bits(o, 1.0 / x)


def test_sums_and_differences(lib):
    rng = np.random.default_rng(8)
    n = 2_000_000
    e = numbers(rng, n, -40, 9)
    o = np.ldexp(numbers(rng, n, 0, 0, True), np.frexp(e)[1] - 1 - rng.integers(0, 75, n))
    o[: n // 50] = 0.0
    o[n // 50: n // 25] = -0.0
    p, m, least = np.empty(n), np.empty(n), np.empty(n, np.int32)
    lib.s_add_sub(ptr(e), ptr(o), ptr(p), ptr(m), ptr(least), ctypes.c_long(n))
    fine = least >= 2
    assert np.array_equal(fine, np.frexp(e)[1] - np.where(o == 0, -1023, np.frexp(o)[1]) >= 2)
    assert same_bits(p[fine], (e + o)[fine]) and same_bits(m[fine], (e - o)[fine])
