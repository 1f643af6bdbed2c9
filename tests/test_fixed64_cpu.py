"""The fixed-point collision (csrc/lbm_fixed64.cuh) against the collision in
extended precision, on the CPU."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jyu-lb_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
C = np.array([(-1, -1, 0), (-1, 0, -1), (-1, 0, 0), (-1, 0, 1), (-1, 1, 0), (0, -1, -1), (0, -1, 0), (0, -1, 1),
              (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, -1), (0, 1, 0), (0, 1, 1), (1, -1, 0), (1, 0, -1), (1, 0, 0),
              (1, 0, 1), (1, 1, 0)])
NNZ = np.abs(C).sum(1)

SRC = r"""
#include "lbm_fixed64.cuh"
using namespace jlb;
extern "C" void s_collide(double *f, int scheme, double we, double wo, const double *g, double *mom, int *ok, long n) {
    const FixConsts k = make_fix_consts(scheme == 1, scheme == 2, we, wo, g);
    for (long i = 0; i < n; ++i)
        ok[i] = k.ok && (scheme == 2 ? collide_fixed<true>(f + 19 * i, k, g, true, mom + 4 * i)
                                     : collide_fixed<false>(f + 19 * i, k, g, true, mom + 4 * i));
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("fixed64")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=gnu++20", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(CUDA, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


def populations(rng, n, speed=0.05, noise=0.01):
    w = np.array([1 / 3, 1 / 18, 1 / 36])[NNZ]
    v = speed * rng.uniform(-1, 1, (n, 3))
    d = 1 + 0.05 * rng.uniform(-1, 1, (n, 1))
    cu = v @ C.T
    return w * (d * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * (v ** 2).sum(1, keepdims=True)) +
                noise * rng.uniform(-1, 1, (n, 19)))


def collide(f, scheme, we, wo, g, T):
    """The reference's collision (jyulb/D3Q19.pyx:655-940) in type T."""
    f = f.astype(T)
    we, wo = T(we), T(wo if scheme == 1 else we)
    a = np.array(g, dtype=T)
    c = C.astype(T)
    one, third = T(1), T(1) / T(3)
    w = np.array([third, one / T(18), one / T(36)], dtype=T)[NNZ]
    den = f.sum(1)
    j = f @ c
    if T is np.longdouble:  # exact: extended precision alone would lose a small j
        x = np.ldexp(f, 61).astype(np.int64)
        den, j = (v.astype(T) / T(2) ** 61 for v in (x.sum(1), x @ C))
    u = j / den[:, None] + a / T(2)
    s = den[:, None] * u
    h2 = we * s[:, :, None] * u[:, None, :] + (one - we / T(2)) * (a[:, None] * s[:, None, :] + a * s[:, :, None])
    if scheme == 2:
        pi = np.einsum("nq,qa,qb->nab", f, c, c) - np.eye(3, dtype=T) * (den * third)[:, None, None]
        h2 = h2 + (one - we) * pi
        h0, h1 = den, j + a * den[:, None]
    else:
        h0, h1 = we * den, wo * s + (one - wo / T(2)) * a * den[:, None]
    cc = np.einsum("qa,qb->qab", c, c) - np.eye(3, dtype=T) * third
    out = w * (h0[:, None] + T(3) * (h1 @ c.T) + T(4.5) * np.einsum("qab,nab->nq", cc, h2))
    if scheme != 2:
        r = (one - (we + wo) / T(2)) * f - (we - wo) / T(2) * f[:, ::-1]
        r[:, 9] = (one - we) * f[:, 9]
        out = out + r
    return out, np.concatenate([den[:, None], u], 1)


def run(lib, f, scheme, we, wo, g):
    f = f.copy()
    n = len(f)
    mom, ok, g = np.empty((n, 4)), np.empty(n, np.int32), np.array(g, dtype=np.float64)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (f, g, mom, ok)]
    lib.s_collide(p[0], scheme, ctypes.c_double(we), ctypes.c_double(wo), p[1], p[2], p[3], ctypes.c_long(n))
    return f, mom, ok != 0


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("tau", [0.505, 0.56, 0.8, 1.0, 3.0])
@pytest.mark.parametrize("g", [(0, 0, 0), (1e-6, 0, 0), (1e-5, -2e-4, 1e-3)])
def test_against_extended_precision(lib, scheme, tau, g):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision")
    rng = np.random.default_rng(int(tau * 1000) + scheme)
    f = populations(rng, 4000)
    we, wo = 1 / tau, 1 / (0.25 / (tau - 0.5) + 0.5)
    got, mom, ok = run(lib, f, scheme, we, wo, g)
    assert ok.all()
    want, wmom = collide(f, scheme, we, wo, g, np.longdouble)
    plain, pmom = collide(f, scheme, we, wo, g, np.float64)
    # half an ulp of the store, and the fixed-point roundings: E and O at most
    # 3/4 of 2^-61 each, the second moments' 3/4 of 2^-59 scaled by at most
    # (18 + 9 sqrt 2 + 3 sqrt 3) we / 72 < 1: below 2^-58 in all
    err = np.abs(got.astype(np.longdouble) - want).astype(np.float64)
    assert (err <= 2.0 ** -53 * np.abs(got) + 2.0 ** -58).all()
    # five roundings of half an ulp: density, its reciprocal, j, their product,
    # the added a/2
    merr = np.abs(mom.astype(np.longdouble) - wmom).astype(np.float64)
    assert (merr <= 5 * 2.0 ** -53 * (np.abs(mom) + np.abs(np.array((0,) + tuple(g))))).all()
    # and closer than the same formulas in FP64
    rms = lambda e: float(np.sqrt((e.astype(np.float64) ** 2).mean()))  # noqa: E731
    assert rms(got - want) <= rms(plain - want)
    assert rms(mom - wmom) <= rms(pmom - wmom)


@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_refuses_what_is_out_of_range(lib, scheme):
    base = populations(np.random.default_rng(0), 1, noise=0.0)
    base /= base.sum()
    for q, v in ((9, 1.0), (9, -0.1), (9, np.nan), (9, np.inf), (3, 0.125), (3, 2.0 ** -9 * 0.99), (3, 0.0), (3, -1e-3),
                 (16, np.inf)):
        f = base.copy()
        f[0, q] = v
        assert not run(lib, f, scheme, 1.0 / 0.8, 1.0, (0, 0, 0))[2][0], (q, v)
    for scale in (0.45, 1.55):
        assert not run(lib, base * scale, scheme, 1.0 / 0.8, 1.0, (0, 0, 0))[2][0]
    assert not run(lib, base, scheme, 1.0 / 0.8, 1.0, (0.5, 0, 0))[2][0]
    assert not run(lib, base, scheme, 2.5, 1.0, (0, 0, 0))[2][0]
    assert not run(lib, base, scheme, 1.0 / 0.8, 1.0, (0, 0, 0))[2][0] == 0
