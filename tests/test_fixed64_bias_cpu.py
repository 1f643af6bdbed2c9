"""The fixed-point collision (csrc/lbm_fixed64.cuh) moves the momentum of many
sites by rounding no more, in the mean over the two steps of a pair, than FP64
arithmetic does: rates that make ties of many products included."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_fixed64_cpu import C, CSRC, CUDA, collide, populations

SRC = r"""
#include "lbm_fixed64.cuh"
using namespace jlb;
template <bool DOWN> static int one(double *f, int scheme, const FixConsts &k, const double *g) {
    double mom[4];
    return k.ok && (scheme == 2 ? collide_fixed<true, DOWN>(f, k, g, false, mom) : collide_fixed<false, DOWN>(f, k, g, false, mom));
}
extern "C" void s_collide(double *f, int scheme, int down, double we, double wo, int *ok, long n) {
    const double g[3] = {0, 0, 0};
    const FixConsts k = make_fix_consts(scheme == 1, scheme == 2, we, wo, g);
    for (long i = 0; i < n; ++i) ok[i] = down ? one<true>(f + 19 * i, scheme, k, g) : one<false>(f + 19 * i, scheme, k, g);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision")
    d = tmp_path_factory.mktemp("bias64")
    src, so = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=gnu++20", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(CUDA, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


# (1, 0.8, 1/4): wo/12 = 1/16; (1, 0.75, 1/4): 1/18; (0, 8/9): we/72 = 1/64
@pytest.mark.parametrize("scheme,tau,magic", [(1, 0.8, 0.25), (1, 0.75, 0.25), (1, 0.56, 0.25), (0, 0.8, 0), (0, 8 / 9, 0),
                                              (0, 1.0, 0), (2, 0.8, 0), (2, 1.0, 0)])
@pytest.mark.parametrize("speed", [1e-9, 1e-4, 0.05])
def test_no_steady_momentum(lib, scheme, tau, magic, speed):
    rng = np.random.default_rng(5)
    n = 200_000
    f = populations(rng, n, speed=speed, noise=speed / 5)
    we = 1 / tau
    wo = 1 / (magic / (tau - 0.5) + 0.5) if scheme == 1 else we
    before = f.astype(np.longdouble) @ C.astype(np.longdouble)
    err = []
    for down in (0, 1):
        got, ok = f.copy(), np.empty(n, np.int32)
        lib.s_collide(got.ctypes.data_as(ctypes.c_void_p), scheme, down, ctypes.c_double(we), ctypes.c_double(wo),
                      ok.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(n))
        assert ok.all()
        err.append(got.astype(np.longdouble) @ C.astype(np.longdouble) - before)
    mean = (err[0] + err[1]) / 2
    plain = collide(f, scheme, we, wo, (0, 0, 0), np.float64)[0].astype(np.longdouble) @ C.astype(np.longdouble) - before
    # five standard deviations of the mean of n sites' independent roundings, of
    # which a site's own two share those of the store
    bias = np.abs(mean.mean(0)).astype(np.float64)
    assert (bias <= 5 * mean.astype(np.float64).std(0) / np.sqrt(n)).all()
    assert mean.astype(np.float64).std() <= plain.astype(np.float64).std()
