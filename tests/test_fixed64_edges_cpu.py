"""The fixed-point collision (csrc/lbm_fixed64.cuh) at the edges of its density
range, on the CPU: a site is refused or agrees with extended precision, and no
accepted site overflows a signed integer on the way."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_fixed64_cpu import C, CSRC, CUDA, NNZ, SRC, collide, populations, run

MAIN = SRC + r"""
#include <cstdio>
#include <vector>
// f and g of stdin (n sites), as written by the test
int main(int argc, char **argv) {
    const int scheme = std::atoi(argv[1]);
    const double we = std::atof(argv[2]), wo = std::atof(argv[3]);
    double g[3], f[19], mom[4];
    int ok;
    if (std::fread(g, 8, 3, stdin) != 3) return 2;
    while (std::fread(f, 8, 19, stdin) == 19) {
        s_collide(f, scheme, we, wo, g, mom, &ok, 1);
        if (!ok) return 3;
    }
    return 0;
}
"""


def compile_(d, name, text, *flags):
    src, out = str(d / (name + ".cpp")), str(d / name)
    with open(src, "w") as f:
        f.write(text)
    subprocess.run(["g++", "-std=gnu++20", "-ffp-contract=off", *flags, "-I", CSRC, "-I", os.path.join(CUDA, "include"),
                    src, "-o", out], check=True)
    return out


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no extended precision")
    return ctypes.CDLL(compile_(tmp_path_factory.mktemp("fixed64"), "t.so", SRC, "-O2", "-shared", "-fPIC"))


@pytest.fixture(scope="module")
def checked(lib, tmp_path_factory):
    """The same collision in a program that an undefined operation ends."""
    return compile_(tmp_path_factory.mktemp("fixed64ub"), "t", "#include <cstdlib>\n" + MAIN, "-O1",
                    "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error")


def sites(rho, n, seed):
    """Equilibria of |u| <= 0.05 whose populations add up to rho exactly."""
    rng = np.random.default_rng(seed)
    v = 0.05 * rng.uniform(-1, 1, (n, 3)) / np.sqrt(3)
    v[0] = (0.05, 0.0, 0.0)
    cu = v @ C.T
    w = np.array([1 / 3, 1 / 18, 1 / 36])[NNZ]
    f = rho * w * (1 + 3 * cu + 4.5 * cu ** 2 - 1.5 * (v ** 2).sum(1, keepdims=True))
    k = np.rint(np.ldexp(f, 54)).astype(np.int64)
    # the rest population takes the remainder, in units of 2^-55
    k[:, 9] = 0
    rest = int(np.ldexp(rho, 55)) - 2 * k.sum(1)
    f = np.ldexp(k.astype(np.float64), -54)
    f[:, 9] = np.ldexp(rest.astype(np.float64), -55)
    assert (np.rint(np.ldexp(f, 55)).astype(np.int64).sum(1) == int(np.ldexp(rho, 55))).all()
    return f


EDGES = [0.5, np.nextafter(0.5, 0), 0.5 + 2.0 ** -53, 0.5 + 1e-12, 0.5 + 1e-10, 0.5 + 1.2e-10, 0.5 + 2.0 ** -29,
         0.5 + 2.0 ** -28, 0.5 + 2.0 ** -27, 0.75, 1.0, 1.5, np.nextafter(1.5, 0), np.nextafter(1.5, 2)]


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("rho", EDGES)
@pytest.mark.parametrize("g", [(0, 0, 0), (1e-5, -2e-4, 1e-3)])
def test_edge_densities(lib, checked, scheme, rho, g):
    f = sites(rho, 500, 11)
    we, wo = 1 / 0.56, 1 / (0.25 / 0.06 + 0.5)
    got, mom, ok = run(lib, f, scheme, we, wo, g)
    if 0.5 + 2.0 ** -27 <= rho < 1.5:
        assert ok.all()
    if not ok.any():
        return
    want, wmom = collide(f, scheme, we, wo, g, np.longdouble)
    # the bound of test_fixed64_cpu.py, and the reciprocal's half an ulp, which
    # reaches a population through den u u times at most 0.5 w_e < 1
    uu = rho * 0.06 ** 2
    err = np.abs(got.astype(np.longdouble) - want).astype(np.float64)
    assert (err[ok] <= 2.0 ** -53 * np.abs(got[ok]) + 2.0 ** -58 + 2.0 ** -53 * uu).all()
    merr = np.abs(mom.astype(np.longdouble) - wmom).astype(np.float64)
    assert (merr[ok] <= 5 * 2.0 ** -53 * (np.abs(mom[ok]) + np.abs(np.array((0,) + tuple(g))))).all()
    data = np.array(g, dtype=np.float64).tobytes() + f[ok].tobytes()
    assert subprocess.run([checked, str(scheme), repr(we), repr(wo)], input=data).returncode == 0


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("tau", [0.5 + 1e-6, 0.6, 3.0, 200.0])
def test_no_overflow_over_the_accepted_range(lib, checked, scheme, tau):
    """Mixtures of populations from the whole range, to the largest densities
    and momenta that are accepted, with forces up to their limit."""
    rng = np.random.default_rng(int(1000 * tau))
    n = 20000
    f = 2.0 ** rng.uniform(-9, -3, (n, 19))
    f[:, 9] = 2.0 ** rng.uniform(-9, 0, n)
    ends = rng.random((n, 19)) < 0.3
    f = np.where(ends, np.where(rng.random((n, 19)) < 0.5, 2.0 ** -9, np.nextafter(0.125, 0)), f)
    f[: n // 4] = populations(rng, n // 4, speed=0.3)
    we, wo = 1 / tau, 1 / (0.25 / (tau - 0.5) + 0.5)
    # |a|, |a| / wo (BGK: we; regularized: a alone) and |a| c2 / we below 1/16
    top = 0.062 * min(1.0, we if scheme == 0 else wo if scheme == 1 else 1.0, we / (1 - we / 2))
    for g in ((0.0, 0.0, 0.0), (top, -top, top)):
        ok = run(lib, f, scheme, we, wo, g)[2]
        assert ok.sum() > 100
        data = np.array(g, dtype=np.float64).tobytes() + f[ok].tobytes()
        assert subprocess.run([checked, str(scheme), repr(we), repr(wo)], input=data).returncode == 0
