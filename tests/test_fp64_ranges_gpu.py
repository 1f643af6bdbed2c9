"""FP64 states on both sides of the integer form's operand ranges: densities
from far below to far above 1, and mixtures within a warp, equal the oracle bit
for bit (the sites outside take the FP64 form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, PERIODIC = 0, 1


def run_both(lat, scheme, kvisc, g, den, vel, acc, steps, magic=0.0, fast=False):
    from jyulb.defs import FP64, FP64_FAST
    from jyulb.isothermal import Solver
    from pyoracle import Oracle

    bc = [PERIODIC, PERIODIC, WALL, WALL, PERIODIC, PERIODIC]
    s = Solver(np.array(lat, dtype=np.int32), scheme, kvisc, np.array(g), np.array(bc, dtype=np.int32),
               trt_magic=magic or None, precision=FP64_FAST if fast else FP64)
    o = Oracle(lat, scheme, kvisc, g, bc, magic)
    for x in (s, o):
        x.get_phase()[:] = 1
        x.get_den()[:] = den
        x.get_vel()[:] = vel
        if acc is not None:
            x.get_acc()[:] = acc
        x.finalize_init()
        x.evolve(steps)
    for a, b, bar in ((s.populations(), o.populations(), 1e-12), (s.get_den(), o.get_den(), 1e-12),
                      (s.get_vel(), o.get_vel(), 1e-11)):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        if fast:
            # the fast form's bars; at rest both velocities are rounding
            # noise of the populations
            assert np.abs(a - b).max() <= bar * max(np.abs(b).max(), 1e-5)
        else:
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale", [0.05, 0.07, 0.2, 1.0, 1.4, 1.55, 5.0, 300.0])
def test_densities(scheme, scale):
    rng = np.random.default_rng(3)
    lat = (6, 7, 33)
    den = scale * (1 + 0.05 * rng.uniform(-1, 1, lat))
    vel = 0.02 * rng.uniform(-1, 1, lat + (3,))
    run_both(lat, scheme, 0.05, (1e-5, 0, 0), den, vel, None, 5)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("g", [(0, 0, 0), (0, 2e-5, 0), (1e-5, 0, -3e-5), (1e-5, 2e-5, 3e-5)])
@pytest.mark.parametrize("field", [False, True])
def test_mixed_sites_and_forces(scheme, g, field):
    rng = np.random.default_rng(4)
    lat = (5, 6, 40)
    # a tenth of the sites far from the rest state
    den = np.where(rng.random(lat) < 0.1, 2.0, 1.0) * (1 + 0.01 * rng.uniform(-1, 1, lat))
    vel = 0.05 * rng.uniform(-1, 1, lat + (3,))
    acc = 1e-5 * rng.uniform(-1, 1, lat + (3,)) if field else None
    run_both(lat, scheme, 0.05, g, den, vel, acc, 4)


# rates whose constants vanish or are tiny: tau = 1 (1 - w_e = 0), equal TRT
# rates (c4 = 0), and magic 1/4, for which c3 is 0 up to rounding
@pytest.mark.parametrize("scheme,kvisc,magic", [(0, 1 / 6, 0.0), (1, 1 / 6, 0.0), (2, 1 / 6, 0.0), (1, 1 / 6, 0.25),
                                                (1, 0.02, 0.25), (1, 0.1, 0.25), (1, 1e-3, 0.25), (0, 50.0, 0.0)])
def test_vanishing_constants(scheme, kvisc, magic):
    rng = np.random.default_rng(5)
    lat = (5, 6, 40)
    den = 1 + 0.01 * rng.uniform(-1, 1, lat)
    vel = 0.02 * rng.uniform(-1, 1, lat + (3,))
    run_both(lat, scheme, kvisc, (0, 0, 0), den, vel, None, 6, magic)


@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_rest_and_large_speeds(scheme):
    lat = (5, 6, 40)
    run_both(lat, scheme, 0.1, (0, 0, 0), np.ones(lat), np.zeros(lat + (3,)), None, 3)
    rng = np.random.default_rng(6)
    run_both(lat, scheme, 0.1, (0, 0, 0), np.ones(lat), 0.4 * rng.uniform(-1, 1, lat + (3,)), None, 2)


# the fixed-point form of FP64_FAST: both sides of its operand ranges (density
# 1/2 to 3/2, momentum 1/4), every force pattern, and sites of both kinds in a warp
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale", [0.3, 0.5, 1.0, 1.49, 1.51, 40.0])
@pytest.mark.parametrize("g", [(0, 0, 0), (1e-5, 2e-5, -3e-5)])
def test_fast_densities(scheme, scale, g):
    rng = np.random.default_rng(7)
    lat = (6, 7, 33)
    den = scale * (1 + 0.02 * rng.uniform(-1, 1, lat))
    vel = 0.05 * rng.uniform(-1, 1, lat + (3,))
    run_both(lat, scheme, 0.05, g, den, vel, None, 5, fast=True)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("speed", [0.0, 0.2, 0.4])
@pytest.mark.parametrize("field", [False, True])
def test_fast_speeds_and_fields(scheme, speed, field):
    rng = np.random.default_rng(8)
    lat = (5, 6, 40)
    vel = speed * rng.uniform(-1, 1, lat + (3,))
    acc = 1e-5 * rng.uniform(-1, 1, lat + (3,)) if field else None
    run_both(lat, scheme, 1 / 6, (0, 1e-5, 0), np.ones(lat), vel, acc, 3, fast=True)


@pytest.mark.parametrize("scheme,kvisc,magic", [(1, 1e-3, 0.25), (1, 30.0, 0.0), (0, 30.0, 0.0), (2, 1e-3, 0.0),
                                                (1, 1 / 6, 0.25)])
def test_fast_rates(scheme, kvisc, magic):
    rng = np.random.default_rng(9)
    lat = (5, 6, 40)
    vel = 0.02 * rng.uniform(-1, 1, lat + (3,))
    run_both(lat, scheme, kvisc, (1e-5, 0, 0), np.ones(lat), vel, None, 4, magic, fast=True)
