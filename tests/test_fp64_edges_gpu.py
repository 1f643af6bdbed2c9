"""FP64 and fast FP64 sites at the edges of the integer forms' operand ranges."""
import numpy as np
import pytest

from test_fp64_ranges_gpu import run_both

pytestmark = pytest.mark.gpu


# the lower edge of the fixed-point form's densities, 1/2: some sites' sums
# round to it or above, the others below
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("rho", [0.5, 0.5 + 1e-11, 0.5 + 2.0 ** -28, 1.5])
@pytest.mark.parametrize("steps", [1, 4])
def test_fast_density_edges(scheme, rho, steps):
    rng = np.random.default_rng(21)
    lat = (6, 7, 33)
    vel = 0.05 * rng.uniform(-1, 1, lat + (3,))
    run_both(lat, scheme, 0.05, (0, 0, 0), np.full(lat, rho), vel, None, steps, fast=True)
    # one velocity everywhere: every bulk site stays at the edge
    run_both(lat, scheme, 0.05, (0, 0, 0), np.full(lat, rho), np.full(lat + (3,), 0.03), None, steps, fast=True)


# acceleration fields with sites far outside the range of the integer form's
# products: NaN and infinities propagate as in the reference, everything else
# keeps its bits
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e160, -1e100, 1e3, 300.0, 1e-200, 3e-310])
@pytest.mark.parametrize("steps", [1, 2])
def test_extreme_acceleration_field(scheme, value, steps):
    rng = np.random.default_rng(22)
    lat = (5, 6, 40)
    den = 1 + 0.01 * rng.uniform(-1, 1, lat)
    vel = 0.02 * rng.uniform(-1, 1, lat + (3,))
    acc = np.where(rng.random(lat + (3,)) < 0.02, value, 1e-5 * rng.uniform(-1, 1, lat + (3,)))
    acc[1, 1, 7] = value
    run_both(lat, scheme, 0.05, (0, 2e-5, 0), den, vel, acc, steps)
