"""An evolve that fails touches the host arrays no more once it has returned:
the halo rules of den / vel, which it applies first, are then complete."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_halo_rules_end_before_a_failing_evolve_returns():
    from jyulb.defs import BGK, PERIODIC
    from jyulb.isothermal import Solver

    lat = (160, 170, 180)
    s = Solver(np.array(lat, np.int32), BGK, 0.1, np.zeros(3), np.array([PERIODIC] * 6, np.int32), kernel="cxx")
    s.get_phase()[:] = 1
    s.get_phase()[80, 80, 80] = 0
    s.finalize_init()
    s.evolve(1)
    rng = np.random.default_rng(31)
    for n in range(4):
        s.get_den()[:] = 1 + 0.01 * rng.uniform(-1, 1, lat)
        s.get_vel()[:] = 0.01 * rng.uniform(-1, 1, lat + (3,))
        # this kernel has no moving solids: found after the halo rules
        with pytest.raises(Exception, match="no moving solids"):
            s.evolve(1 + n)
        den, vel = s.den.copy(), s.vel.copy()
        np.testing.assert_array_equal(den[:, :, 0], den[:, :, -2])
        np.testing.assert_array_equal(den[:, :, -1], den[:, :, 1])
        np.testing.assert_array_equal(vel[:, :, -1], vel[:, :, 1])
        np.testing.assert_array_equal(vel[:, -1, 1:-1], vel[:, 1, 1:-1])
        np.testing.assert_array_equal(vel[0, 1:-1, 1:-1], vel[-2, 1:-1, 1:-1])
