"""Which domains of an ensemble run in groups, by the launches a call makes:
short calls and domains with boundary nodes run together, small domains join a
group whatever their place in the list -- with the values of the ensemble
stepped together."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, FIXED_DEN, FIXED_VEL = 0, 2, 3


def domain(shape, d, duct=False):
    from jyulb.ensemble import Domain

    rng = np.random.default_rng(d)
    phase = np.ones(shape, np.uint8)
    vel = 0.01 * rng.uniform(-1, 1, shape + (3,))
    bc = [FIXED_VEL, FIXED_DEN, WALL, WALL, WALL, WALL] if duct else None
    if not duct:
        phase[:, 0] = phase[:, -1] = 0
        vel[phase == 0] = 0
    return Domain(phase, None, vel, 0.05 + 0.002 * d, [1e-6, 0.0, 0.0], bc)


LARGE, MIDDLE, SMALL = (40, 30, 25), (20, 15, 10), (8, 8, 8)  # 2.28, 0.23 and 0.04 MB; groups of 1 MB
CASES = {
    # name: (domains, launches a step in groups, together)
    "alternating": ([(LARGE, False), (SMALL, False)] * 4, 4, 1),
    "small first": ([(SMALL, False)] * 3 + [(LARGE, False)], 1, 1),
    "ducts": ([(LARGE, True), (MIDDLE, True)] * 3, 2, 2),
    "ducts and channels": ([(MIDDLE, True), (MIDDLE, False)] * 4 + [(LARGE, False)], 4, 2),
    "middle": ([(MIDDLE, False)] * 10, 3, 1),
    "few": ([(MIDDLE, False)] * 5, 1, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_launches_and_values(name, monkeypatch):
    from jyulb.ensemble import Ensemble

    kinds, grouped, together = CASES[name]
    monkeypatch.setenv("JLB_BATCH_BLOCK", "128")
    out = []
    for group in ("1", "0"):
        monkeypatch.setenv("JLB_BATCH_GROUP", group)
        e = Ensemble([domain(shape, d, duct) for d, (shape, duct) in enumerate(kinds)])
        res, per_step = [], []
        for n in (1, 8, 3, 5):
            before = e.info()["launches"]
            e.evolve(n)
            per_step.append((e.info()["launches"] - before) / n)
            for d in range(len(kinds)):
                res += list(e.moments(d))
        res += [e.populations(d) for d in range(len(kinds))]
        out.append(res)
        long = grouped if group == "1" else together
        assert per_step == [together, long, together, long]
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
