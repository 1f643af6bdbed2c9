"""An ensemble whose domains run in groups, one group after another for all
steps of a call, equals the ensemble stepped together, bit for bit: odd and
even step counts, moving walls, and domains with boundary nodes whose table
ranges begin inside a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALL, PERIODIC, FIXED_DEN, FIXED_VEL, SYMMETRIC = 0, 1, 2, 3, 4


def domains():
    from jyulb.ensemble import Domain

    rng = np.random.default_rng(12)
    out = []
    for d, (shape, bc) in enumerate([((20, 12, 9), None), ((16, 9, 11), [FIXED_VEL, FIXED_DEN, WALL, WALL, WALL, WALL]),
                                     ((7, 13, 30), None), ((9, 8, 7), [PERIODIC, PERIODIC, WALL, SYMMETRIC, PERIODIC, PERIODIC]),
                                     ((33, 10, 6), None), ((12, 9, 10), [WALL, WALL, FIXED_VEL, FIXED_DEN, PERIODIC, PERIODIC])]):
        phase = np.ones(shape, np.uint8)
        vel = np.zeros(shape + (3,))
        if bc is None:
            phase[:, 0, :] = phase[:, -1, :] = 0
            vel[:, -1, :, 0] = 0.02 * (d % 2)
        else:
            vel[..., 0] = 0.01 * rng.uniform(0, 1, shape)
        out.append(Domain(phase, None, vel, 0.05 + 0.01 * d, [1e-6 * (d + 1), 0.0, 0.0], bc))
    return out


def run(monkeypatch, scheme, group, chunks):
    from jyulb.ensemble import Ensemble

    monkeypatch.setenv("JLB_BATCH_GROUP", group)
    monkeypatch.setenv("JLB_BATCH_BLOCK", "128")
    e = Ensemble(domains(), scheme)
    out = []
    for n in chunks:
        e.evolve(n)
        out += [x for d in range(6) for x in e.moments(d)]
    return out + [e.populations(d) for d in range(6)]


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("group", ["0.001", "0.3"])  # every domain alone; two or three together
def test_groups_equal_one_group(monkeypatch, scheme, group):
    chunks = [1, 6, 35]
    for a, b in zip(run(monkeypatch, scheme, group, chunks), run(monkeypatch, scheme, "0", chunks)):
        np.testing.assert_array_equal(a, b)
