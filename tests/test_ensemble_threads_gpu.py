"""Threads that read different domains of one ensemble at once each get their
own domain's moments."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first_serial", [True, False])
def test_concurrent_moments(first_serial):
    from jyulb.ensemble import Domain, Ensemble

    def domain(d):
        shape = (64, 48, 40 - 3 * d)
        phase = np.ones(shape, np.uint8)
        phase[:, 0] = phase[:, -1] = 0
        vel = np.zeros(shape + (3,))
        vel[..., 0] = 0.01 * (d + 1) * phase
        return Domain(phase, np.full(shape, 1 + 0.01 * d), vel, 0.05, [1e-6, 0.0, 0.0])

    def build():
        e = Ensemble([domain(d) for d in range(4)])
        e.evolve(3)
        return e

    other = build()
    want = [other.moments(d) for d in range(4)]
    e = build()
    if first_serial:
        e.moments(0)
    wrong = [0] * 4

    def read(d):
        for _ in range(40):
            den, vel = e.moments(d)
            wrong[d] += not (np.array_equal(den, want[d][0]) and np.array_equal(vel, want[d][1]))

    threads = [threading.Thread(target=read, args=(d,)) for d in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0] * 4
