"""Launches without a single site to advance keep the order of the steps around
them: slabs that hold nothing but boundary sites, and ensemble groups whose
domain is all solid."""
import numpy as np
import pytest

from test_download_paths_gpu import _case, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_slabs_of_boundary_sites(precision, monkeypatch):
    # two layers between Zou-He faces: every site is a boundary site
    c = _case((64, 48, 2), [1, 1, 1, 1, 3, 2], 1, 60)
    c["vel0"][:, :, 0] = [0.0, 0.0, 0.01]
    f0, out0 = _run(c, precision, monkeypatch, True, True)
    f1, out1 = _run(c, precision, monkeypatch, False, False)
    np.testing.assert_array_equal(f1, f0)
    for (d0, v0), (d1, v1) in zip(out0, out1):
        np.testing.assert_array_equal(d1, d0)
        np.testing.assert_array_equal(v1, v0)


@pytest.mark.parametrize("order", [(0, 1), (1, 0), (0, 1, 1, 0, 1)])
def test_all_solid_domains(order, monkeypatch):
    from jyulb.ensemble import Domain, Ensemble

    rng = np.random.default_rng(61)
    flow = 0.01 * rng.uniform(-1, 1, (160, 64, 64, 3))

    def domain(kind):
        phase = np.ones((160, 64, 64) if kind == 0 else (9, 8, 7), np.uint8)
        if kind == 1:
            phase[:] = 0
            return Domain(phase)
        phase[:, 0] = phase[:, -1] = 0
        return Domain(phase, None, flow * phase[..., None], 0.05, [1e-6, 0.0, 0.0])

    out = []
    for group in ("0.001", "0"):  # every domain alone; all together
        monkeypatch.setenv("JLB_BATCH_GROUP", group)
        monkeypatch.setenv("JLB_BATCH_BLOCK", "128")
        e = Ensemble([domain(k) for k in order])
        res = []
        for n in (1, 7, 2):
            e.evolve(n)
            res += [x for d in range(len(order)) for x in e.moments(d)]
        out.append(res)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
