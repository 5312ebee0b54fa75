"""FP64 energies at the edges of the 64-body tiles, and state read-back (GPU).

PE and KE in FP64 against numpy in extended precision: n^2 / 2 terms of one
sign, each within a few 2^-53, added in partial sums of at most n terms, so
the relative error is far below n 2^-53; the bound is 1e-12 (the tolerance of
the full-FP64 system in tests/test_integrator_gpu.py).  Read-back through the
one-kernel path (at most 8,192 bodies) and by copies returns the same values
as the initial state.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pe(s, eps):
    x = np.stack([s[k].astype(np.float64) for k in ("x", "y", "z")])
    m = s["m"].astype(np.float64)
    pe = 0.0
    for i in range(len(m) - 1):
        r2 = ((x[:, i + 1:] - x[:, i:i + 1]) ** 2).sum(0) + float(np.float32(eps)) ** 2
        pe -= float(m[i] * (m[i + 1:] / np.sqrt(r2)).sum())
    return pe


@pytest.mark.parametrize("eps", [0.01, 0.0])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 1000, 4160])
def test_tile_edges(nb, n, eps):
    s = nb.ics.plummer(n, seed=60 + n)
    s["m"] = (s["m"] * np.random.default_rng(n).uniform(0.5, 1.5, n)).astype(np.float32)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(eps)
    sysm = nb.System(calc, s)
    for _ in range(2):  # the counter is left at zero
        ke, pe, mom = sysm.energy()
        v = np.stack([s[k].astype(np.float64) for k in ("vx", "vy", "vz")])
        m = s["m"].astype(np.float64)
        ref = float((0.5 * m * (v ** 2).sum(0)).sum())
        assert abs(ke - ref) <= 1e-12 * max(ref, 1e-300)
        assert np.abs(mom - (m * v).sum(1)).max() <= 1e-12 * np.abs(m * v).sum()
        want = _pe(s, eps)
        assert abs(pe - want) <= 1e-12 * abs(want)
    sysm.close()
    calc.close()


@pytest.mark.parametrize("scale", [1e-12, 1e12])
def test_extreme_distances(nb, scale):
    # squared distances outside the fast reciprocal root's range
    n = 200
    s = nb.ics.plummer(n, seed=4)
    for k in ("x", "y", "z"):
        s[k] = (s[k] * np.float32(scale) * np.float32(1e6 if scale > 1 else 1e-6)).astype(np.float32)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(0.0)
    sysm = nb.System(calc, s)
    _, pe, _ = sysm.energy()
    want = _pe(s, 0.0)
    assert abs(pe - want) <= 1e-12 * abs(want)
    sysm.close()
    calc.close()


@pytest.mark.parametrize("n", [1, 255, 257, 8192, 8193])
def test_read_back(nb, n):
    s = nb.ics.plummer(n, seed=n)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(0.01)
    sysm = nb.System(calc, s)
    got, f64 = sysm.read(), sysm.read_f64()
    for k in ("x", "y", "z", "vx", "vy", "vz", "m"):
        np.testing.assert_array_equal(got[k], s[k])
        if k != "m":
            np.testing.assert_array_equal(f64[k], s[k].astype(np.float64))
    with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": s["m"]}) as p:
        calc.computeForces(p.device)
        p.download()
        for k in "xyz":
            np.testing.assert_array_equal(got["a" + k], p.host["acc_" + k])
    sysm.close()
    calc.close()
