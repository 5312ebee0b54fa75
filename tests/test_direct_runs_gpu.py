"""Length of the plain FP32 runs in a compensated direct sum (GPU).

All sources lie at one place, one unit from the target.  A few have mass M, the
others a mass m whose term is 0.97 of half a unit in the last place of M's: a
plain chain that begins with M loses every term of m, and a compensated sum
keeps those of other chains and those after a fold.  The heavy sources begin
the 32 chains (16 slices, even and odd sources) that a slice-wise sum of 64
sources in turn has.  A plain chain has at most 256 terms, so 32 chains lose at
most 255 terms each, and the terms themselves, products of a reciprocal square
root, are off by at most 2^-21:

    |error| / (32 terms of M) <= 255 * 0.97 * 2^-24 / 1.5 + 2^-21

Chains of 304 terms (9,728 sources in 16 slices) would lose 1.16 times that.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("through", ["forces", "system"])
@pytest.mark.parametrize("n", [4864, 8192, 8193, 9000, 9728])
def test_terms_lost_by_plain_chains(nb, n, through):
    eps = np.float32(0.01)
    unit = 0.97 * 2.0 ** -24 / 1.5
    m = np.full(n, 1.5 * unit, np.float32)
    j = np.arange(n)
    m[(j < 64) & (j % 4 < 2)] = 1.5  # the first term of each of 32 chains
    s = {k: np.zeros(n, np.float32) for k in ("x", "y", "z", "vx", "vy", "vz")}
    s["x"][n - 1] = -1.0  # the target
    s["m"] = m
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(float(eps))
    if through == "forces":
        with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                       "mass": s["m"]}) as p:
            calc.computeForces(p.device)
            p.download()
            got = float(p.host["acc_x"][n - 1])
    else:
        sysm = nb.System(calc, s)
        got = float(sysm.read()["ax"][n - 1])
        sysm.close()
    calc.close()
    term = (1.0 + float(eps) ** 2) ** -1.5
    want = float(m[:-1].astype(np.float64).sum()) * term
    assert abs(got - want) <= 32 * 1.5 * term * (255 * unit + 2.0 ** -21)
