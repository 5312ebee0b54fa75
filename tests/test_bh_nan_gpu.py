"""A body with a NaN coordinate in the reference walk (GPU).

No cell contains it and no cell passes its opening test, so it takes every leaf:
with one body per leaf its interaction count is the number of bodies, as in the
per-target rules, whoever shares its warp.  And no body accepts a cell whose
centre of mass is NaN: in a small tree every count equals the per-target rules'
(in float64 on the exported nodes: no quotient of these sets is near theta^2).
"""
from __future__ import annotations

import numpy as np
import pytest

from test_bh_gpu import _bh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", ["x", "y", "z"])
@pytest.mark.parametrize("n", [40, 1000, 40000])
def test_interaction_count(nb, n, axis):
    s = nb.ics.plummer(n, seed=5)
    s[axis][n // 2] = np.nan
    assert _bh(nb, s, theta=0.8)["inter"][n // 2] == n


def _counts(s, nodes, theta, eps):
    out = np.zeros(len(s["x"]), np.int64)
    for t in range(len(out)):
        p = np.array([s["x"][t], s["y"][t], s["z"][t]], np.float64)
        stack = [0]
        while stack:
            q = nodes[stack.pop()]
            inside = bool(np.all(np.abs(p - q["center"]) <= q["half"]))
            if q["is_leaf"]:
                out[t] += not (inside and q["particle_count"] == 1)
                continue
            d2 = ((q["com"].astype(np.float64) - p) ** 2).sum() + eps * eps
            if not inside and (2.0 * q["half"]) ** 2 / d2 < theta * theta:
                out[t] += 1
            else:
                stack += [k for k in q["children"] if k >= 0]
    return out


@pytest.mark.parametrize("theta", [0.5, 2.0])
@pytest.mark.parametrize("n", [17, 18, 33, 200])
def test_counts_of_the_others(nb, n, theta):
    s = nb.ics.plummer(n, seed=5)
    s["y"][n // 2] = np.nan
    r = _bh(nb, s, theta=theta)
    np.testing.assert_array_equal(r["inter"], _counts(s, r["nodes"], theta, 0.01))
