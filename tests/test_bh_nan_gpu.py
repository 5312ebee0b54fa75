"""A body with a NaN coordinate in the reference walk (GPU).

No cell contains it and no cell passes its opening test, so it takes every leaf:
with one body per leaf its interaction count is the number of bodies, as in the
per-target rules, whoever shares its warp.
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
