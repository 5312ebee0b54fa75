"""Spatial hash grids far above the cell cap are refused (GPU).

2^22 cells per axis are 2^66 cells, which is 0 modulo 2^64, and 10^12 cells do
not fit an int: each axis is checked before it is converted and multiplied, so
nothing is launched on such a grid.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [(8388606.0,) * 3, (2e12, 1.0, 1.0), (1.0, 2e12, 1.0),
                                    (1.0, 1.0, 2e12), (2e12,) * 3, (1e30,) * 3, (6e9,) * 3])
def test_oversize_grids_are_refused(nb, extent):
    s = {k: np.array([0.0, 0.5, 1.0], np.float32) * np.float32(e) for k, e in zip("xyz", extent)}
    calc = nb.SpatialHashCalculator(2.0, 2.0)
    with nb.ScopedParticleData(3, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": np.ones(3, np.float32)}) as p:
        with pytest.raises(nb.CapacityError, match="too large"):
            calc.computeForces(p.device)
    with nb.ScopedParticleData(3, {"pos_x": np.arange(3, dtype=np.float32)}) as p:
        calc.computeForces(p.device)  # and the calculator goes on
        assert calc.grid_info()["total_cells"] == 3 * 2 * 2
    calc.close()
