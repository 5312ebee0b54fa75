"""Direct sum of the largest systems: the tile-ring kernel (GPU).

Against the FP64 direct sum of sampled targets, with the tolerances of
tests/test_direct_gpu.py (per-target vector error <= 2e-5 at the 99th
percentile, <= 1e-3 worst case): both sides of the line from which the kernel
is used, sources that do not fill a tile, zero softening and plain sums.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,eps,comp", [(294911, 0.01, True), (294912, 0.01, True),
                                        (294913, 0.01, True), (900007, 0.01, False),
                                        (1000191, 0.0, True)])
def test_lines(nb, orc, n, eps, comp):
    s = nb.ics.plummer(n, seed=n)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(eps)
    if not comp:
        calc.set_flags(nb.FLAG_SYNC)
    with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": s["m"]}) as p:
        got = []
        for _ in range(2):  # the finished-run counters are left at zero
            calc.computeForces(p.device)
            p.download()
            got.append([p.host[k].copy() for k in ("acc_x", "acc_y", "acc_z")])
    calc.close()
    t = np.concatenate([np.random.default_rng(1).choice(n, 60, replace=False), [0, n - 1]])
    G = nb.default_params().G
    ref = orc.direct_f64(s["x"], s["y"], s["z"], s["m"], G, eps, targets=t)
    err = vec_rel_err(*(a[t] for a in got[0]), *ref)
    assert np.percentile(err, 99) <= 2e-5 and err.max() <= 1e-3
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
