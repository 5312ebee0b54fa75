"""Direct sum at the edges of its target blocks, source runs and tiles (GPU).

Against the FP64 direct sum, with the tolerances of tests/test_direct_gpu.py
(per-target vector error <= 2e-5 at the 99th percentile, <= 1e-3 worst case);
the SoA route (nbgb_compute_forces) and the packed route (a system's a(0), or
accelerations that overlap an input) run the same sums in the same order, so
they agree bitwise.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err

pytestmark = pytest.mark.gpu


def _state(nb, n, seed):
    s = nb.ics.plummer(n, seed=seed)
    s["m"] = (s["m"] * np.random.default_rng(seed).uniform(0.5, 1.5, n)).astype(np.float32)
    return s


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 511, 512, 513, 1025, 2431, 2433, 4097,
                               4864, 4865, 7296, 7297, 8191, 9728, 9729, 19457, 33000])
def test_block_run_and_tile_edges(nb, orc, n):
    s = _state(nb, n, 40 + n)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(0.01)
    with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": s["m"]}) as p:
        got = []
        for _ in range(2):  # the finished-run counters are left at zero
            calc.computeForces(p.device)
            p.download()
            got.append([p.host[k].copy() for k in ("acc_x", "acc_y", "acc_z")])
    sysm = nb.System(calc, s)
    packed = sysm.read()
    sysm.close()
    calc.close()
    for a, b, k in zip(got[0], got[1], ("ax", "ay", "az")):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, packed[k])
    if n == 1:
        assert all(g[0] == 0.0 for g in got[0])
        return
    tgt = np.random.default_rng(1).choice(n, min(n, 2048), replace=False)
    ref = orc.direct_f64(s["x"], s["y"], s["z"], s["m"], 1.0, 0.01, targets=tgt)
    err = vec_rel_err(*[g[tgt] for g in got[0]], *ref)
    assert np.percentile(err, 99) <= 2e-5 and err.max() <= 1e-3, (np.percentile(err, 99), err.max())


def test_accelerations_that_overlap_an_input(nb):
    # acc_x is pos_x itself: the forces of the positions before the call
    n = 3000
    s = _state(nb, n, 9)
    arrays = {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"], "mass": s["m"]}
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(0.01)
    with nb.ScopedParticleData(n, arrays) as p, nb.ScopedParticleData(n, arrays) as q:
        calc.computeForces(p.device)
        p.download()
        own = q.device.struct.acc_x
        q.device.struct.acc_x = q.device.struct.pos_x
        calc.computeForces(q.device)
        q.download()
        q.device.struct.acc_x = own
        for k in ("acc_x", "acc_y", "acc_z"):
            np.testing.assert_array_equal(p.host[k], q.host[k])
    calc.close()
