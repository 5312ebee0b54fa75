"""Handles of their own in two host threads (GPU).

Distinct handles may be used from different threads.  Two systems whose sizes
take the same kernel with different amounts of shared memory step side by
side; every call succeeds and gives, bit for bit, what it gives alone.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the small-system kernel (32 targets per CTA of 152 SMs above 2,432 bodies), and above it
@pytest.mark.parametrize("sizes", [(4000, 3000), (9728, 7400)])
def test_small_direct_sums_of_two_sizes(nb, sizes):
    calls = 1500

    def make(n):
        s = nb.ics.plummer(n, seed=n)
        p = nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                      "mass": s["m"]})
        c = nb.DirectForceCalculator()
        c.setSofteningParameter(0.01)
        return c, p

    def forces(p):
        p.download()
        return [p.host[f"acc_{a}"].copy() for a in "xyz"]

    work = [make(n) for n in sizes]
    want = []
    for c, p in work:
        c.computeForces(p.device)
        want.append(forces(p))
    failed = []

    def run(c, p):
        try:
            for _ in range(calls):
                c.computeForces(p.device)
        except Exception as e:  # noqa: BLE001  (reported below)
            failed.append(e)

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for (c, p), w in zip(work, want):
        for a, b in zip(forces(p), w):
            np.testing.assert_array_equal(a, b)
        c.close()
        p.close()
