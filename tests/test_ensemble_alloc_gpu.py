"""Every device allocation of an ensemble's ticks fails once, with either walk (GPU).

The tick that needed it reports the failure and has changed no state: the
engine goes on, and every request ends with the results of a run without the
failure, bit for bit.  The failures begin when direct-sum systems are under way
and the first Barnes-Hut systems arrive (systems that have not started yet are
neither kicked nor drifted, so a tick repeated for them alone shows nothing).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walk", [0, 1])
def test_each_allocation_of_the_ticks_fails_once(nb, walk):
    from nbgb.serving import Ensemble
    fail = nb.lib().nbgb_selftest_fail_allocation
    reqs = [(nb.ics.plummer(n, seed=40 + n), 6) for n in (600, 2500, 9000, 12001)]

    def run(nth):
        ens = Ensemble(hbm_budget_bytes=2 << 30, direct_config=0, group_walk=walk)
        errors = 0
        try:
            ids = {}
            for i, (st, steps) in enumerate(reqs):
                if i == 2:
                    ens.tick()
                    ens.tick()
                ids[ens.submit(st, steps, 1e-3)] = i
            fail(nth)
            for _ in range(200):
                try:
                    if ens.tick() == (0, 0):
                        break
                except nb.ResourceException:
                    errors += 1
            fail(0)
            ens.synchronize()
            out = {}
            while (res := ens.poll(want_state=True)) is not None:
                out[ids[res[0]["request_id"]]] = res[1]
        finally:
            fail(0)
            ens.close()
        return out, errors

    clean, e0 = run(0)
    assert e0 == 0 and len(clean) == len(reqs)
    nth = 0
    while True:
        nth += 1
        got, errors = run(nth)
        if errors == 0:  # fewer allocations than that
            break
        assert errors == 1 and sorted(got) == sorted(clean), nth
        for i in clean:
            for k in ("x", "y", "z", "vx", "vy", "vz"):
                np.testing.assert_array_equal(got[i][k], clean[i][k], err_msg=f"allocation {nth}")
    assert nth > 10
