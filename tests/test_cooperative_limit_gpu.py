"""Small-system steps where a cooperative launch is refused (GPU).

A process that has fewer SMs than the device reports (a share of the GPU) cannot
launch one CTA per SM that wait on one another.  The driver's refusal is made on
the host; the steps are then taken one at a time, with the same state and
accelerations bit for bit, also when a pending half kick is carried over.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ctas", [(9, 1), (1217, 64), (4864, 151)])
def test_refused_launches_take_single_steps(nb, n, ctas):
    limit = nb.lib().nbgb_selftest_cooperative_limit
    s = nb.ics.plummer(n, seed=n)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(0.01)
    calc.set_flags(nb.FLAG_COMPENSATED)

    def run(limits):
        sysm = nb.System(calc, s)
        try:
            for lim in limits:
                nb.check(limit(lim))
                sysm.step(1e-3, 3)
            out = {**sysm.read_f64(), **{"f" + k: v for k, v in sysm.read().items()}}
        finally:
            nb.check(limit(0))
            sysm.close()
        return out

    want = run([0, 0, 0])
    for limits in ([ctas] * 3, [0, ctas, 0]):
        got = run(limits)
        for k in want:
            np.testing.assert_array_equal(got[k], want[k])
    calc.close()


def test_limit_is_validated(nb):
    assert nb.lib().nbgb_selftest_cooperative_limit(-1) == 1  # NBGB_ERR_INVALID_ARG
