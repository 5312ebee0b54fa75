"""The FP64 pair term of the energies, one pair at a time (GPU).

Two bodies of mass 1, one at the origin and one on an axis at a float distance
d: PE = -1 / sqrt(d^2 + eps^2) is one reciprocal square root of a sum that is
rounded once (its two squares of floats are exact in FP64), and every other
operation is exact.  With u = 2^-53: the rounded sum contributes u / 2, the
refined seed's last operation u and its series 2^-63, so |error| <= 2 u inside
the seed's range; outside it the math library's rsqrt (1 ulp, 2 u) gives 3 u.
"""
from __future__ import annotations

from decimal import Decimal, getcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_pair_term(nb, eps):
    getcontext().prec = 60
    r = np.random.default_rng(5)
    # both sides of the seed's range (2^-112 .. 2^112 squared), and its middle
    d = np.concatenate([2.0 ** r.uniform(-60, 60, 300), 2.0 ** r.uniform(-57, -55, 40),
                        2.0 ** r.uniform(55, 57, 40), 2.0 ** np.arange(-58.0, 59.0)]).astype(np.float32)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(eps)
    z = np.zeros(2, np.float32)
    worst = [0.0, 0.0]
    for v in d:
        s = dict(x=np.array([0.0, v], np.float32), y=z, z=z, vx=z, vy=z, vz=z,
                 m=np.ones(2, np.float32))
        sysm = nb.System(calc, s)
        pe = sysm.energy()[1]
        sysm.close()
        r2 = Decimal(float(v)) ** 2 + Decimal(float(np.float32(eps))) ** 2
        err = float(abs(Decimal(pe) * r2.sqrt() + 1))
        out = not Decimal(2) ** -112 <= r2 < Decimal(2) ** 112
        worst[out] = max(worst[out], err)
    calc.close()
    u = 2.0 ** -53
    assert worst[0] <= 2 * u and worst[1] <= 3 * u, (worst[0] / u, worst[1] / u)
