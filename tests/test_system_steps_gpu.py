"""Several steps in one call (one launch for a small direct-sum system) (GPU).

Bitwise the same as one-step calls (asynchronous calculators: a synchronous
call closes its last half kick, which rounds v once more).  Against an FP64 kick-drift-kick of the
same initial state: each step's forces carry at most the direct sum's
worst-case error (1e-3 relative, tests/test_direct_gpu.py), so after K steps
of dt the velocities are off by at most 1e-3 K dt |a|max (twice that with the
drift's effect on the forces) and the positions by K dt times that.  The
sizes lie around the changes of the number of targets per CTA (8, 16, 32, 64
times 152 SMs) and the limits of the small-system kernel.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kdk64(orc, s, dt, steps, eps):
    x = [s[k].astype(np.float64) for k in ("x", "y", "z")]
    v = [s[k].astype(np.float64) for k in ("vx", "vy", "vz")]
    dt = float(np.float32(dt))

    def forces():
        d = [c[None, :] - c[:, None] for c in x]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + float(np.float32(eps)) ** 2
        np.fill_diagonal(r2, 1.0)
        f = s["m"].astype(np.float64)[None, :] * r2 ** -1.5
        np.fill_diagonal(f, 0.0)
        return [(f * c).sum(1) for c in d]

    a = forces()
    for _ in range(steps):
        v = [p + 0.5 * dt * q for p, q in zip(v, a)]
        x = [p + dt * q for p, q in zip(x, v)]
        a = forces()
        v = [p + 0.5 * dt * q for p, q in zip(v, a)]
    return x, v, max(np.abs(q).max() for q in a)


@pytest.mark.parametrize("eps", [0.01, 0.0])
@pytest.mark.parametrize("n", [1, 3, 8, 9, 500, 1216, 1217, 2432, 2433, 4864, 4865, 7297, 9728, 9729])
def test_steps_in_one_call(nb, orc, n, eps):
    steps, dt = 3, 1e-4
    s = nb.ics.plummer(n, seed=n)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(eps)
    calc.set_flags(nb.FLAG_COMPENSATED)
    one, many = nb.System(calc, s), nb.System(calc, s)
    for _ in range(steps):
        one.step(dt, 1)
    many.step(dt, steps)
    a, b, fa, fb = one.read_f64(), many.read_f64(), one.read(), many.read()
    one.close()
    many.close()
    calc.close()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k])
    for k in fa:
        np.testing.assert_array_equal(fa[k], fb[k])
        assert np.all(np.isfinite(fb[k]))
    if n <= 2433:
        x, v, acc = _kdk64(orc, s, dt, steps, eps)
        tol = 2e-3 * steps * dt * acc + 1e-15
        for k, c in enumerate("xyz"):
            assert np.abs(b["v" + c] - v[k]).max() <= tol
            assert np.abs(b[c] - x[k]).max() <= steps * dt * tol + 1e-15


def test_long_calls_and_changed_steps(nb):
    # more steps than one launch takes, then another step size
    n, eps = 600, 0.05
    s = nb.ics.plummer(n, seed=2)
    calc = nb.DirectForceCalculator()
    calc.setSofteningParameter(eps)
    calc.set_flags(nb.FLAG_COMPENSATED)
    one, many = nb.System(calc, s), nb.System(calc, s)
    for k in range(300):
        one.step(1e-4, 1)
    one.step(2e-4, 1)
    one.step(2e-4, 1)
    many.step(1e-4, 300)
    many.step(2e-4, 2)
    a, b = one.read_f64(), many.read_f64()
    one.close()
    many.close()
    calc.close()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k])
