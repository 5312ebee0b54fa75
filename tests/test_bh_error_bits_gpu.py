"""Errors of earlier asynchronous calls outlive a capacity regrow (GPU).

A group walk that runs out of overflow chunks, or a tree that outgrows its nodes,
says so in the calculator's error word.  The next call waits, and needs more
tree nodes than it has: it builds again with more, and still reports the
earlier call's failure.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(n):
    """Coincident pairs: 12 tree nodes and more per body, of which an asynchronous
    call has 4 and a first waiting one 3."""
    r = np.random.default_rng(1)
    at = r.random((n // 2, 3), dtype=np.float32)[np.arange(n) // 2]
    return {"pos_x": at[:, 0].copy(), "pos_y": at[:, 1].copy(), "pos_z": at[:, 2].copy(),
            "mass": np.full(n, 1.0 / n, np.float32)}


@pytest.mark.parametrize("what,message", [("walk", "group walk stack overflow"),
                                          ("tree", "octree capacity exceeded")])
def test_regrow_keeps_the_error_of_an_asynchronous_call(nb, what, message):
    hook = nb.lib().nbgb_selftest_group_walk_stack
    calc = nb.BarnesHutCalculator(0.0, group_walk=True)
    calc.setSofteningParameter(0.01)
    flags = calc.params.flags
    if what == "walk":
        s = nb.ics.plummer(20000, seed=23)
        first = {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"], "mass": s["m"]}
    else:
        first = _pairs(2000)
    n0, n = len(first["mass"]), 30000
    with nb.ScopedParticleData(n0, first) as p, nb.ScopedParticleData(n, _pairs(n)) as q:
        try:
            if what == "walk":
                nb.check(hook(64))
            calc.set_flags(flags & ~nb.FLAG_SYNC)
            calc.computeForces(p.device)  # overflows; nobody has looked yet
        finally:
            nb.check(hook(512))
        calc.set_flags(flags)
        calc.setTheta(0.5)
        with pytest.raises(nb.NbodyError, match=message):
            calc.computeForces(q.device)
        assert calc.tree_stats()[0] > max(4 * n0, 3 * n) + 64  # it did build again
        calc.computeForces(q.device)  # and the word is clear
        q.download()
        assert np.isfinite(q.host["acc_x"]).all() and np.any(q.host["acc_x"] != 0)
    calc.close()
