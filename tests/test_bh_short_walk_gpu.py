"""Short reference walks of large systems, node by node (GPU).

Around the lines of the rule (body count, theta, leaf capacity) every body has
the oracle's interaction count, whichever way its walk goes, and forces within
1e-5 (99th percentile, vector relative: the tolerance of tests/test_bh_gpu.py) of
the oracle's.  In an ensemble the sums of a large system do not depend on what
else is walked with it.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err
from test_bh_gpu import _bh, _oracle_tree

pytestmark = pytest.mark.gpu


LINE = [(196607, 1.25, 1), (196608, 1.25, 1), (196608, 1.125, 1), (196608, 0.9, 16),
        (196609, 1.2, 8), (196639, 2.0, 16)]
LARGE = [(1310720, 1.0, 1), (1310721, 1.0, 1), (1310721, 0.9, 8)]


@pytest.mark.parametrize("gen,n,theta,leaf", [(g, *c) for g in ("cube", "plummer") for c in LINE] +
                         [("cube", *c) for c in LARGE])
def test_counts_and_forces_match_the_oracle(nb, orc, gen, n, theta, leaf):
    s = nb.ics.uniform_cube(n, seed=7) if gen == "cube" else nb.ics.plummer(n, seed=7)
    _, _, nodes, _, merges = _oracle_tree(orc, s)
    assert merges == 0
    ox, oy, oz, oint = orc.bh_forces(nodes, s["x"], s["y"], s["z"], s["m"], theta, 1.0, 0.01,
                                     leaf_cap=leaf)
    r = _bh(nb, s, theta=theta, leaf=leaf)
    np.testing.assert_array_equal(r["inter"], oint)
    for acc in (r["acc"], _bh(nb, s, theta=theta, leaf=leaf, count=False)["acc"]):
        err = vec_rel_err(*acc, ox, oy, oz)
        assert np.percentile(err, 99) <= 1e-5, np.percentile(err, 99)


@pytest.mark.parametrize("leaf", [1, 16])
def test_ensemble_sums_do_not_depend_on_the_mix(nb, leaf):
    from nbgb.serving import Ensemble
    large, others = nb.ics.uniform_cube(200000, seed=1), [nb.ics.plummer(n, seed=n)
                                                          for n in (9000, 40000)]

    def run(states):
        ens = Ensemble(hbm_budget_bytes=4 << 30, group_walk=0, theta=1.25, leaf_capacity=leaf)
        ids = [ens.submit(st, 2, 1e-4) for st in states]
        while ens.tick() != (0, 0):
            pass
        ens.synchronize()
        out = {}
        while (res := ens.poll(want_state=True)) is not None:
            out[res[0]["request_id"]] = res[1]
        ens.close()
        return out[ids[0]]

    alone, mixed = run([large]), run([large, *others])
    for k in alone:
        np.testing.assert_array_equal(alone[k], mixed[k])
