"""Long runs of bodies that share their first 21 octants (GPU).

One body far away makes the root cube so large that all others lie in a few cells
of depth 21, and many in shared cells of depth 32: the tree equals the oracle's
insertion tree node for node, and the Morton order its stable sort.  A run is
sorted by one thread up to 32 bodies and by its block above.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_bh_gpu import _bh, _oracle_tree
from treeutil import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e6, 1e8])
@pytest.mark.parametrize("n", [3, 33, 34, 35, 66, 257, 300, 1025, 3000])
def test_a_system_beside_a_far_body(nb, orc, n, far):
    s = nb.ics.plummer(n, seed=n)
    s["x"][n // 3] = far
    if n >= 300:  # other clusters, and a run that starts at a block's end
        s["x"][-40:] += np.float32(far / 2)
        s["y"][-80:-40] += np.float32(far / 3)
    ks, si, ref, depth, _ = _oracle_tree(orc, s, max_nodes=34 * n + 4096)
    r = _bh(nb, s, count=False)
    np.testing.assert_array_equal(r["keys"][0], ks)
    np.testing.assert_array_equal(r["keys"][1], si)
    assert r["stats"] == (len(ref), depth)
    assert compare(r["nodes"], ref) == []


def test_two_long_runs_in_two_segments(nb):
    # systems walked together sort their runs apart: bitwise as alone
    from nbgb.serving import Ensemble
    states = []
    for n in (9000, 9001):
        s = nb.ics.plummer(n, seed=n)
        s["x"][7] = 1e8
        states.append(s)

    def run(sel):
        ens = Ensemble(hbm_budget_bytes=2 << 30, softening=0.01)
        ids = [ens.submit(s, 2, 1e-6) for s in sel]
        while ens.tick() != (0, 0):
            pass
        ens.synchronize()
        out = {}
        while (res := ens.poll(want_state=True)) is not None:
            out[res[0]["request_id"]] = res[1]
        ens.close()
        return [out[i] for i in ids]

    both = run(states)
    for s, b in zip(states, both):
        alone = run([s])[0]
        for k in alone:
            np.testing.assert_array_equal(alone[k], b[k])
