"""Path sort of the Barnes-Hut build at its edges (GPU).

The tree built on the sorted bodies equals the oracle's insertion tree node
for node (bit-exact, as in tests/test_bh_gpu.py): sizes around one and two
buckets, the part and warp sizes within a bucket, the largest bucket count and
the change of scatter width; bodies that share their key (coincident sets
larger than a bucket, in one place and in several); and bodies in sorted and
in reversed order.  Larger sizes, across the change to the radix sort, by node
count and depth.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_bh_gpu import _bh, _oracle_tree
from treeutil import compare

pytestmark = pytest.mark.gpu


def _same_tree(nb, orc, s):
    _, _, ref, depth, _ = _oracle_tree(orc, s, max_nodes=34 * len(s["x"]) + 4096)
    r = _bh(nb, s, count=False)
    assert r["stats"] == (len(ref), depth)
    assert compare(r["nodes"], ref) == []


@pytest.mark.parametrize("n", [1, 2, 31, 33, 191, 192, 193, 255, 257, 383, 384, 385, 1000, 4097,
                               20000])
def test_sizes(nb, orc, n):
    _same_tree(nb, orc, nb.ics.plummer(n, seed=300 + n))


@pytest.mark.parametrize("order", ["sorted", "reversed", "shuffled"])
def test_input_order(nb, orc, order):
    n = 6000
    s = nb.ics.uniform_cube(n, seed=2)
    by = np.lexsort((s["z"], s["y"], s["x"]))
    if order == "reversed":
        by = by[::-1]
    if order == "shuffled":
        by = np.random.default_rng(1).permutation(n)
    _same_tree(nb, orc, {k: np.ascontiguousarray(v[by]) for k, v in s.items()})


@pytest.mark.parametrize("places", [1, 3])
def test_coincident_bodies(nb, orc, places):
    # thousands of equal keys per place, among spread bodies
    n = 9000
    s = nb.ics.plummer(n, seed=11)
    pick = np.random.default_rng(2).permutation(n)[:6000]
    for k in ("x", "y", "z"):
        s[k][pick] = s[k][pick[np.arange(6000) % places]]
    _same_tree(nb, orc, s)


@pytest.mark.parametrize("n", [196607, 196609, 262143, 262145, 1310720, 1310721])
def test_large_sizes(nb, orc, n):
    s = nb.ics.uniform_cube(n, seed=5, side=10.0)
    calc = nb.BarnesHutCalculator(2.0)
    with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": s["m"]}) as p:
        calc.computeForces(p.device)
    got = calc.tree_stats()
    calc.close()
    _, _, ref, depth, _ = _oracle_tree(orc, s, max_nodes=4 * n)
    assert got == (len(ref), depth)
