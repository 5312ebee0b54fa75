"""Nodes and centres of mass of the Barnes-Hut build at the edges of its blocks (GPU).

Small trees equal the oracle's insertion tree node for node.  Larger ones are
checked against themselves: every node's mass and centre of mass, recomputed
in float32 from its children in octant order, is the same bit for bit (single
products, sums and quotients, which IEEE rounds alike everywhere), and a leaf
of one body is that body.  Sizes: the 256-body blocks of the node kernels, the
512-body blocks of the centres of mass, one thread block over the edges between
them (128 blocks) or several, more edges between those than threads; chains of
one-child cells that overflow what a block holds; and several segments.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_bh_gpu import _bh, _oracle_tree
from treeutil import compare

pytestmark = pytest.mark.gpu


def _check_sums(s, nodes):
    kids = nodes["children"]
    leaf = nodes["is_leaf"] != 0
    assert np.array_equal(leaf, (kids < 0).all(axis=1))
    one = leaf & (nodes["particle_count"] == 1)
    b = nodes["particle_index"][one]
    pos = np.stack([s["x"][b], s["y"][b], s["z"][b]], 1).astype(np.float32)
    assert np.array_equal(nodes["com"][one], pos)
    assert np.array_equal(nodes["mass"][one], s["m"][b].astype(np.float32))
    p = np.flatnonzero(~leaf)
    m = np.zeros(len(p), np.float32)
    c = np.zeros((len(p), 3), np.float32)
    cnt = np.zeros(len(p), np.int64)
    for o in range(8):
        k = kids[p, o]
        on = np.flatnonzero(k >= 0)
        q = k[on]
        w = nodes["mass"][q]
        m[on] = m[on] + w
        c[on] = c[on] + nodes["com"][q] * w[:, None]
        cnt[on] += nodes["particle_count"][q]
    assert np.array_equal(nodes["particle_count"][p], cnt)
    assert np.array_equal(nodes["mass"][p], m)
    assert np.array_equal(nodes["com"][p], c / m[:, None])
    assert nodes["particle_count"][0] == len(s["x"])


def _clusters(n, size, seed):
    """Coincident sets of `size` bodies, their places spread over a cube."""
    r = np.random.default_rng(seed)
    at = r.random((-(-n // size), 3), dtype=np.float32)[np.arange(n) // size]
    return {"x": at[:, 0].copy(), "y": at[:, 1].copy(), "z": at[:, 2].copy(),
            "m": r.random(n, dtype=np.float32) + np.float32(0.5)}


@pytest.mark.parametrize("n", [256, 511, 512, 513, 1023, 1025, 4608])
def test_oracle_tree(nb, orc, n):
    s = nb.ics.plummer(n, seed=n)
    _, _, ref, depth, _ = _oracle_tree(orc, s, max_nodes=34 * n + 4096)
    r = _bh(nb, s, count=False)
    assert r["stats"] == (len(ref), depth)
    assert compare(r["nodes"], ref) == []


# pairs and triples: 12 cells and more per body, and cells around most edges
@pytest.mark.parametrize("n,size", [(513, 2), (1537, 3), (2047, 600), (4096, 4096)])
def test_chains(nb, orc, n, size):
    s = _clusters(n, size, seed=n)
    _, _, ref, depth, _ = _oracle_tree(orc, s, max_nodes=34 * n + 4096)
    r = _bh(nb, s, count=False)
    assert r["stats"] == (len(ref), depth)
    assert compare(r["nodes"], ref) == []


@pytest.mark.parametrize("n,size", [(65535, 1), (65536, 1), (65537, 1), (200001, 1),
                                    (60001, 3), (100001, 3), (8400001, 1)])
def test_edges_between_blocks(nb, n, size):
    if size > 1:
        s = _clusters(n, size, seed=9)
    elif n > 1000000:
        s = nb.ics.uniform_cube(n, seed=9)
    else:
        s = nb.ics.plummer(n, seed=9)
    _check_sums(s, _bh(nb, s, theta=2.0, count=False)["nodes"])


def test_repeated_builds_of_changing_size(nb):
    # counters that a build leaves for the next, in one calculator: the same
    # forces bit for bit as from a new one
    calc = nb.BarnesHutCalculator(0.7, group_walk=True)
    calc.setGravitationalConstant(1.0)
    calc.setSofteningParameter(0.01)
    for n in (700, 70000, 33, 70001, 2):
        s = nb.ics.uniform_cube(n, seed=n)
        with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                       "mass": s["m"]}) as p:
            for _ in range(2):
                calc.computeForces(p.device)
            p.download()
            got = [p.host[f"acc_{a}"].copy() for a in "xyz"]
        _check_sums(s, calc.nodes())
        fresh = _bh(nb, s, theta=0.7, eps=0.01, count=False, group=True)["acc"]
        for a, b in zip(got, fresh):
            np.testing.assert_array_equal(a, b)
    calc.close()


@pytest.mark.parametrize("group", [False, True])
def test_forces_after_a_capacity_regrow(nb, group):
    # chains of one-child cells need more nodes than a first call provides: the
    # walk that followed the failed build wrote nothing that stays
    s = _clusters(1536, 3, seed=4)
    n = len(s["x"])
    calc = nb.BarnesHutCalculator(0.5, group_walk=group)
    calc.setSofteningParameter(0.01)
    got = []
    with nb.ScopedParticleData(n, {"pos_x": s["x"], "pos_y": s["y"], "pos_z": s["z"],
                                   "mass": s["m"]}) as p:
        for _ in range(2):
            calc.computeForces(p.device)
            p.download()
            got.append([p.host[f"acc_{a}"].copy() for a in "xyz"])
    assert calc.tree_stats()[0] > 3 * n + 64
    calc.close()
    for a, b in zip(*got):
        assert np.all(np.isfinite(a)) and np.any(a != 0)
        np.testing.assert_array_equal(a, b)
