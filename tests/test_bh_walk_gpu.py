"""Reference walk at the edges of its tasks, margins and stack (GPU).

Per-target interaction counts equal the oracle's walk bit for bit and forces
agree within 1e-5 (p99, vector relative), as in tests/test_bh_gpu.py: sizes
around the tasks of 16 and 32 targets and the change between them, opening
angles from 0 to 2, coordinates far from the origin and of extreme scale
(where the margins of the per-warp decisions leave every node to the
per-target test), bodies on cube faces, and a stack so small that subtrees
are walked node by node.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err
from test_bh_gpu import _bh, _oracle_tree

pytestmark = pytest.mark.gpu


def _check(nb, orc, s, theta, eps=0.01, leaf=1):
    _, _, nodes, _, merges = _oracle_tree(orc, s, max_nodes=8 * len(s["x"]) + 4096)
    r = _bh(nb, s, theta=theta, eps=eps, leaf=leaf)
    ox, oy, oz, oint = orc.bh_forces(nodes, s["x"], s["y"], s["z"], s["m"], theta, 1.0, eps,
                                     leaf_cap=leaf)
    np.testing.assert_array_equal(r["inter"], oint)
    n0 = np.sqrt(ox.astype(np.float64) ** 2 + oy.astype(np.float64) ** 2 +
                 oz.astype(np.float64) ** 2)
    ok = np.isfinite(n0) & (n0 > 0)
    if ok.any():
        err = vec_rel_err(*[a[ok] for a in r["acc"]], ox[ok], oy[ok], oz[ok])
        assert np.percentile(err, 99) <= 1e-5, np.percentile(err, 99)


@pytest.mark.parametrize("leaf", [1, 8])
@pytest.mark.parametrize("n", [100, 127, 129, 1025, 32767, 32768, 32769])
def test_task_edges(nb, orc, n, leaf):
    _check(nb, orc, nb.ics.plummer(n, seed=n), 0.5, leaf=leaf)


@pytest.mark.parametrize("leaf", [1, 4])
@pytest.mark.parametrize("theta", [0.0, 0.1, 1.0, 1.5, 2.0])
def test_opening_angles(nb, orc, theta, leaf):
    _check(nb, orc, nb.ics.plummer(3000, seed=5), theta, leaf=leaf)


@pytest.mark.parametrize("scale,shift", [(1.0, 3000.0), (1e-12, 0.0), (1e-18, 0.0), (1e15, 0.0)])
def test_scales_and_offsets(nb, orc, scale, shift):
    s = nb.ics.plummer(2000, seed=6)
    for k in ("x", "y", "z"):
        s[k] = (s[k] * np.float32(scale) + np.float32(shift)).astype(np.float32)
    _check(nb, orc, s, 0.5, eps=0.01 if scale >= 1.0 else 0.0)


def test_lattice_bodies_on_cube_faces(nb, orc):
    # a lattice whose root cube subdivides exactly: bodies on the faces of cubes
    # (a face belongs to both its cubes in the containment test)
    g = np.linspace(-1.0, 1.0, 17, dtype=np.float32)
    x, y, z = (a.ravel() for a in np.meshgrid(g, g, g, indexing="ij"))
    rng = np.random.default_rng(3)
    s = dict(x=x.copy(), y=y.copy(), z=z.copy(),
             m=rng.uniform(0.5, 1.5, x.size).astype(np.float32))
    for theta in (0.5, 1.2):
        _check(nb, orc, s, theta)


@pytest.mark.parametrize("leaf", [1, 8])
@pytest.mark.parametrize("n", [1500, 40000])
def test_small_stack_walks_subtrees_node_by_node(nb, orc, n, leaf):
    from nbgb import _lib
    nb.check(_lib.lib().nbgb_selftest_group_walk_stack(64))
    try:
        _check(nb, orc, nb.ics.plummer(n, seed=8), 0.4, leaf=leaf)
    finally:
        nb.check(_lib.lib().nbgb_selftest_group_walk_stack(512))
