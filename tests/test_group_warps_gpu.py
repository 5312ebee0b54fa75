"""Group walk with one, two and four warps per group (GPU).

The number of warps follows from the body count.  On both sides of each line,
and for the smallest systems, the list lengths per body equal the oracle's
group walk on the same tree, forces agree within 1e-5 (p99, vector relative:
the lists are the same, their order differs), with buckets, zero softening and a
stack so small that every group spills to its overflow chunk.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err
from test_bh_gpu import _bh, _gmax, _oracle_tree, small_group_stack  # noqa: F401

pytestmark = pytest.mark.gpu


def _check(nb, orc, s, theta, eps, leaf):
    _, _, nodes, _, _ = _oracle_tree(orc, s, max_nodes=34 * len(s["x"]) + 4096)
    r = _bh(nb, s, theta=theta, eps=eps, leaf=leaf, group=True)
    ox, oy, oz, oint = orc.bh_group_forces(nodes, s["x"], s["y"], s["z"], s["m"], theta, 1.0, eps,
                                           group_max=_gmax(nb, s), leaf_capacity=leaf)
    np.testing.assert_array_equal(r["inter"], oint)
    if len(s["x"]) > 1:
        assert np.percentile(vec_rel_err(*r["acc"], ox, oy, oz), 99) <= 1e-5


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 130, 39999, 40000, 114999, 115000])
@pytest.mark.parametrize("leaf,eps", [(1, 0.01), (8, 0.0)])
def test_lines(nb, orc, n, leaf, eps):
    _check(nb, orc, nb.ics.plummer(n, seed=70 + n), 0.6, eps, leaf)


@pytest.mark.parametrize("n,theta", [(400, 0.1), (3000, 0.2)])
def test_spill(nb, orc, small_group_stack, n, theta):  # noqa: F811
    # (at most 256 groups may spill at a time; more are reported as an overflow)
    _check(nb, orc, nb.ics.plummer(n, seed=n), theta, 0.01, 1)
