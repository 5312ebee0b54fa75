"""Cell order and gather of the spatial hash at the edges of their kernels (GPU).

Cell ids, cell starts, the ascending index list and neighbour counts equal the
oracle's bit for bit; forces agree within 1e-5 (p99, vector relative), as in
tests/test_hash_gpu.py.  Covered: cells of fewer, as many and more bodies than a
block has slots, next to each other and astride blocks; all bodies in one
place; cell tables on both sides of the one-block scan; the lines between the
ways the gather's work is split; positions far from the origin and NaN positions.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import vec_rel_err
from test_hash_gpu import _cube, _run, _uniform

pytestmark = pytest.mark.gpu


def _check(nb, orc, s, cell=2.0, targets=None):
    (ax, ay, az), cells, nbrs = _run(nb, s, cell=cell, cutoff=cell)
    g = orc.hash_build(s["x"], s["y"], s["z"], cell)
    for k in ("dims", "cell_start", "cell_end", "particle_cell", "sorted_indices"):
        np.testing.assert_array_equal(cells[k], g[k])
    t = np.arange(len(s["x"])) if targets is None else targets
    ox, oy, oz, onb = orc.hash_forces(g, s["x"], s["y"], s["z"], s["m"], cell, 1.0, 0.01, targets=t)
    np.testing.assert_array_equal(nbrs[t], onb)
    has = onb > 0
    err = vec_rel_err(ax[t][has], ay[t][has], az[t][has], ox[has], oy[has], oz[has])
    if err.size:
        assert np.percentile(err, 99) <= 1e-5 and err.max() <= 1e-3
    assert np.all(ax[t][~has] == 0.0)
    return cells


def _counts(sizes, seed):
    """sizes[k] bodies in cell k of a row along x (cells of 2), shuffled."""
    rng = np.random.default_rng(seed)
    cell = np.repeat(np.arange(len(sizes)), sizes)
    rng.shuffle(cell)
    n = len(cell)
    s = {"x": (2 * cell + 0.2 + 1.6 * rng.random(n)).astype(np.float32),
         "y": (rng.random(n)).astype(np.float32), "z": (rng.random(n)).astype(np.float32)}
    s["m"] = np.full(n, 1.0 / n, np.float32)
    s["x"][np.argmax(cell == 0)] = np.float32(0.2)  # the grid starts at the lowest body
    return s


@pytest.mark.parametrize("sizes", [(255, 256, 257), (257, 257, 1), (1, 511, 512, 513), (300, 3, 300),
                                   (100, 700, 256, 300, 20, 2000), (256, 256, 256, 256), (1537,)])
def test_crowded_cells(nb, orc, sizes):
    cells = _check(nb, orc, _counts(sizes, seed=sum(sizes)))
    got = cells["cell_end"] - cells["cell_start"]
    assert sorted(got[got > 0].tolist()) == sorted(sizes)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 512, 4097])
def test_one_place(nb, orc, n):
    # coincident bodies: no force between them (a zero offset), all neighbours
    s = {k: np.full(n, 1.5, np.float32) for k in ("x", "y", "z")}
    s["m"] = np.full(n, 1.0 / n, np.float32)
    (ax, _, _), cells, nbrs = _run(nb, s)
    assert np.all(ax == 0.0) and np.all(nbrs == n - 1)
    np.testing.assert_array_equal(cells["sorted_indices"], np.arange(n))


@pytest.mark.parametrize("side", [16.0, 31.0, 47.9, 50.1, 120.0])
def test_table_sizes(nb, orc, side):
    _check(nb, orc, _uniform(3001, side, seed=int(side)))


# on both sides of each line of the gather's split
@pytest.mark.parametrize("n,per_cell", [(131071, 8), (131072, 8), (524287, 8), (524289, 8),
                                        (20001, 22), (20001, 60), (131071, 60), (131073, 60)])
def test_split_lines(nb, orc, n, per_cell):
    s = _cube(n, density=per_cell / 8.0, seed=n)
    _check(nb, orc, s, targets=np.random.default_rng(2).choice(n, 10000, replace=False))


@pytest.mark.parametrize("at", [-1.0e29, 1.0e29])
def test_far_from_the_origin(nb, at):
    # an empty slot's offset must not overflow: three bodies in one place, one beside
    s = {"x": np.full(4, at, np.float32), "y": np.array([0, 0, 0, 1], np.float32),
         "z": np.zeros(4, np.float32), "m": np.ones(4, np.float32)}
    (ax, ay, az), _, nbrs = _run(nb, s)
    assert nbrs.tolist() == [3, 3, 3, 3]
    assert np.all(ax == 0.0) and np.all(az == 0.0)
    f = 1.0 / (1.0 + 1e-4) ** 1.5
    np.testing.assert_allclose(ay, [f, f, f, -3 * f], rtol=1e-5)
    (ax, ay, az), _, nbrs = _run(nb, {k: v[:3] for k, v in s.items()})
    assert nbrs.tolist() == [2, 2, 2]
    assert np.all(ax == 0.0) and np.all(ay == 0.0) and np.all(az == 0.0)


@pytest.mark.parametrize("n", [2001, 400001])
def test_nan_position(nb, orc, n):
    s = _cube(n, seed=n)
    bad = np.array([5, n // 2, n - 1])
    for b, k in zip(bad, ("x", "y", "z")):
        s[k][b] = np.nan
    (ax, ay, az), _, nbrs = _run(nb, s)
    ok = np.setdiff1d(np.arange(n), bad)
    q = {k: np.ascontiguousarray(s[k][ok]) for k in s}
    g = orc.hash_build(q["x"], q["y"], q["z"], 2.0)
    t = np.arange(len(ok))[:: max(1, n // 20000)]
    ox, oy, oz, onb = orc.hash_forces(g, q["x"], q["y"], q["z"], q["m"], 2.0, 1.0, 0.01, targets=t)
    np.testing.assert_array_equal(nbrs[ok][t], onb)
    assert np.percentile(vec_rel_err(ax[ok][t], ay[ok][t], az[ok][t], ox, oy, oz)[onb > 0], 99) <= 1e-5
    for a in (ax, ay, az, nbrs):
        assert np.all(a[bad] == 0)
