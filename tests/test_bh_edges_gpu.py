"""Centres of mass with more edges between thread blocks than threads (GPU).

com_top_kernel's last CTA takes the edges between CTAs of 32 blocks of 512
bodies: 513 of them, one more than its 512 threads, need 514 CTAs, that is
513 * 16,384 + 1 bodies.
"""
from __future__ import annotations

import pytest

from test_bh_gpu import _bh
from test_bh_nodes_gpu import _check_sums

pytestmark = pytest.mark.gpu


def test_more_edges_than_threads(nb):
    n = 513 * 16384 + 1
    s = nb.ics.uniform_cube(n, seed=9)
    _check_sums(s, _bh(nb, s, theta=2.0, count=False)["nodes"])
