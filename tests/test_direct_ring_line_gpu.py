"""Direct sums of 262,144 to 294,912 bodies, where either kernel may be taken (GPU).

The checks of tests/test_direct_large_gpu.py at both sides of the lower line, and
at sizes whose whole waves of the tile-ring kernel leave little or more of the SMs idle.
"""
from __future__ import annotations

import pytest

import test_direct_large_gpu as large

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,eps,comp", [(262144, 0.01, True), (262145, 0.01, False),
                                        (265003, 0.0, True), (270001, 0.01, True),
                                        (275000, 0.01, True), (290001, 0.01, True)])
def test_between_the_lines(nb, orc, n, eps, comp):
    large.test_lines(nb, orc, n, eps, comp)
