"""On-chip PCG on meshes whose neighbours lie in other CTAs: as many copies of
rows as own ones, several times as many, and more than have room for both z and
the direction; at every width of the column groups."""

from __future__ import annotations

import pytest
from test_gpu_cluster import _check, _grid, _scrambled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("n", [5000, 12000, 40000])
def test_scrambled_rows(cuda_ok, n, ncol):
    _check([_scrambled(n, n + ncol)], ncol)


def test_both_forms_side_by_side(cuda_ok):
    """Clusters of different sizes, of few and of many copies, in one solve."""
    _check([_scrambled(30000, 1), _grid(30000), _scrambled(3000, 2), _grid(700), _scrambled(15000, 3)], 2)
