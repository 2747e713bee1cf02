"""The profile's timers change no result: same checks, same basis, same bits."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels,k,block", [([5], 50, 8), ([4, 2, 3], 20, 4), ([3] * 12, 30, 2)])
def test_eigenvalues_and_basis(cuda_ok, levels, k, block):
    import torch

    from lapy_gb300 import _lib, meshes, shapedna

    fem = shapedna.BatchedFEM(meshes.deformed_icospheres(levels, range(len(levels))))
    plain, vec, info = fem.eigs(k=k, block=block)
    _lib.profile_enable(True)
    try:
        timed, vec2, info2 = fem.eigs(k=k, block=block)
    finally:
        _lib.profile_enable(False)
        _lib.profile_reset()
    assert np.array_equal(info["nbasis"], info2["nbasis"]) and info["inner_iters"] == info2["inner_iters"]
    assert torch.equal(plain, timed) and torch.equal(vec, vec2)
