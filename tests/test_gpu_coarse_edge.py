"""Two-level eigensolves of a batch in which a mesh has no coarse space: its many
small pieces would make more aggregates than the solver keeps."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.linalg import eigh

import oracle

pytestmark = pytest.mark.gpu

PIECES = 12


def _pieces():
    """Disjoint nine-vertex patches of different sizes."""
    from lapy_gb300 import TriaMesh, meshes

    g = meshes.square_grid(2)
    v = np.vstack([np.asarray(g.v) * (1 + 0.1 * i) + [3.0 * i, 0, 0] for i in range(PIECES)])
    t = np.vstack([np.asarray(g.t) + len(g.v) * i for i in range(PIECES)])
    return TriaMesh(v, t)


@pytest.mark.parametrize("order", [(1, 0), (0,)])
@pytest.mark.parametrize("block", [4, 8])
def test_mesh_without_aggregates(cuda_ok, monkeypatch, order, block):
    """Whatever the workspace held before (here NaN in every float)."""
    import torch

    from lapy_gb300 import meshes, shapedna, solver

    monkeypatch.setattr(solver, "workspace",
                        lambda n: torch.full((max(int(n), 256),), 255, dtype=torch.uint8, device="cuda"))
    ms = [(_pieces(), meshes.sh_deform(meshes.icosphere(3), seed=4))[i] for i in order]
    k = block  # the pieces' constants: a block finds as many of them as it has columns
    evals, _, info = shapedna.BatchedFEM(ms).eigs(k=k, block=block)
    assert not np.any(np.asarray(info["status"]))
    for got, m in zip(evals.cpu().numpy(), ms):
        A, M = oracle.assemble_scipy(np.asarray(m.v, np.float64), m.t)
        want = eigh(A.toarray(), M.toarray(), eigvals_only=True, subset_by_index=[0, k - 1])
        assert np.all(np.abs(got - want) <= 1.01e-8 * (want + 0.01))  # the solver's tolerance


@pytest.mark.parametrize("order", [(0, 1), (1, 0, 1), (0, 0, 1), (0, 1, 0, 1)])
@pytest.mark.parametrize("block", [1, 4, 8])
def test_mesh_without_aggregates_first(cuda_ok, order, block):
    """Aggregates after rows that belong to none."""
    from lapy_gb300 import meshes, shapedna

    ms = [(_pieces(), meshes.sh_deform(meshes.icosphere(3), seed=4))[i] for i in order]
    evals, evecs, info = shapedna.BatchedFEM(ms).eigs(k=block, block=block)
    assert not np.any(np.asarray(info["status"]))
    for got, m in zip(evals.cpu().numpy(), ms):
        A, M = oracle.assemble_scipy(np.asarray(m.v, np.float64), m.t)
        want = eigh(A.toarray(), M.toarray(), eigvals_only=True, subset_by_index=[0, block - 1])
        assert np.all(np.abs(got - want) <= 1.01e-8 * (want + 0.01))


def test_mesh_without_aggregates_beside_a_large_one(cuda_ok):
    """68,121 rows do not fit on chip: the grid-wide solver with the same aggregates."""
    from scipy.sparse.linalg import eigsh

    from lapy_gb300 import TriaMesh, meshes, shapedna

    grid = meshes.square_grid(260)
    ms = [_pieces(), TriaMesh(grid.v * 10, grid.t)]
    evals, _, info = shapedna.BatchedFEM(ms).eigs(k=4, block=4)
    assert not np.any(np.asarray(info["status"]))
    A, M = oracle.assemble_scipy(np.asarray(ms[1].v, np.float64), ms[1].t)
    want = np.sort(eigsh(A, k=4, M=M, sigma=-0.01, tol=0, return_eigenvectors=False))
    assert np.all(np.abs(evals.cpu().numpy()[1] - want) <= 1.01e-8 * (want + 0.01))
