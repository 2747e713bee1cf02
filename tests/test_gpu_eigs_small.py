"""Meshes whose rows a few Lanczos blocks use up: right eigenvalues, or a status
that says so; never wrong ones with status 0."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.linalg import eigh

import oracle
from lapy_gb300 import _lib

pytestmark = pytest.mark.gpu


def _strip(n):
    """A bent strip of n vertices; its eigenvalues are simple."""
    from lapy_gb300 import TriaMesh

    rng = np.random.default_rng(n)
    i = np.arange(n)
    v = np.column_stack((i // 2 + 0.2 * rng.random(n), i % 2 + 0.2 * rng.random(n), 0.3 * rng.random(n)))
    t = np.column_stack((i[:-2], i[1:-1], i[2:]))
    t[1::2] = t[1::2][:, [0, 2, 1]]
    return TriaMesh(v / ((n + 1) // 2), t)


def _want(m, k):
    A, M = oracle.assemble_scipy(np.asarray(m.v, np.float64), m.t)
    return eigh(A.toarray(), M.toarray(), eigvals_only=True, subset_by_index=[0, k - 1])


def _close(got, want):
    return np.all(np.abs(got - want) <= 1.01e-8 * (want + 0.01))  # the solver's tolerance


SIZES = [(k, b, n) for k in (3, 10, 20, 50) for b in (1, 2, 4, 8, 16)
         for n in sorted({k + 2 * b + 1, k + 2 * b + 2, k + 2 * b + 6, 2 * k + 2 * b + 3, (5 * k) // 2 + 2 * b + 1,
                          ((5 * k) // 2 // b + 3) * b})]


@pytest.mark.parametrize("k,block,n", SIZES)
def test_status_and_values(cuda_ok, k, block, n):
    from lapy_gb300 import shapedna

    m = _strip(n)
    evals, _, info = shapedna.BatchedFEM([m]).eigs(k=k, block=block)
    st = int(info["status"][0])
    # blocks that use up the rows exactly reach every tolerance
    assert st == 0 or (st == _lib.ERR_BREAKDOWN and n % block != 0)
    assert info["nbasis"][0] <= n
    if st == 0:
        assert _close(evals.cpu().numpy()[0], _want(m, k))


@pytest.mark.parametrize("k,n", [(3, 11), (10, 27), (10, 36), (10, 41), (20, 37), (20, 59), (50, 67), (50, 119)])
def test_solver_fills_the_blocks(cuda_ok, k, n):
    from lapy_gb300 import Solver

    m = _strip(n)
    for lump in (False, True):
        fem = Solver(m, lump=lump)
        got, X = fem.eigs(k=k)
        M = fem.mass.toarray() if not lump else np.diag(fem.mass.diagonal())
        want = eigh(fem.stiffness.toarray(), M, eigvals_only=True, subset_by_index=[0, k - 1])
        assert _close(got, want) and X.shape == (n, k)
        assert np.abs(X.T @ M @ X - np.eye(k)).max() <= 1e-9


def test_batch_fills_the_blocks_where_needed(cuda_ok):
    from lapy_gb300 import meshes, shapedna

    ms = [_strip(35), meshes.sh_deform(meshes.icosphere(3), seed=4), _strip(28), _strip(90)]
    for got, m in zip(shapedna.compute_shapedna_batch(ms, k=10, block=8), ms):
        assert _close(got["Eigenvalues"], _want(m, 10)) and got["Eigenvectors"].shape == (len(m.v), 10)


@pytest.mark.parametrize("level,k", [(0, 3), (1, 6), (1, 10), (1, 20)])
def test_symmetric_mesh(cuda_ok, level, k):
    """Eigenvalues of up to five copies, and blocks that find a space smaller than they are."""
    from lapy_gb300 import Solver, meshes

    m = meshes.icosphere(level)
    got, _ = Solver(m).eigs(k=k)
    assert _close(got, _want(m, k))


def test_pieces_that_all_have_a_constant(cuda_ok):
    """Twelve disjoint patches: zero is there twelve times, a block finds as many as it has columns."""
    from lapy_gb300 import shapedna
    from test_gpu_coarse_edge import _pieces

    for block in (1, 2, 4, 8):
        evals, _, info = shapedna.BatchedFEM([_pieces()]).eigs(k=block, block=block)
        assert int(info["status"][0]) == 0
        assert np.all(np.abs(evals.cpu().numpy()) <= 1.01e-10)
