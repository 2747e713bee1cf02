"""Block Lanczos at the edges of its kernels' ranges: the dense eigensolver's
row lengths (up to 128, 256, 384 and beyond), the coarse inverse around 16
aggregates and in ragged blocks of 32, and every block size of the Gram-Schmidt
products, against ARPACK in shift-invert mode."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.sparse.linalg import eigsh

import oracle

pytestmark = pytest.mark.gpu

SIGMA = -0.01
TOL = 1e-8  # default tolerance of the residual relative to the shift-inverted value


def _reference(v, t, k):
    A, M = oracle.assemble_scipy(v, t)
    return np.sort(eigsh(A, k=k, M=M, sigma=SIGMA, tol=0, return_eigenvectors=False))


def _close(got, want):
    """A residual of TOL theta moves the shift-inverted value theta = 1 / (lambda - sigma) by TOL theta at most."""
    assert np.all(np.abs(got - want) <= 1.01 * TOL * (want - SIGMA))


@pytest.mark.parametrize("k,block", [(8, 8), (12, 1), (25, 2), (45, 4), (75, 8), (110, 8)])
def test_basis_sizes(cuda_ok, k, block):
    from lapy_gb300 import meshes, shapedna

    m = meshes.sh_deform(meshes.icosphere(3), seed=4)
    got = shapedna.BatchedFEM([m]).eigs(k=k, block=block)[0]
    _close(got.cpu().numpy().reshape(-1)[:k], _reference(m.v, m.t, k))


@pytest.mark.parametrize("sizes,block", [((31,), 4), ((32,), 2), ((33,), 1), ((45,), 4), ((46,), 8), ((52,), 4),
                                         ((9, 46, 31, 34), 4),
                                         pytest.param((5, 33), 8, marks=pytest.mark.xfail(strict=True, reason=
                                             "36 rows hold 4.5 blocks: a rank-deficient block is taken as converged"))])
def test_coarse_sizes(cuda_ok, sizes, block):
    from lapy_gb300 import meshes, shapedna

    ms = [meshes.square_grid(n) for n in sizes]
    got = shapedna.BatchedFEM(ms).eigs(k=10, block=block)[0]
    for g, m in zip(got.cpu().numpy().reshape(len(ms), -1), ms):
        _close(g[:10], _reference(np.asarray(m.v, np.float64), m.t, 10))


@pytest.mark.parametrize("sizes,block", [((5,), 2), ((5,), 4), ((6,), 4), ((7,), 4), ((7,), 8), ((5, 33), 2),
                                         ((5, 33), 4), ((33, 5), 4), ((9, 33), 4), ((7, 33), 8)])
def test_basis_that_fills_a_mesh(cuda_ok, sizes, block):
    """36 to 100 rows: convergence comes with, or shortly before, the last block that fits."""
    from lapy_gb300 import meshes, shapedna

    ms = [meshes.square_grid(n) for n in sizes]
    evals, _, info = shapedna.BatchedFEM(ms).eigs(k=8, block=block)
    assert not np.any(np.asarray(info["status"]))
    for g, m in zip(evals.cpu().numpy().reshape(len(ms), -1), ms):
        _close(g[:8], _reference(np.asarray(m.v, np.float64), m.t, 8))
