"""Small meshes in coarse units: A - sigma M close to singular in FP32, where the
inner solve is as good as the recurrences of its conjugate gradients.

``K = A + 0.01 M`` of a sphere of radius r has its constant mode at 0.005 r^2 of
the next one: 5e-6 at r = 0.03, where a scalar product that comes out of a
difference keeps two digits of FP32's seven."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.linalg import eigh

import oracle

pytestmark = pytest.mark.gpu

RTOL, INNER = 1e-9, 1e-3
RADII = [0.03, 0.1, 1.0]
MESHES = [(3, 4), (3, 5), (4, 6)]  # icosphere level, seed of its deformation


def _mesh(level, seed, radius):
    from lapy_gb300 import TriaMesh, meshes

    base = meshes.sh_deform(meshes.icosphere(level), seed=seed)
    return TriaMesh(base.v * radius, base.t)


def _plain_cg_iterations(K, b):
    """Jacobi-preconditioned CG in FP32 inside FP64 refinement, as textbooks have it."""
    K32, dinv = K.astype(np.float32), (1 / K.diagonal()).astype(np.float32)
    x, r, total, reduce_by = np.zeros(len(b)), b.copy(), 0, INNER
    for _ in range(12):
        d, res, p = (np.zeros(len(b), np.float32), r.astype(np.float32), np.zeros(len(b), np.float32))
        goal, rz = np.float32(reduce_by**2) * (res @ res), None
        while res @ res > goal:
            z = dinv * res
            new = res @ z
            p = z if rz is None else z + (new / rz) * p
            q, rz = K32 @ p, new
            alpha = rz / (p @ q)
            d, res, total = d + alpha * p, res - alpha * q, total + 1
        x += d
        r = b - K @ x
        if np.linalg.norm(r) <= RTOL * np.linalg.norm(b):
            return total
        reduce_by = max(INNER, min(0.5, 0.25 * RTOL * np.linalg.norm(b) / np.linalg.norm(r)))
    raise AssertionError("the plain iteration does not converge")


@pytest.mark.parametrize("radius", RADII)
@pytest.mark.parametrize("level,seed", MESHES)
def test_iterations_of_plain_cg(cuda_ok, level, seed, radius):
    """Rounding moves the count; twice the plain iteration's is far beyond it."""
    import torch

    from lapy_gb300._device import pcg_solve

    m = _mesh(level, seed, radius)
    A, M = oracle.assemble_scipy(m.v, m.t)
    K = (A + 0.01 * M).tocsr()
    K.sort_indices()
    b = M @ np.random.default_rng(seed).standard_normal((K.shape[0], 2))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data, b)]
    for cols in (1, 2):
        _, relres, iters = pcg_solve(dev[0], dev[1], dev[2], K.shape[0], K.nnz, dev[3][:, :cols].contiguous(), RTOL,
                                     inner_rtol=INNER)
        assert np.all(relres <= RTOL)
        assert iters <= 2 * max(_plain_cg_iterations(K, b[:, c]) for c in range(cols))


@pytest.mark.parametrize("precond", ["jacobi", "twolevel"])
@pytest.mark.parametrize("radius", RADII)
@pytest.mark.parametrize("level,seed", MESHES)
def test_eigenvalues(cuda_ok, level, seed, radius, precond):
    """The solver's tolerance on the shift-inverted values: 1e-8 (lambda - sigma)."""
    from lapy_gb300 import Solver

    m = _mesh(level, seed, radius)
    A, M = oracle.assemble_scipy(m.v, m.t)
    want = eigh(A.toarray(), M.toarray(), eigvals_only=True, subset_by_index=[0, 19])
    got, _ = Solver(m).eigs(k=20, precond=precond)
    # the constant mode: 1e-8 of the next eigenvalue, as rounding of A leaves it
    assert abs(got[0]) <= 1e-8 * want[1]
    assert np.all(np.abs(got[1:] - want[1:]) <= 1.01e-8 * (want[1:] + 0.01))
