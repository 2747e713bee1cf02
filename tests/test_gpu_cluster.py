"""On-chip refined PCG (csrc/pcg_cluster.cu) against SciPy's sparse LU.

The solve is one thread-block cluster per segment and column group: the sizes
here sit at the edges of its 32-row units, of the units a CTA holds, of the
cluster sizes, and of what fits on chip at all (larger segments take the
persistent PCG); columns at the edges of the column groups."""

from __future__ import annotations

import numpy as np
import pytest
from scipy import sparse
from scipy.sparse.linalg import splu

pytestmark = pytest.mark.gpu

SHIFT = 0.05
RTOL = 1e-11


def _laplacian(edges, n):
    i, j = np.asarray(edges, dtype=np.int64).reshape(-1, 2).T
    w = np.ones(len(i))
    W = sparse.coo_matrix((np.r_[w, w], (np.r_[i, j], np.r_[j, i])), shape=(n, n)).tocsr()
    W.data[:] = 1.0
    K = (sparse.diags(np.asarray(W.sum(1)).ravel() + SHIFT) - W).tocsr()
    K.sort_indices()
    return K


def _grid(n):
    """First n vertices of a square grid with one diagonal per cell (a planar mesh's pattern)."""
    m = max(1, int(np.ceil(np.sqrt(n))))
    v = np.arange(n)
    e = []
    for step in (1, m, m + 1):
        a = v[v + step < n]
        if step != m:
            a = a[a % m != m - 1]
        e.append(np.column_stack((a, a + step)))
    return _laplacian(np.vstack(e) if n > 1 else np.zeros((0, 2)), n)


def _star(n):
    return _laplacian(np.column_stack((np.zeros(n - 1, int), np.arange(1, n))), n)


def _scrambled(n, seed):
    """The grid with its rows in random order: nearly every neighbour lies in another CTA."""
    p = np.random.default_rng(seed).permutation(n)
    K = _grid(n)[p][:, p].tocsr()
    K.sort_indices()
    return K


def _solve(blocks, ncol, seed=0):
    import torch

    from lapy_gb300._device import pcg_solve

    seg = np.concatenate([[0], np.cumsum([b.shape[0] for b in blocks])]).astype(np.int32)
    K = sparse.block_diag(blocks, format="csr")
    K.sort_indices()
    b = np.random.default_rng(seed).standard_normal((K.shape[0], ncol))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data, b)]
    x, relres, iters = pcg_solve(dev[0], dev[1], dev[2], K.shape[0], K.nnz, dev[3], RTOL, seg_row=seg)
    return x.cpu().numpy(), relres, iters, b, seg


def _check(blocks, ncol):
    x, relres, _, b, seg = _solve(blocks, ncol)
    assert np.all(relres <= RTOL)
    for s, K in enumerate(blocks):
        r0, r1 = seg[s], seg[s + 1]
        if r1 == r0:
            continue
        ref = splu(sparse.csc_matrix(K)).solve(b[r0:r1])
        kappa = (2 * np.abs(K.diagonal()).max()) / SHIFT  # Gershgorin over the smallest eigenvalue
        err = np.linalg.norm(x[r0:r1] - ref, axis=0) / np.linalg.norm(ref, axis=0)
        assert np.all(err <= kappa * RTOL), (s, r1 - r0, err)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 511, 512, 513, 1025, 4096, 4097, 16385, 65536, 65537, 70000])
def test_sizes(cuda_ok, n):
    _check([_grid(n)], 1)


@pytest.mark.parametrize("ncol", [1, 2, 3, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("n", [40, 2500])
def test_columns(cuda_ok, n, ncol):
    _check([_grid(n)], ncol)


def test_uneven_segments(cuda_ok):
    """Clusters of every size side by side, a row alone, an empty segment."""
    sizes = [1, 30000, 33, 0, 700, 12000, 64, 5000, 2, 2049, 160, 25000]
    for ncol in (1, 4):
        _check([_grid(n) if n else sparse.csr_matrix((0, 0)) for n in sizes], ncol)


@pytest.mark.parametrize("n", [700, 9000])
def test_far_neighbours_and_wide_rows(cuda_ok, n):
    """Every neighbour in another CTA (halo as large as the mesh); one row of n entries."""
    _check([_scrambled(n, 3), _star(300), _scrambled(n, 4)], 2)


def test_repeatable(cuda_ok):
    blocks = [_grid(n) for n in (9000, 300, 2500)]
    a, b = _solve(blocks, 4), _solve(blocks, 4)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


def test_zero_and_nonfinite_columns(cuda_ok):
    """A zero column is solved by zero; a NaN column is reported, not spread."""
    import torch

    from lapy_gb300 import _lib
    from lapy_gb300._device import pcg_solve

    K = _grid(3000)
    ip, ix, v = (torch.from_numpy(x).cuda() for x in
                 (K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data))
    b = np.random.default_rng(1).standard_normal((3000, 4))
    b[:, 1] = 0.0
    x, relres, _ = pcg_solve(ip, ix, v, 3000, K.nnz, torch.from_numpy(b).cuda(), RTOL)
    assert torch.all(x[:, 1] == 0) and relres[1] == 0.0 and np.all(relres <= RTOL)
    b[17, 2] = np.inf
    with pytest.raises(_lib.LapyGpuError):
        pcg_solve(ip, ix, v, 3000, K.nnz, torch.from_numpy(b).cuda(), RTOL)


@pytest.mark.parametrize("freq_level,block", [(2, 8), (3, 1), (4, 4), (5, 2)])
def test_two_level_eigs(cuda_ok, freq_level, block):
    """The two-level clusters at other block widths: eigenvalues as Jacobi's."""
    from lapy_gb300 import Solver, meshes

    fem = Solver(meshes.sh_deform(meshes.icosphere(freq_level), seed=freq_level), lump=False)
    ev, _ = fem.eigs(k=8, block=block)
    ref, _ = fem.eigs(k=8, block=block, precond="jacobi")
    np.testing.assert_allclose(ev[1:], ref[1:], rtol=1e-8)
    assert abs(ev[0]) <= 1e-8 * ref[1]
