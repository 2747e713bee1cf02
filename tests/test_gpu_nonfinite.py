"""Right-hand sides with NaN or Inf: the column is reported, its solution is zero,
and the other columns and meshes of the same solve come out as without it."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
from scipy import sparse

from lapy_gb300 import _lib
from test_gpu_cluster import _grid

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _solve(blocks, b, mixed=1, ic0=False):
    """Solution, status and relative residual of every mesh and column."""
    import torch

    from lapy_gb300._device import dptr, stream, workspace

    L = _lib.lib()
    seg = np.concatenate([[0], np.cumsum([x.shape[0] for x in blocks])]).astype(np.int32)
    K = sparse.block_diag(blocks, format="csr")
    K.sort_indices()
    n, ncol, nseg = K.shape[0], b.shape[1], len(blocks)
    ip, ix, kv, rhs = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
                       (K.indptr.astype(np.int32), K.indices.astype(np.int32), K.data, b))
    x = torch.full((n, ncol), 7.0, dtype=torch.float64, device="cuda")
    status, relres, iters = np.zeros((nseg, ncol), np.int32), np.zeros((nseg, ncol)), C.c_int64(0)
    head = (n, dptr(ip), dptr(ix), dptr(kv), K.nnz, nseg, seg.ctypes.data, ncol, dptr(rhs), dptr(x), RTOL, 20000)
    if ic0:
        ws = workspace(L.lapy_ic0_pcg_workspace_bytes(n, K.nnz, nseg, seg.ctypes.data, ncol))
        fixed = C.c_int32(0)
        st = L.lapy_ic0_pcg_solve(*head, 1e-4, status.ctypes.data, relres.ctypes.data, C.byref(iters), C.byref(fixed),
                                  dptr(ws), ws.numel(), stream())
    else:
        ws = workspace(L.lapy_pcg_solve_workspace_bytes(n, K.nnz, nseg, seg.ctypes.data, ncol, mixed))
        st = L.lapy_pcg_solve(*head, mixed, 1e-4, status.ctypes.data, relres.ctypes.data, C.byref(iters), dptr(ws),
                              ws.numel(), stream())
    assert st == 0
    return x.cpu().numpy(), status, relres, seg


@pytest.mark.parametrize("sizes,how", [((300,), "mixed"), ((9000,), "mixed"), ((300, 9000, 40), "mixed"),
                                       ((66000, 300), "mixed"), ((300, 9000), "ic0"), ((300, 9000), "f64")])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_column_is_reported_and_not_spread(cuda_ok, sizes, how, value):
    """On one CTA, on a cluster, on several of them, on the whole GPU; IC(0); FP64."""
    blocks = [_grid(n) for n in sizes]
    kw = {"mixed": {}, "ic0": {"ic0": True}, "f64": {"mixed": 0}}[how]
    b = np.random.default_rng(5).standard_normal((sum(sizes), 4))
    b[:, 3] = 0.0
    ref, _, _, seg = _solve(blocks, b, **kw)
    last = len(sizes) - 1
    b[seg[last] + 17, 1] = value  # one entry of one column of the last mesh
    x, status, relres, _ = _solve(blocks, b, **kw)
    want = np.zeros_like(status)
    want[last, 1] = _lib.ERR_NAN
    assert np.array_equal(status, want)
    assert np.isnan(relres[last, 1])
    good = want == 0
    assert np.all(relres[good] <= RTOL)
    for s in range(len(sizes)):
        for c in range(4):
            got = x[seg[s]:seg[s + 1], c]
            if not good[s, c]:
                assert how == "f64" or np.all(got == 0)
                continue
            # both within RTOL of ||b|| in the residual; the smallest eigenvalue is 0.05
            bound = 2 * RTOL * np.linalg.norm(b[seg[s]:seg[s + 1], c]) / 0.05
            assert np.linalg.norm(got - ref[seg[s]:seg[s + 1], c]) <= bound
