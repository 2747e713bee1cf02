"""Assembly (csrc/assemble.cu) at the edges of its row sort: rows of 32, 64,
128 and more entries, degenerate elements (second numeric pass), output types;
mean edge lengths and weighted sums per mesh (csrc/csr_util.cu) on meshes that
fill their CTAs unevenly.  Whole numbers are exact; values are exact too where
no element is degenerate, as the oracle's local values are summed in the same
order."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import lapy_oracle

pytestmark = pytest.mark.gpu


def _fan(k, npe, seed=0):
    """k elements around one vertex (npe 3) or one edge (npe 4), in random order."""
    rng = np.random.default_rng(seed)
    phi = 2 * np.pi * np.arange(k) / k
    ring = np.c_[np.cos(phi), np.sin(phi), 0.1 * rng.standard_normal(k)]
    hubs = np.array([[0, 0, 0.5], [0, 0, -0.5]])[:npe - 2]
    i = np.arange(k)
    t = np.column_stack([np.full(k, h) for h in range(npe - 2)] + [npe - 2 + i, npe - 2 + (i + 1) % k])
    t = t[rng.permutation(k)]
    return np.r_[hubs, ring], np.ascontiguousarray(np.roll(t, rng.integers(npe), axis=1)).astype(np.int32)


def _reference(v, t, lump, dtype):
    """indptr, indices, values in the order of positions, and the sums of absolute values."""
    npe = t.shape[1]
    la, lm = (lapy_oracle.tria_local if npe == 3 else lapy_oracle.tet_local)(v, t, False)
    if lump:
        b = (lapy_oracle.tria_local if npe == 3 else lapy_oracle.tet_local)(v, t, True)[1]
    i, j = lapy_oracle._pairs(t, npe)
    order = np.lexsort((np.arange(len(i)), j, i))
    keys, at = np.unique(i.astype(np.int64) * len(v) + j, return_inverse=True)
    out = []
    for loc in (la, lm):
        x = loc.reshape(-1).astype(dtype)
        s, w = np.zeros(len(keys), dtype), np.zeros(len(keys))
        np.add.at(s, at[order], x[order])
        np.add.at(w, at[order], np.abs(x[order]))
        out.append((s, w))
    if lump:
        d, w = np.zeros(len(v), dtype), np.zeros(len(v))
        flat, x = t.reshape(-1), b.reshape(-1).astype(dtype)
        np.add.at(d, flat, x)
        np.add.at(w, flat, np.abs(x))
        out[1] = (d, w)
    indptr = np.searchsorted(keys // len(v), np.arange(len(v) + 1))
    return indptr, keys % len(v), out


def _device(v, t, lump, f32):
    import torch

    from lapy_gb300 import _device

    class Mesh:
        pass

    m = Mesh()
    m.v, m.t = v, t
    md, pat = _device.pattern_of(m)
    a, b = _device.assemble(md, pat, lump, torch.float32 if f32 else torch.float64)
    return pat, a.cpu().numpy(), b.cpu().numpy()


@pytest.mark.parametrize("lump,f32", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("npe,k", [(3, 3), (3, 10), (3, 11), (3, 21), (3, 22), (3, 42), (3, 43), (3, 86), (3, 171),
                                   (4, 4), (4, 8), (4, 9), (4, 16), (4, 17), (4, 32), (4, 33), (4, 65)])
def test_rows_at_the_edges_of_the_sort(cuda_ok, npe, k, lump, f32):
    v, t = _fan(k, npe, seed=k)
    ptr, idx, ((a, _), (m, _)) = _reference(v, t, lump, np.float32 if f32 else np.float64)
    pat, ga, gm = _device(v, t, lump, f32)
    np.testing.assert_array_equal(pat.indptr.cpu().numpy(), ptr)
    np.testing.assert_array_equal(pat.indices.cpu().numpy(), idx)
    assert int(pat.seg_ptr[-1]) == t.size * npe
    np.testing.assert_array_equal(ga, a)
    np.testing.assert_array_equal(gm, m)


@pytest.mark.parametrize("npe", [3, 4])
@pytest.mark.parametrize("lump", [False, True])
def test_degenerate_elements(cuda_ok, npe, lump):
    """Elements of no measure take the clamp: 1e-4 of the mean, whose sum may round by one part in 2^53 per element."""
    v, t = _fan(40, npe, seed=5)
    v[npe + 3] = v[npe + 2]  # two neighbours of the ring coincide
    ptr, idx, refs = _reference(v, t, lump, np.float64)
    pat, *got = _device(v, t, lump, False)
    for (want, size), g in zip(refs, got):
        assert np.all(np.abs(g - want) <= (len(t) + 16) * 2.0**-53 * size)


@pytest.mark.parametrize("npe", [3, 4])
def test_elements_that_name_a_vertex_twice(cuda_ok, npe):
    v, t = _fan(30, npe, seed=8)
    t[4, 1] = t[4, 0]
    t[9, 2] = t[9, 0]
    ptr, idx, refs = _reference(v, t, False, np.float64)
    pat, *got = _device(v, t, False, False)
    np.testing.assert_array_equal(pat.indptr.cpu().numpy(), ptr)
    np.testing.assert_array_equal(pat.indices.cpu().numpy(), idx)
    for (want, size), g in zip(refs, got):  # clamped elements as above
        assert np.all(np.abs(g - want) <= (len(t) + 16) * 2.0**-53 * size)


def test_many_rows(cuda_ok):
    """Rows of 6 corners in whole warps and CTAs, and a wide row among narrow ones."""
    from lapy_gb300 import meshes

    m = meshes.icosphere(5)
    v, t = np.asarray(m.v, np.float64), np.asarray(m.t, np.int32)
    fv, ft = _fan(100, 3, seed=2)
    v, t = np.r_[v, fv, v], np.r_[t, ft + len(v), t + len(v) + len(fv)].astype(np.int32)
    ptr, idx, ((a, _), (mm, _)) = _reference(v, t, False, np.float64)
    pat, ga, gm = _device(v, t, False, False)
    np.testing.assert_array_equal(pat.indptr.cpu().numpy(), ptr)
    np.testing.assert_array_equal(pat.indices.cpu().numpy(), idx)
    np.testing.assert_array_equal(ga, a)
    np.testing.assert_array_equal(gm, mm)


def test_out_of_range_index_is_refused(cuda_ok):
    import torch

    from lapy_gb300 import _device

    v, t = _fan(12, 3)
    for bad in (-1, len(v)):
        tb = t.copy()
        tb[7, 1] = bad
        md = _device.MeshDevice(torch.from_numpy(v).cuda(), torch.from_numpy(tb).cuda(), len(v), len(v), len(t), 3)
        with pytest.raises(Exception, match="outside"):
            _device.build_pattern(md)


@pytest.mark.parametrize("f32", [False, True])
def test_edge_lengths_and_sums_per_mesh(cuda_ok, f32):
    """Meshes of 4 to 2,300 rows: fewer rows than CTAs, than threads, and several rows per thread."""
    import torch

    from lapy_gb300 import _lib
    from lapy_gb300._device import dptr, stream

    parts = [_fan(k, 3, seed=k) for k in (3, 7, 255, 2300, 16, 300)]
    seg = np.r_[0, np.cumsum([len(v) for v, _ in parts])].astype(np.int32)
    v = np.concatenate([v for v, _ in parts]).astype(np.float32 if f32 else np.float64)
    t = np.concatenate([t + o for (_, t), o in zip(parts, seg)]).astype(np.int32)
    ptr, idx, ((x, _), (y, _)) = _reference(v.astype(np.float64), t, False, np.float64)
    n, ns = len(v), len(parts)
    dev = {k: torch.from_numpy(np.ascontiguousarray(a)).cuda() for k, a in dict(
        v=v, seg=seg, ptr=ptr.astype(np.int32), idx=idx.astype(np.int32), x=x, y=y, d=np.arange(n) + 0.5,
        al=np.linspace(0.3, 2, ns), be=np.linspace(-1, 1, ns)).items()}
    rows = np.repeat(np.arange(n), np.diff(ptr))
    which = np.searchsorted(seg, rows, side="right") - 1
    L = _lib.lib()
    mean, t2 = (torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(2))
    _lib.check(L.lapy_seg_avg_edge_length(dptr(dev["v"]), int(f32), ns, dptr(dev["seg"]), dptr(dev["ptr"]),
                                          dptr(dev["idx"]), 2.0, dptr(mean), dptr(t2), stream()), "edge")
    up = rows < idx
    length = np.linalg.norm(v[rows[up]] - v[idx[up]], axis=1)
    want = np.bincount(which[up], length.astype(np.float64)) / np.bincount(which[up])
    # a length rounds five times in the coordinate type, a sum of m lengths in 64 bits m times
    tol = 8 * (2.0**-24 if f32 else 2.0**-53) + 7000 * 2.0**-53
    np.testing.assert_allclose(mean.cpu().numpy(), want, rtol=tol, atol=0)
    np.testing.assert_array_equal(t2.cpu().numpy(), 2.0 * (mean * mean).cpu().numpy())

    out = torch.empty_like(dev["x"])
    diag = np.searchsorted(rows * n + idx, np.arange(n) * (n + 1))
    ddiag = torch.from_numpy(diag.astype(np.int32)).cuda()
    al, be = dev["al"].cpu().numpy()[which], dev["be"].cpu().numpy()[which]
    for y_is_diag in (0, 1):
        _lib.check(L.lapy_csr_seg_axpby(ns, dptr(dev["seg"]), dptr(dev["ptr"]), dptr(ddiag), dptr(dev["al"]),
                                        dptr(dev["x"]), dptr(dev["be"]), dptr(dev["d" if y_is_diag else "y"]),
                                        y_is_diag, dptr(out), stream()), "axpby")
        ref = al * x
        if y_is_diag:
            ref[diag] = ref[diag] + be[diag] * (np.arange(n) + 0.5)
        else:
            ref = ref + be * y
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
