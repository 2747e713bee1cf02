"""The work this framework is measured on: spectra, heat solves, geodesics,
assembly, the inner SpMM and the training pass of the learned preconditioner,
through the public entry points and over the sizes its configurations cover.

A case is a dict of plain values.  ``prepare`` makes what a user's program has
in hand (host meshes, a device batch, a matrix copy), ``run`` is one pass and
``exact`` the same outputs from dense or conjugate-gradient torch arithmetic in
64 bits, without this package's code.

Surfaces are closed star-shaped spheres with random smooth radii: a geodesic
polyhedron of frequency f has 10 f^2 + 2 vertices (f = 8, 16, 32, 64 are
icosphere levels 3 to 6), so sizes need not be powers of two.  Solids
are boxes of jittered cells cut into six tetrahedra each.
"""

from __future__ import annotations

import functools
import itertools
import math
from pathlib import Path

import numpy as np
import torch

import lapy_gb300
from lapy_gb300 import Solver, TetMesh, TriaMesh, diffgeo, heat, shapedna, spai
from lapy_gb300._device import SellF32

# Each spectrum's heat kernel signature is taken at these multiples of the
# usual smallest time 4 ln(10) / lambda_k.
HKS_TIMES = (1.0, 4.0, 16.0, 64.0)


def listed():
    return [
        # one small surface, the default number of eigenpairs: the smallest spectrum, launches and latency
        dict(name="eigs-sphere-642", kind="eigs", mesh="sphere", size=8, k=10),
        # one 10,242-vertex surface, k = 50: the usual ShapeDNA call for a single subject
        dict(name="eigs-sphere-10242", kind="eigs", mesh="sphere", size=32, k=50),
        # a tetrahedral solid of odd size, k = 50
        dict(name="eigs-tets-11466", kind="eigs", mesh="tets", size=20, k=50),
        # a small study from host arrays: upload, assembly and spectra of 24 uneven meshes
        dict(name="shapedna-24", kind="shapedna", count=24, low=8, high=64, k=50),
        # a larger study whose meshes already lie on the device
        dict(name="spectra-128", kind="spectra", count=128, low=8, high=64, k=50),
        # one backward-Euler step on one float32 surface (FreeSurfer meshes are float32)
        dict(name="heat-sphere-2562", kind="heat", mesh="sphere", size=16, seeds=1, m=1.0, dtype="float32"),
        # heat from several seed sets on a solid, one solve for all of them
        dict(name="heat-tets-44649-x8", kind="heat", mesh="tets", size=32, seeds=8, m=10.0, dtype="float64"),
        # one heat step on each of many meshes on the device: assembly, time steps and the batched solve
        dict(name="heat-batch-256", kind="heat-batch", count=256, low=8, high=64, precond="jacobi"),
        # geodesic distance from a heat solution on one surface: gradient, divergence, Poisson
        dict(name="geodesic-40962", kind="geodesic", size=64),
        # the matrices of a batch of surfaces: CSR pattern, stiffness, consistent mass
        dict(name="assemble-128", kind="assemble", count=128, low=8, high=64, lump=False),
        # the eigensolver's FP32 product, four columns (a Lanczos block)
        dict(name="spmm-256-x4", kind="spmm", count=256, low=8, high=64, columns=4),
        # one gradient of the learned preconditioner over a batch of heat systems
        dict(name="train-12", kind="train", count=12, low=16, high=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eigs", "eigs", "shapedna", "spectra", "heat", "heat", "heat-batch", "geodesic", "assemble",
                       "spmm", "train"])
    if kind == "eigs":
        mesh = rng.choice(["sphere", "tets"])
        size = _log(rng, 8, 48) if mesh == "sphere" else _log(rng, 7, 24)
        return dict(kind=kind, mesh=mesh, size=size, k=rng.choice([10, 20, 30, 50, 60]))
    if kind == "heat":
        mesh = rng.choice(["sphere", "tets"])
        size = _log(rng, 8, 200) if mesh == "sphere" else _log(rng, 7, 36)
        return dict(kind=kind, mesh=mesh, size=size, seeds=rng.randint(1, 8), m=rng.choice([0.5, 1.0, 3.0, 10.0]),
                    dtype=rng.choice(["float32", "float64"]))
    if kind == "geodesic":
        return dict(kind=kind, size=_log(rng, 12, 64))
    low = _log(rng, 8, 20)
    high = _log(rng, low + 4, 64)
    if kind == "shapedna":
        return dict(kind=kind, count=_log(rng, 4, 32), low=low, high=high, k=rng.choice([20, 30, 50]))
    if kind == "spectra":
        return dict(kind=kind, count=_log(rng, 16, 128), low=low, high=high, k=rng.choice([20, 30, 50]))
    if kind == "heat-batch":
        return dict(kind=kind, count=_log(rng, 8, 256), low=low, high=high,
                    precond=rng.choice(["jacobi", "jacobi", "learned"]))
    if kind == "assemble":
        return dict(kind=kind, count=_log(rng, 1, 128), low=low, high=high, lump=rng.random() < 0.5)
    if kind == "spmm":
        return dict(kind=kind, count=_log(rng, 16, 256), low=low, high=high, columns=rng.choice([1, 2, 4, 8]))
    return dict(kind="train", count=_log(rng, 2, 24), low=16, high=rng.randint(24, 48))


# ---------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(f):
    """Geodesic polyhedron of frequency f: unit vertices and outward triangles."""
    phi = (1 + math.sqrt(5)) / 2
    base = np.array([p for a, b in itertools.product((-1, 1), repeat=2)
                     for p in ((0, a, b * phi), (a, b * phi, 0), (b * phi, 0, a))], dtype=np.float64)
    faces = []
    for i, j, k in itertools.combinations(range(12), 3):
        if all(abs(np.sum((base[p] - base[q]) ** 2) - 4) < 1e-6 for p, q in ((i, j), (j, k), (i, k))):
            out = np.cross(base[j] - base[i], base[k] - base[i]) @ (base[i] + base[j] + base[k]) > 0
            faces.append((i, j, k) if out else (i, k, j))
    a, b = np.array([(a, b) for a in range(f + 1) for b in range(f + 1 - a)]).T
    at = np.full((f + 2, f + 2), -1)
    at[a, b] = np.arange(len(a))
    up = np.array([(at[i, j], at[i + 1, j], at[i, j + 1]) for i in range(f) for j in range(f - i)])
    dn = [(at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]) for i in range(f) for j in range(f - i - 1)]
    local = np.vstack([up, np.array(dn, dtype=up.dtype).reshape(-1, 3)])
    pts, tri = [], []
    for n, (i, j, k) in enumerate(faces):
        pts.append(((f - a - b)[:, None] * base[i] + a[:, None] * base[j] + b[:, None] * base[k]) / f)
        tri.append(local + n * len(a))
    pts, tri = np.vstack(pts), np.vstack(tri)
    # the faces' copies of a shared vertex differ in the last bits only: 21 bits per coordinate tell vertices apart
    q = np.floor(pts * 2.0**19 + 0.37).astype(np.int64) + 2**20
    _, first, inv = np.unique((q[:, 0] << 42) | (q[:, 1] << 21) | q[:, 2], return_index=True, return_inverse=True)
    order = np.argsort(first)  # vertices numbered as they first occur
    rank = np.empty(len(first), dtype=np.int64)
    rank[order] = np.arange(len(first))
    v = pts[first[order]]
    return v / np.linalg.norm(v, axis=1, keepdims=True), rank[inv][tri].astype(np.int32)


def _surface(f, rng):
    """A sphere of frequency f with a smooth random radius (float64 host arrays)."""
    u, t = _sphere(f)
    w = rng.standard_normal((12, 3)) * rng.uniform(0.5, 3.0, (12, 1))
    c, ph = rng.standard_normal(12) * 0.04, rng.uniform(0, 2 * np.pi, 12)
    ud, wd, cd, pd = (torch.from_numpy(x).cuda() for x in (u, w, c, ph))
    r = 1.0 + torch.cos(ud @ wd.T + pd) @ cd
    return (ud * r[:, None]).cpu().numpy(), t


def _solid(n, rng):
    """A box of n x n x (n + n // 4) jittered cells, six tetrahedra each (a box: no symmetric spectrum)."""
    nx, ny, nz = n, n, n + n // 4
    g = np.stack(np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), np.arange(nz + 1), indexing="ij"), -1)
    inner = np.all((g > 0) & (g < (nx, ny, nz)), axis=-1)
    v = (g + rng.uniform(-0.2, 0.2, g.shape) * inner[..., None]).reshape(-1, 3) / (nx, 1.1 * ny, nz)
    step = np.array([(ny + 1) * (nz + 1), nz + 1, 1])
    base = (np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1) @ step).ravel()
    tets = []
    for p in itertools.permutations(range(3)):
        b, c = base + step[p[0]], base + step[p[0]] + step[p[1]]
        d = base + step.sum()
        even = p in ((0, 1, 2), (1, 2, 0), (2, 0, 1))
        tets.append(np.column_stack((base, b, c, d) if even else (base, c, b, d)))
    return v, np.stack(tets, 1).reshape(-1, 4).astype(np.int32)


def _mesh(case, rng):
    v, t = (_surface if case.get("mesh", "sphere") == "sphere" else _solid)(case["size"], rng)
    return v.astype(case.get("dtype", "float64")), t


def _batch(case, rng):
    """Uneven meshes: frequencies spread over the logarithm of the range, in random order."""
    n, lo, hi = case["count"], case["low"], case["high"]
    f = np.round(np.exp(np.linspace(math.log(lo), math.log(hi), n))).astype(int) if n > 1 else np.array([hi])
    return [_surface(int(x), rng) for x in rng.permutation(f)]


def _sizes(case):
    """(vertices, elements, matrix entries, coordinate bytes) of a case's meshes together."""
    if "count" in case:
        n, lo, hi = case["count"], case["low"], case["high"]
        f = np.round(np.exp(np.linspace(math.log(lo), math.log(hi), n))).astype(int) if n > 1 else np.array([hi])
        nv, ne = int(np.sum(10 * f * f + 2)), int(np.sum(20 * f * f))
    elif case.get("mesh", "sphere") == "sphere":
        nv, ne = 10 * case["size"] ** 2 + 2, 20 * case["size"] ** 2
    else:
        a, b = case["size"], case["size"] + case["size"] // 4
        nv, ne = (a + 1) ** 2 * (b + 1), 6 * a * a * b
        # edges of the Kuhn subdivision: the 7 monotone directions of every cell
        e = sum((a + 1 - i) * (a + 1 - j) * (b + 1 - k) for i, j, k in itertools.product((0, 1), repeat=3)
                if i + j + k)
        return nv, ne, nv + 2 * e, 8
    return nv, ne, nv + 3 * ne, 4 if case.get("dtype") == "float32" else 8


def _rng(case, seed):
    return np.random.default_rng([int(seed), len(case["kind"]), case.get("size", 0), case.get("count", 0)])


def _seeds(case, n, rng):
    """Seed sets of a heat call: one vertex, or several sets of one to four vertices."""
    if case["seeds"] == 1:
        return int(rng.integers(n))
    return [rng.choice(n, size=1 + i % 4, replace=False).tolist() for i in range(case["seeds"])]


def _distance_like(v, rng):
    """A function like a heat solution's: positive, falling exponentially with the angle from a source."""
    u = v / np.linalg.norm(v, axis=1, keepdims=True)
    s = rng.standard_normal(3)
    return np.exp(-5.0 * np.arccos(np.clip(u @ (s / np.linalg.norm(s)), -1, 1)))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    rng, kind = _rng(case, seed), case["kind"]
    s = {"case": dict(case)}
    if kind in ("eigs", "heat", "geodesic"):
        s["v"], s["t"] = _mesh(case, rng)
        if kind == "heat":
            s["vids"] = _seeds(case, len(s["v"]), rng)
        if kind == "geodesic":
            s["f"] = _distance_like(s["v"], rng)
        return s
    meshes = [TriaMesh(v, t) for v, t in _batch(case, rng)]
    if kind == "shapedna":
        s["meshes"] = meshes
        return s
    inp = shapedna.BatchInput(meshes)
    if kind == "spmm":
        fem = shapedna.BatchedFEM.from_input(inp)
        s["sell"] = SellF32(fem.indptr, fem.indices, fem.a_vals, fem.n, fem.nnz, seg_row=inp.seg_row)
        x = rng.standard_normal((fem.n, case["columns"]), dtype=np.float32)
        s["x"] = torch.from_numpy(x).cuda()
        s["y"] = torch.empty_like(s["x"])
    elif kind == "heat-batch":
        s["batch"] = heat.HeatBatch(inp, 0)
    elif kind == "train":
        s["systems"] = spai.SpaiSystems(inp, "heat", t=_times(case, rng))
        s["net"] = spai.SpaiNet.load()
    else:
        s["input"] = inp
    return s


def _times(case, rng):
    """Heat times of the training systems: log-uniform in [1e-4, 1e-1]."""
    return 10.0 ** rng.uniform(-4, -1, case["count"])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "eigs":
        # spectrum and heat kernel signature (float32 features); the eigenvectors themselves are fixed only up to sign
        mesh = (TriaMesh if s["t"].shape[1] == 3 else TetMesh)(s["v"], s["t"])
        k = case["k"]
        evals, evecs = Solver(mesh).eigs(k=k)
        t = 4 * math.log(10) / evals[-1] * np.array([HKS_TIMES])
        hks = heat.diagonal(t, np.arange(len(s["v"])), evecs, evals[:, None], k)
        return evals, hks.astype(np.float32)
    if kind == "shapedna":
        out = shapedna.compute_shapedna_batch(s["meshes"], k=case["k"], block=4, return_vectors=False)
        return [d["Eigenvalues"] for d in out]
    if kind == "spectra":
        return shapedna.BatchedFEM.from_input(s["input"]).eigs(k=case["k"], block=4)[0]
    if kind == "heat":
        mesh = (TriaMesh if s["t"].shape[1] == 3 else TetMesh)(s["v"], s["t"])
        return heat.diffusion(mesh, s["vids"], m=case["m"])
    if kind == "heat-batch":
        u, info = s["batch"].solve(precond=case["precond"])
        return u, info["t"]
    if kind == "geodesic":
        return diffgeo.compute_geodesic_f(TriaMesh(s["v"], s["t"]), s["f"])
    if kind == "assemble":
        fem = shapedna.BatchedFEM.from_input(s["input"], lump=case["lump"])
        return fem.indptr, fem.indices, fem.a_vals, fem.m_vals
    if kind == "spmm":
        return s["sell"].spmm(s["x"], s["y"])
    w = s["net"].forward(s["systems"].feat)
    g, _, logq, dldw = s["systems"].factor(w, grad=True)
    return g, logq, s["net"].backward(s["systems"].feat, dldw, 1.0 / s["systems"].n)


def work(case):
    nv, ne, nnz, cb = _sizes(case)
    kind = case["kind"]
    npe = 4 if case.get("mesh") == "tets" else 3
    mesh = nv * 3 * cb + ne * npe * 4
    local = ne * (60 if npe == 3 else 200)  # one element's matrices
    if kind in ("eigs", "shapedna", "spectra"):
        # the mesh in, eigenvalues and eigenvectors out; 2 k products with the matrix and one orthogonalisation
        # of 2 k vectors, the least that a Krylov method of k pairs does
        k = case["k"]
        return dict(bytes=mesh + 8 * nv * k, flops=local + 2 * k * (2 * nnz + 4 * k * nv))
    if kind == "heat":
        c = case["seeds"]
        return dict(bytes=mesh + 8 * nv * c, flops=local + 4 * nnz * c)
    if kind == "heat-batch":
        return dict(bytes=mesh + 16 * nv, flops=local + 4 * nnz)
    if kind == "geodesic":
        return dict(bytes=mesh + 16 * nv, flops=local + 4 * nnz)
    if kind == "assemble":
        return dict(bytes=mesh + 4 * nv + 4 * nnz + 8 * nnz + (8 * nv if case["lump"] else 8 * nnz), flops=local)
    if kind == "spmm":
        return dict(bytes=8 * nnz + 8 * nv * case["columns"], flops=2 * nnz * case["columns"])
    m = (nnz + nv) // 2
    return dict(bytes=m * (24 + 4) + 8 * nnz + 8 * nv, flops=3 * 2 * m * (6 * 64 + 64 * 64 + 64))


# ---------------------------------------------------------------------------
# 64-bit values of the same outputs
# ---------------------------------------------------------------------------
def _elements(v, t):
    """Element stiffness and mass matrices (float64 torch, on the GPU)."""
    v, t = torch.from_numpy(np.asarray(v, dtype=np.float64)).cuda(), torch.from_numpy(np.asarray(t)).cuda().long()
    p = v[t]
    if t.shape[1] == 3:
        e = p[:, [2, 0, 1]] - p[:, [1, 2, 0]]  # the edge opposite each corner
        area = torch.linalg.norm(torch.linalg.cross(e[:, 0], e[:, 1]), dim=1) / 2
        a = e @ e.mT / (4 * area)[:, None, None]
        m = (torch.ones(3, 3, device="cuda", dtype=v.dtype) + torch.eye(3, device="cuda", dtype=v.dtype)) / 12
    else:
        d = p[:, 1:] - p[:, :1]
        area = torch.linalg.det(d).abs() / 6
        g = torch.linalg.inv(d).mT
        g = torch.cat([-g.sum(1, keepdim=True), g], 1)
        a = g @ g.mT * area[:, None, None]
        m = (torch.ones(4, 4, device="cuda", dtype=v.dtype) + torch.eye(4, device="cuda", dtype=v.dtype)) / 20
    return v, t, a, m * area[:, None, None]


def _matrices(v, t, lump):
    """(row starts, columns, stiffness, mass or its lumped diagonal): entries of a row by column."""
    v, t, a, m = _elements(v, t)
    n, k = len(v), t.shape[1]
    rows, cols = t[:, :, None].expand(-1, k, k).reshape(-1), t[:, None, :].expand(-1, k, k).reshape(-1)
    key, inv = torch.unique(rows * n + cols, return_inverse=True)
    A = torch.zeros(len(key), dtype=torch.float64, device="cuda").index_add_(0, inv, a.reshape(-1))
    M = torch.zeros(n if lump else len(key), dtype=torch.float64, device="cuda")
    M.index_add_(0, rows if lump else inv, m.reshape(-1))
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
    return ptr, key % n, A, M


def _csr(ptr, col, val):
    n = len(ptr) - 1
    return torch.sparse_csr_tensor(ptr, col, val, size=(n, n))


def _rows(ptr):
    return torch.repeat_interleave(torch.arange(len(ptr) - 1, device="cuda"), ptr[1:] - ptr[:-1])


def _cg(ptr, col, val, b, constants=False, tol=1e-15, most=6000):
    """Jacobi CG on every column of b to the last digits; `constants`: the matrix's kernel, kept out of the residual."""
    K, rows = _csr(ptr, col, val), _rows(ptr)
    d = torch.zeros(len(ptr) - 1, dtype=torch.float64, device="cuda")
    d[rows[rows == col]] = val[rows == col]
    x, r = torch.zeros_like(b), b.clone()
    z = r / d[:, None]
    p, rz, bn = z.clone(), (r * z).sum(0), torch.linalg.norm(b, dim=0)
    for i in range(most):
        q = K @ p
        al = rz / (p * q).sum(0)
        x, r = x + al * p, r - al * q
        if constants:
            r = r - r.mean(0)
        if i % 20 == 0 and bool((torch.linalg.norm(r, dim=0) <= tol * bn).all()):
            break
        z = r / d[:, None]
        new = (r * z).sum(0)
        p, rz = z + new / rz * p, new
    return x


def _spectrum(v, t, k, seed=0):
    """The k smallest eigenpairs by block inverse iteration with a dense Cholesky factor."""
    ptr, col, A, M = _matrices(v, t, False)
    n = len(ptr) - 1
    Ms, sigma = _csr(ptr, col, M), -0.01
    K = _csr(ptr, col, A - sigma * M).to_dense()
    L = torch.linalg.cholesky(K)
    del K
    b = min(n - 1, max(2 * k + 40, 60))
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn(n, b, dtype=torch.float64, device="cuda", generator=g)
    for _ in range(45):
        X = torch.cholesky_solve(Ms @ X, L)
        # M-orthonormal columns: Cholesky of the Gram matrix, twice
        for _ in range(2):
            X = X / torch.linalg.norm(X, dim=0)
            R = torch.linalg.cholesky(X.T @ (Ms @ X), upper=True)
            X = torch.linalg.solve_triangular(R, X, upper=True, left=False)
        As = _csr(ptr, col, A)
        w, S = torch.linalg.eigh(X.T @ (As @ X))
        X = X @ S
    return w[:k], X[:, :k]


def _mean_edge(ptr, col, v):
    rows = _rows(ptr)
    up = rows < col
    return torch.linalg.norm(v[rows[up]] - v[col[up]], dim=1).mean()


def _heat_matrix(v, t, m):
    ptr, col, A, M = _matrices(v, t, True)
    step = m * _mean_edge(ptr, col, torch.from_numpy(np.asarray(v, dtype=np.float64)).cuda()) ** 2
    K, rows = step * A, _rows(ptr)
    K[rows == col] += M
    return ptr, col, K, step


def exact(case, seed):
    rng, kind = _rng(case, seed), case["kind"]
    if kind == "eigs":
        v, t = _mesh(case, rng)
        if len(v) > 12000:
            return None
        w, X = _spectrum(v, t, case["k"])
        times = 4 * math.log(10) / w[-1] * torch.tensor(HKS_TIMES, dtype=torch.float64, device="cuda")
        return w, (X * X) @ torch.exp(-w[:, None] * times)
    if kind == "heat":
        v, t = _mesh(case, rng)
        seeds = _seeds(case, len(v), rng)
        sets = [[seeds]] if case["seeds"] == 1 else seeds
        ptr, col, K, _ = _heat_matrix(v, t, case["m"])
        b = torch.zeros(len(v), len(sets), dtype=torch.float64, device="cuda")
        for i, x in enumerate(sets):
            b[x, i] = 1.0
        u = _cg(ptr, col, K, b)
        return u[:, 0] if case["seeds"] == 1 else u
    if kind == "geodesic":
        v, t = _mesh(case, rng)
        f = torch.from_numpy(_distance_like(v, rng)).cuda()
        vd, td, _, _ = _elements(v, t)
        e = (vd[td])[:, [2, 0, 1]] - (vd[td])[:, [1, 2, 0]]
        nrm = torch.linalg.cross(e[:, 0], e[:, 1])
        area = torch.linalg.norm(nrm, dim=1) / 2
        hats = torch.linalg.cross((nrm / (2 * area[:, None]))[:, None].expand(-1, 3, -1), e) / (2 * area)[:, None, None]
        g = (hats * f[td][:, :, None]).sum(1)
        g = -g / torch.linalg.norm(g, dim=1, keepdim=True)
        b = torch.zeros(len(vd), dtype=torch.float64, device="cuda")
        b.index_add_(0, td.reshape(-1), ((hats * g[:, None]).sum(2) * area[:, None]).reshape(-1))
        ptr, col, A, _ = _matrices(v, t, False)
        x = _cg(ptr, col, A, (b - b.mean())[:, None], constants=True, tol=1e-14)[:, 0]
        return x - x.min()
    meshes = _batch(case, rng)
    if kind == "shapedna":
        return [_spectrum(v, t, case["k"])[0] if len(v) < 6000 else None for v, t in meshes]
    if kind == "spectra":
        return None
    first = np.concatenate([[0], np.cumsum([len(v) for v, _ in meshes])])
    V = np.vstack([v for v, _ in meshes])
    T = np.vstack([t.astype(np.int64) + first[i] for i, (_, t) in enumerate(meshes)])
    if kind == "heat-batch":
        parts = [_heat_matrix(v, t, 1.0) for v, t in meshes]
        ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda")] +
                        [torch.diff(p[0]) for p in parts]).cumsum(0)
        col = torch.cat([p[1] + int(first[i]) for i, p in enumerate(parts)])
        b = torch.zeros(len(V), 1, dtype=torch.float64, device="cuda")
        b[torch.from_numpy(first[:-1]).cuda()] = 1.0
        return _cg(ptr, col, torch.cat([p[2] for p in parts]), b)[:, 0], torch.stack([p[3] for p in parts])
    if kind == "assemble":
        ptr, col, A, M = _matrices(V, T, case["lump"])
        return None, None, A, M
    ptr, col, A, M = _matrices(V, T, kind == "train")
    if kind == "spmm":
        x = rng.standard_normal((len(V), case["columns"]), dtype=np.float32)
        return _csr(ptr, col, A) @ torch.from_numpy(x.astype(np.float64)).cuda()
    return _exact_gradient(case, rng, meshes, first, V, ptr, col, A, M)


def _exact_gradient(case, rng, meshes, first, V, ptr, col, A, M):
    """Factor, log q and the gradient of the mean log q in the network's parameters, by torch autograd."""
    times = torch.from_numpy(_times(case, rng)).cuda()
    sizes = torch.from_numpy(np.diff(first)).cuda()
    mesh_of = torch.repeat_interleave(torch.arange(len(meshes), device="cuda"), sizes)
    n, rows, vd = len(V), _rows(ptr), torch.from_numpy(V).cuda()
    length = torch.linalg.norm(vd[rows] - vd[col], dim=1)
    up = rows < col
    zero = torch.zeros(len(meshes), dtype=torch.float64, device="cuda")
    edges = zero.index_add(0, mesh_of[rows[up]], torch.ones_like(length[up]))
    h = zero.index_add(0, mesh_of[rows[up]], length[up]) / edges
    K = times[mesh_of[rows]] * A
    K[rows == col] += M
    low = torch.nonzero(col < rows)[:, 0]
    i, j = rows[low], col[low]
    hi, ti = h[mesh_of[i]], times[mesh_of[i]]
    feat = torch.stack([-A[low], length[low] / hi, M[i] / hi**2, M[j] / hi**2, torch.log(ti / hi**2),
                        torch.zeros_like(hi)], 1)
    theta = np.load(Path(lapy_gb300.__file__).parent / "data" / "spai_weights.npz")["theta"]
    theta = torch.from_numpy(theta.ravel()).bfloat16().double().cuda().requires_grad_()
    W1, b1, W2, b2, W3, b3 = torch.split(theta, [384, 64, 4096, 64, 64, 1])
    w = torch.tanh(torch.tanh(feat @ W1.view(64, 6).T + b1) @ W2.view(64, 64).T + b2) @ W3 + b3
    diag = K[rows == col]
    q = diag.index_add(0, i, -2 * w * K[low])
    # pairs of lower neighbours of a row whose own entry is in the pattern
    keys = rows * n + col
    start = torch.searchsorted(i, torch.arange(n + 1, device="cuda"))
    for d in range(int(torch.diff(start).max())):
        other = start[i] + d
        e = torch.nonzero(other < start[i + 1])[:, 0]
        o = other[e]
        want = j[e] * n + j[o]
        at = torch.searchsorted(keys, want).clamp(max=len(keys) - 1)
        q = q.index_add(0, i[e], torch.where(keys[at] == want, K[at], 0.0) * w[e] * w[o])
    logq = torch.log(q)
    (grad,) = torch.autograd.grad(logq.sum() / n, theta)
    gd = q.detach() ** -0.5
    g = torch.zeros(len(keys), dtype=torch.float64, device="cuda")
    g[low] = -w.detach() * gd[i]
    g[rows == col] = gd
    return g[col <= rows], logq.detach(), grad
