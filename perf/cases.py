"""The work that programs built on this library have it do, as cases that can be timed and
compared: each case names a path and its sizes; ``prepare`` makes what such a program holds
before the call, ``run`` is one pass through the public entry points, ``work`` the bytes and
operations the path cannot do without, and ``exact`` the same results in 64 bits.

The paths, by the part of a drape that uses them:

* ``step``: whole implicit steps of a drape (scene or batch -> step -> readback), with the
  state written from the host as a host engine does it. The cloth starts just above what it
  falls onto and moves down, so the steps assemble, solve, collect contact stencils and run
  the step-size filter;
* ``hessian``: the exact Hessian that the adjoint's backward pass solves with, assembled at
  given positions and read back. (The adjoint's gradients themselves are not a case: along a
  drape with seams a change in the last bit of one vertex moves them by 1e-4 to 1e-1 of their
  size, so two correct builds cannot be compared by them.);
* ``solve``: the linear-solver seam (CSR and right-hand side in host memory, x back), called
  with new values on a known pattern, as every Newton iteration of a host engine does;
* ``spmv`` and ``schwarz``: the operators on device vectors, for programs that run their own
  Krylov loop; a Schwarz preconditioner is factored once per system and then applied;
* ``sort`` and ``lbvh``: the broad phase on device buffers: pair sorts, tree builds and point
  queries, the pairs put in order before they are used (the query appends them as found).
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nguo-3d_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mguso  # noqa: E402
from mguso import lbvh as mlbvh  # noqa: E402
from mguso import scenes  # noqa: E402

_CTX = None


def _ctx():
    """The program's one context on this GPU."""
    global _CTX
    if _CTX is None:
        _CTX = mguso.Context(0)
    return _CTX


def _stream():
    return torch.cuda.current_stream().cuda_stream


def listed():
    return [
        # a program's own Krylov loop on the 1024 x 1024 cloth grid (larger than L2)
        {"name": "spmv_grid1024", "path": "spmv", "n": 1024},
        # its preconditioner: one factorisation and four applies at the same size
        {"name": "schwarz_grid1024", "path": "schwarz", "n": 1024, "domain": 32, "levels": 1, "applies": 4},
        # the two-level form at the reference command line's domain size and weight
        {"name": "schwarz_ml_grid200", "path": "schwarz", "n": 200, "domain": 16, "levels": 2, "applies": 4},
        # one Newton system of a 64 x 64 sheet through the linear-solver seam
        {"name": "solve_schwarz_grid64", "path": "solve", "n": 64, "precond": "schwarz", "domain": 32,
         "precision": "mixed", "tol": 1e-6},
        # a finer, ragged sheet with the plain preconditioner, all in FP32
        {"name": "solve_block_grid181", "path": "solve", "n": 181, "precond": "block", "domain": 32,
         "precision": "fp32", "tol": 1e-5},
        # a small pair sort, where launches count (the largest the reference's sort takes)
        {"name": "sort_u32_65536", "path": "sort", "n": 65536, "bits": 32},
        # broad phase over one garment's worth of triangles, 63-bit keys, ragged count
        {"name": "lbvh63_41401", "path": "lbvh", "nt": 41401, "bits": 63},
        # the large broad phase: 4 194 304 triangles, 30-bit keys
        {"name": "lbvh30_4m", "path": "lbvh", "nt": 4 << 20, "bits": 30},
        # the small drape: a 64 x 64 sheet falling onto a sphere, plain FP32
        {"name": "step_sheet64", "path": "step", "scene": "sheet", "n": 64, "speed": 0.6, "steps": 1,
         "precision": "fp32"},
        # one garment: the seamed sheath of 41k triangles falling onto its 20k-triangle torso
        {"name": "step_sheath", "path": "step", "scene": "sheath", "edge": 8e-3, "speed": 2.0, "steps": 2,
         "precision": "mixed"},
        # the sheath graded into six sizes, draped as one batch
        {"name": "step_batch6", "path": "step", "scene": "batch", "sizes": 6, "edge": 8e-3, "speed": 2.0, "steps": 2,
         "precision": "mixed"},
        # the system of the adjoint's backward pass on the XS sheath
        {"name": "hessian_sheath", "path": "hessian", "edge": 8e-3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    path = rng.choice(["spmv", "schwarz", "solve", "sort", "lbvh", "step", "step", "hessian"])
    if path == "spmv":
        return {"path": path, "n": _log(rng, 24, 1024)}
    if path == "schwarz":
        return {"path": path, "n": _log(rng, 24, 512), "domain": rng.choice([8, 13, 16, 24, 32, 32]),
                "levels": rng.choice([1, 1, 2]), "applies": rng.randint(1, 8)}
    if path == "solve":
        return {"path": path, "n": _log(rng, 12, 181), "precond": rng.choice(["schwarz", "schwarz", "block", "schwarz-ml"]),
                "domain": rng.choice([16, 32]), "precision": "mixed", "tol": 1e-6}
    if path == "sort":
        return {"path": path, "n": _log(rng, 1000, 4 << 20), "bits": rng.choice([30, 32, 48, 63, 64])}
    if path == "lbvh":
        return {"path": path, "nt": _log(rng, 500, 4 << 20), "bits": rng.choice([30, 63])}
    if path == "hessian":
        return {"path": path, "edge": round(rng.uniform(8e-3, 40e-3), 5)}
    scene = rng.choice(["sheet", "sheath", "batch"])
    c = {"path": path, "scene": scene, "steps": rng.choice([1, 2]), "speed": round(rng.uniform(0.2, 2.0), 3),
         "precision": rng.choice(["mixed", "mixed", "fp32"])}
    if scene == "sheet":
        c["n"] = rng.randint(16, 80)
        c["speed"] = round(rng.uniform(0.2, 0.8), 3)
    elif scene == "sheath":
        c["edge"] = round(rng.uniform(8e-3, 40e-3), 5)
    else:
        c["sizes"] = rng.randint(2, 6)
        c["edge"] = round(rng.uniform(12e-3, 40e-3), 5)
    return c


# ---- inputs -----------------------------------------------------------------------------
def _cloth_system(n, seed):
    """One Newton system of an n x n cloth grid: per-vertex inertia m / h^2 plus a spring of
    stiffness k along every edge (the jittered sheet's directions), and a right-hand side of
    gravity with per-vertex noise. Returns BSR arrays and b."""
    rng = np.random.default_rng(seed)
    nv = n * n
    s = np.linspace(-0.5, 0.5, n)
    X, Z = np.meshgrid(s, s)
    pos = np.stack([X, np.zeros_like(X), Z], -1).reshape(-1, 3) + rng.uniform(-1e-3, 1e-3, (nv, 3))
    e = scenes.grid_edges(n)
    d = pos[e[:, 1]] - pos[e[:, 0]]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = 50.0 * rng.uniform(0.8, 1.2, (len(e), 1, 1))
    blk = k * (d[:, :, None] * d[:, None, :])
    m_h2 = 0.2 / nv * 3600.0
    diag = np.tile(np.eye(3) * m_h2, (nv, 1, 1))
    np.add.at(diag, e[:, 0], blk)
    np.add.at(diag, e[:, 1], blk)
    rows = np.concatenate([np.arange(nv), e[:, 0], e[:, 1]])
    cols = np.concatenate([np.arange(nv), e[:, 1], e[:, 0]])
    vals = np.concatenate([diag, -blk, -blk])
    order = np.lexsort((cols, rows))
    rp = np.zeros(nv + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=nv), out=rp[1:])
    b = np.tile([0.0, -9.8 * 0.2 / nv, 0.0], (nv, 1)) + 1e-4 * rng.standard_normal((nv, 3))
    return (nv, rp.astype(np.uint32), cols[order].astype(np.uint32), vals[order].astype(np.float32),
            b.reshape(-1).astype(np.float32))


def _soup(nt, seed):
    """nt triangles with centroids uniform in the unit cube and 2 mm edges, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.rand((nt, 1, 3), generator=g, device="cuda")
    off = (torch.rand((nt, 3, 3), generator=g, device="cuda") - 0.5) * 2e-3
    return (c + off).reshape(-1, 3).contiguous(), torch.arange(3 * nt, dtype=torch.int32, device="cuda")


def _vectors(count, n, seed):
    rng = np.random.default_rng(seed + 1)
    return [rng.standard_normal(n).astype(np.float32) for _ in range(count)]


def _drape_scenes(case, seed):
    if case["scene"] == "sheet":
        return [scenes.sheet_on_sphere(case["n"], height=0.305, seed=seed)]
    res = max(24, int(round(100 * 8e-3 / case["edge"])))
    kw = dict(edge=case["edge"], seed=seed, torso_res=(res, res - 1))
    if case["scene"] == "sheath":
        return [scenes.sheath_on_torso(**kw)]
    return scenes.graded_sheaths(case["sizes"], **kw)


def prepare(case, seed):
    path = case["path"]
    if path == "spmv":
        nb, rp, col, val = scenes.grid_bsr(case["n"], seed)
        a = mguso.Bsr(_ctx(), nb, rp, col, val)
        a.autotune()
        x = torch.from_numpy(_vectors(1, 3 * nb, seed)[0]).cuda()
        return {"path": path, "a": a, "x": x, "y": torch.empty_like(x)}
    if path == "schwarz":
        nb, rp, col, val = scenes.grid_bsr(case["n"], seed)
        a = mguso.Bsr(_ctx(), nb, rp, col, val)
        s = mguso.Schwarz(a, case["domain"], levels=case["levels"])
        r = [torch.from_numpy(v).cuda() for v in _vectors(case["applies"], 3 * nb, seed)]
        return {"path": path, "a": a, "s": s, "r": r, "z": [torch.empty_like(v) for v in r]}
    if path == "solve":
        nb, rp, col, val, b = _cloth_system(case["n"], seed)
        m = mguso.CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val))
        s = mguso.CudaLinearSolver(_ctx(), precond=case["precond"], domain=case["domain"], precision=case["precision"])
        return {"path": path, "solver": s, "m": m, "b": b, "tol": case["tol"]}
    if path == "sort":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, bits = case["n"], case["bits"]
        lo = torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)
        if bits > 32:
            hi = torch.randint(0, 1 << (bits - 32), (n,), generator=g, device="cuda", dtype=torch.int64)
            k = lo | (hi << 32)
        else:
            k = (lo & ((1 << bits) - 1)).to(torch.int32)
        v = torch.arange(n, dtype=torch.int32, device="cuda")
        return {"path": path, "ctx": _ctx(), "k0": k, "v0": v, "k": k.clone(), "v": v.clone(), "bits": bits}
    if path == "lbvh":
        pos, tris = _soup(case["nt"], seed)
        cap = 4 * case["nt"] + 1024  # about 3.5 pairs a triangle at the densest
        return {"path": path, "b": mlbvh.Lbvh(_ctx()), "pos": pos, "tris": tris, "nt": case["nt"], "bits": case["bits"],
                "pairs": torch.empty((cap, 2), dtype=torch.int32, device="cuda"), "cap": cap,
                "count": torch.zeros(1, dtype=torch.int64, device="cuda")}
    if path == "hessian":
        sc = scenes.graded_sheath(0, edge=case["edge"], seed=seed)
        # stretched by up to 1%, as a drape under way is
        x = sc["positions"].copy()
        free = sc["inv_mass"] > 0
        x[free, 1] = x[free, 1].min() + (x[free, 1] - x[free, 1].min()) * np.float32(1.01)
        x[free] += np.random.default_rng(seed).uniform(-1e-4, 1e-4, (int(free.sum()), 3)).astype(np.float32)
        sc["params"] = dict(sc["params"], factor_storage=1)
        return {"path": path, "solver": mguso.ImplicitSolver(_ctx(), sc, "mixed"), "x": x}
    scs = _drape_scenes(case, seed)
    if case["scene"] == "batch":
        solver = mguso.ImplicitBatch(_ctx(), scs, case["precision"])
    else:
        solver = mguso.ImplicitSolver(_ctx(), scs[0], case["precision"])
    p = np.concatenate([s["positions"] for s in scs])
    v = np.zeros_like(p)
    v[np.concatenate([s["inv_mass"] for s in scs]) > 0, 1] = -case["speed"]
    return {"path": path, "solver": solver, "p": p, "v": v, "steps": case["steps"], "sheet": case["scene"] == "sheet"}


# ---- one pass ---------------------------------------------------------------------------
def run(st):
    path = st["path"]
    if path == "spmv":
        st["a"].spmv(st["x"].data_ptr(), st["y"].data_ptr(), _stream())
        return st["y"]
    if path == "schwarz":
        st["s"].factor(_stream())
        for r, z in zip(st["r"], st["z"]):
            st["s"].apply(r.data_ptr(), z.data_ptr(), _stream())
        return st["z"]
    if path == "solve":
        return st["solver"].solve(st["m"], st["b"], st["tol"], 2000)
    if path == "sort":
        st["k"].copy_(st["k0"])
        st["v"].copy_(st["v0"])
        mlbvh.radix_sort_pairs(st["ctx"], st["k"].data_ptr(), st["v"].data_ptr(), st["k"].numel(), st["bits"], _stream())
        return st["k"], st["v"]
    if path == "lbvh":
        nv = st["pos"].shape[0]
        st["pairs"].fill_(-1)
        st["b"].build(st["pos"].data_ptr(), nv, st["tris"].data_ptr(), st["nt"], st["bits"], _stream())
        st["b"].query_points(st["pos"].data_ptr(), nv, 1e-3, st["pairs"].data_ptr(), st["cap"], st["count"].data_ptr(),
                             _stream())
        # (query, triangle) as one key, the triangle above the query; unused entries first
        return torch.sort(st["pairs"].view(torch.int64).reshape(-1)).values, st["count"]
    if path == "hessian":
        a = st["solver"].assemble(st["x"], exact=True)
        return {"ps": a["ps"], "c": a["c"], "rhs": a["rhs"]}
    s = st["solver"]
    s.positions = st["p"]
    s.velocities = st["v"]
    s.step(st["steps"])
    if st["sheet"]:
        return {"x": s.positions, "v": s.velocities}
    # a garment's positions are what its host draws; over two steps the velocities are in them
    return {"x": s.positions}


# ---- what a pass cannot do without ------------------------------------------------------
def _grid_nnz(n):
    return n * n + 2 * (2 * n * (n - 1) + (n - 1) ** 2)


def _sheath_counts(edge, sizes=1):
    """(vertices, triangles) of the free cloth, roughly."""
    nx, ny = 0.6 / edge, 1.1 / edge
    return sizes * 2 * (nx + 1) * (ny + 1), sizes * 4 * nx * ny


def work(case):
    path = case["path"]
    if path == "spmv":
        nb, nnz = case["n"] ** 2, _grid_nnz(case["n"])
        return {"bytes": 40 * nnz + 4 * (nb + 1) + 24 * nb, "flops": 18 * nnz}
    if path == "schwarz":
        nb, nnz, m = case["n"] ** 2, _grid_nnz(case["n"]), 3 * case["domain"]
        nd = nb / case["domain"]
        tri = 4 * nd * m * (m + 1) / 2
        return {"bytes": 40 * nnz + tri + case["applies"] * (tri + 24 * nb),
                "flops": nd * (2 * m**3 / 3 + case["applies"] * 2 * m * m)}
    if path == "solve":
        nb, nnz = case["n"] ** 2, _grid_nnz(case["n"])
        # the system once from the host and x back; what the iterations read again is on chip
        return {"bytes": 72 * nnz + 4 * 3 * nb + 24 * nb, "flops": 60 * (18 * nnz + 40 * nb)}
    if path == "sort":
        return {"bytes": 2 * case["n"] * (4 + (4 if case["bits"] <= 32 else 8)), "flops": case["n"]}
    if path == "lbvh":
        nt, np_ = case["nt"], 3 * case["nt"]
        # vertices and triangles in, one box a node out, every point's query and its pair
        return {"bytes": 12 * np_ + 12 * nt + 24 * 2 * nt + 12 * np_ + 8 * np_, "flops": 60 * nt}
    if path == "hessian":
        nv, nt = _sheath_counts(case["edge"])
        return {"bytes": 24 * nv + 12 * nt + 13 * 40 * nv + 12 * nv, "flops": 2000 * nt}
    if case["scene"] == "sheet":
        nv, nt = case["n"] ** 2, 2 * (case["n"] - 1) ** 2
    else:
        nv, nt = _sheath_counts(case["edge"], case.get("sizes", 1))
    # per step: state in and out, the elements read, two Newton systems built and solved
    per = 48 * nv + 40 * nt + 2 * (13 * 40 * nv + 600 * nv)
    return {"bytes": case["steps"] * per, "flops": case["steps"] * 2 * (2000 * nt + 100 * 18 * 13 * nv)}


# ---- the same results in 64 bits --------------------------------------------------------
def _domains(n_nodes, neighbours, size):
    """Greedy breadth-first aggregates of at most `size` nodes, seeds in order; `neighbours(v)`
    ascending. Returns the node lists."""
    taken = bytearray(n_nodes)
    out = []
    for seed in range(n_nodes):
        if taken[seed]:
            continue
        dom = [seed]
        taken[seed] = 1
        i = 0
        while len(dom) < size and i < len(dom):
            for w in neighbours(dom[i]):
                if len(dom) >= size:
                    break
                if not taken[w]:
                    taken[w] = 1
                    dom.append(w)
            i += 1
        out.append(dom)
    return out


def _dense_solve(doms, blocks, vecs):
    """z = sum over domains of (dense block + floor)^-1 r in float64. blocks: (row, col, val)
    of the 3x3 entries; vecs: (count, nodes, 3)."""
    n = vecs.shape[1]
    size = max(len(d) for d in doms)
    nd = len(doms)
    lens = np.array([len(d) for d in doms])
    flat = np.concatenate([np.asarray(d, np.int64) for d in doms])
    dom_of = np.empty(n, np.int64)
    loc = np.empty(n, np.int64)
    dom_of[flat] = np.repeat(np.arange(nd), lens)
    loc[flat] = np.concatenate([np.arange(k) for k in lens])
    rows, cols, val = blocks
    inside = dom_of[rows] == dom_of[cols]
    rows, cols, val = (torch.from_numpy(np.ascontiguousarray(a[inside])).cuda() for a in (rows, cols, val))
    dom_t, loc_t = torch.from_numpy(dom_of).cuda(), torch.from_numpy(loc).cuda()
    m3 = 3 * size
    out = torch.zeros((vecs.shape[0], n, 3), dtype=torch.float64, device="cuda")
    v64 = torch.from_numpy(vecs.astype(np.float64)).cuda()
    lens_t = torch.from_numpy(lens).cuda()
    for d0 in range(0, nd, 4096):
        d1 = min(nd, d0 + 4096)
        k = (dom_t[rows] >= d0) & (dom_t[rows] < d1)
        D = torch.zeros((d1 - d0, size, 3, size, 3), dtype=torch.float64, device="cuda")
        D[dom_t[rows[k]] - d0, loc_t[rows[k]], :, loc_t[cols[k]], :] = val[k].double()
        D = D.reshape(d1 - d0, m3, m3)
        m = 3 * lens_t[d0:d1].double()
        floor = 1e-6 * (D.diagonal(dim1=1, dim2=2).sum(1) / m) + 1e-8
        used = (torch.arange(m3, device="cuda")[None, :] < m[:, None]).double()
        D += torch.diag_embed(floor[:, None] * used + (1 - used))
        nodes = torch.nonzero((dom_t >= d0) & (dom_t < d1))[:, 0]
        r = torch.zeros((d1 - d0, size, 3, vecs.shape[0]), dtype=torch.float64, device="cuda")
        r[dom_t[nodes] - d0, loc_t[nodes]] = v64[:, nodes].permute(1, 2, 0)
        z = torch.linalg.solve(D, r.reshape(d1 - d0, m3, -1)).reshape(d1 - d0, size, 3, -1)
        out[:, nodes] = z[dom_t[nodes] - d0, loc_t[nodes]].permute(2, 0, 1)
    return out, dom_of


def _exact_schwarz(case, seed):
    nb, rp, col, val = scenes.grid_bsr(case["n"], seed)
    rp64 = rp.astype(np.int64)
    starts, cols = rp64.tolist(), col.tolist()

    def neighbours(v):
        return [w for w in cols[starts[v]:starts[v + 1]] if w != v]

    doms = _domains(nb, neighbours, case["domain"])
    rows = np.repeat(np.arange(nb), np.diff(rp64))
    c64 = col.astype(np.int64)
    vecs = np.stack(_vectors(case["applies"], 3 * nb, seed)).reshape(-1, nb, 3)
    z, dom_of = _dense_solve(doms, (rows, c64, val), vecs)
    if case["levels"] == 2:
        nd = len(doms)
        key, inv = np.unique(dom_of[rows] * nd + dom_of[c64], return_inverse=True)
        a1 = np.zeros((len(key), 3, 3))
        np.add.at(a1, inv, val.astype(np.float64))
        crow, ccol = key // nd, key % nd
        adj = [[] for _ in range(nd)]
        for g, h in zip(crow.tolist(), ccol.tolist()):
            if g != h:
                adj[g].append(h)
        cdoms = _domains(nd, adj.__getitem__, case["domain"])
        rc = np.zeros((vecs.shape[0], nd, 3))
        for k in range(vecs.shape[0]):
            np.add.at(rc[k], dom_of, vecs[k].astype(np.float64))
        zc, _ = _dense_solve(cdoms, (crow, ccol, a1), rc)
        z = z + 0.7 * zc[:, torch.from_numpy(dom_of).cuda()]
    return [z[k].reshape(-1) for k in range(z.shape[0])]


def _spmv64(rp, col, val, x):
    prod = np.einsum("kij,kj->ki", val, x.reshape(-1, 3)[col])
    return np.add.reduceat(prod, rp[:-1], axis=0).reshape(-1)


def exact(case, seed):
    path = case["path"]
    if path == "spmv":
        nb, rp, col, val = scenes.grid_bsr(case["n"], seed)
        x = _vectors(1, 3 * nb, seed)[0].astype(np.float64)
        return _spmv64(rp.astype(np.int64), col.astype(np.int64), val.astype(np.float64), x)
    if path == "schwarz":
        return _exact_schwarz(case, seed)
    if path == "solve":
        nb, rp, col, val, b = _cloth_system(case["n"], seed)
        rows = np.repeat(np.arange(nb), np.diff(rp.astype(np.int64)))
        inv = torch.linalg.inv(torch.from_numpy(val[col == rows].astype(np.float64)).cuda())
        rows, col = torch.from_numpy(rows).cuda(), torch.from_numpy(col.astype(np.int64)).cuda()
        val, b = torch.from_numpy(val.astype(np.float64)).cuda(), torch.from_numpy(b.astype(np.float64)).cuda().view(-1, 3)

        def mul(m, v):
            return (m @ v[:, :, None])[:, :, 0]

        x, r = torch.zeros_like(b), b.clone()
        z = mul(inv, r)
        p, rz, b2 = z.clone(), (r * z).sum(), (b * b).sum()
        for k in range(6000):  # conjugate gradients to 1e-13
            ap = torch.zeros_like(p).index_add_(0, rows, mul(val, p[col]))
            al = rz / (p * ap).sum()
            x += al * p
            r -= al * ap
            if k % 20 == 0 and bool((r * r).sum() <= 1e-26 * b2):
                break
            z = mul(inv, r)
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return x.view(-1)
    # sorted keys and pairs are whole numbers; a drape step and the assembled Hessian have no
    # value that plain numpy gives in reasonable time
    return None
