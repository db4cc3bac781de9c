"""The workloads this library is timed on, through its public Python entry points.

Every case is plain values: ``op`` names the call, ``matrix`` the generator, ``n`` its size
(grid side for ``poisson`` and ``stencil27``, rows otherwise), ``r`` the rows per block, ``vt``
the value type (``f64``; ``f32``: the float layout; ``mixed``: float values in the 8-column
layout, float x, double y) and ``k`` the right-hand sides or requests.  The matrices are the
ones of ``spc5_b200.matrices`` and of ``bench.py`` (the same shapes and distributions), drawn on
the GPU from the seed.

ops:
* ``spmv``    y += A x on a converted handle (the call an iterative solver makes),
* ``spmm``    Y += A X for k right-hand sides (row-major),
* ``core``    the reference-named kernel interface over device arrays, without a handle,
* ``batch``   many banded matrices with their own k in one launch,
* ``convert`` CSR arrays -> handle -> beta(r,VS) -> its first product (a new matrix),
* ``decode``  CSR arrays -> handle -> beta(r,VS) -> COO triplets (there and back),
* ``serve``   a burst of requests on resident matrices through the request loop.
"""
import math

import numpy as np
import torch

import spc5_b200 as S

# Average values per block of the beta(r,8) conversion, for work().
FILL = {
    "poisson": {1: 1.67, 2: 3.33, 4: 6.66, 8: 10.0},
    "stencil27": {1: 2.98, 2: 5.97, 4: 11.9, 8: 11.9},
    "powerlaw": {1: 2.18, 2: 2.18, 4: 2.19, 8: 2.19},
    "banded": {1: 1.72, 2: 2.51, 4: 4.06, 8: 7.09},
}
MEAN_ROW = {"poisson": 5.0, "stencil27": 27.0, "powerlaw": 15.8}


def listed():
    return [
        # the smallest call: one short banded matrix of the batched workload by itself; launch and host latency
        {"name": "spmv_banded_2003_r4", "op": "spmv", "matrix": "banded", "n": 2003, "bw": 57, "r": 4, "vt": "f64"},
        # the 5-point Poisson system of the benchmark: everything fits L2
        {"name": "spmv_poisson_512_r2", "op": "spmv", "matrix": "poisson", "n": 512, "r": 2, "vt": "f64"},
        # the 27-point stencil of the benchmark, at the format its users pick
        {"name": "spmv_stencil_160_r4", "op": "spmv", "matrix": "stencil27", "n": 160, "r": 4, "vt": "f64"},
        # an odd grid at the widest block: block-rows run across grid lines
        {"name": "spmv_stencil_127_r8", "op": "spmv", "matrix": "stencil27", "n": 127, "r": 8, "vt": "f64"},
        # the reference's float format (16 columns per block)
        {"name": "spmv_stencil_101_r1_f32", "op": "spmv", "matrix": "stencil27", "n": 101, "r": 1, "vt": "f32"},
        # the headline matrix: irregular rows, the largest SpMV
        {"name": "spmv_powerlaw_4m_r1", "op": "spmv", "matrix": "powerlaw", "n": 4_000_000, "r": 1, "vt": "f64"},
        # irregular rows in mixed precision at the widest block
        {"name": "spmv_powerlaw_1m_r8_mixed", "op": "spmv", "matrix": "powerlaw", "n": 1_000_003, "r": 8,
         "vt": "mixed"},
        # several vectors at once (block solvers) on irregular rows
        {"name": "spmm_powerlaw_600k_r2_k16", "op": "spmm", "matrix": "powerlaw", "n": 600_000, "r": 2, "vt": "f64",
         "k": 16},
        # the batched workload of the benchmark, at a quarter of its matrices
        {"name": "batch_banded_64", "op": "batch", "matrix": "banded", "n": 200_000, "r": 0, "vt": "f64", "k": 64},
        # the drop-in kernel a caller of the reference links against
        {"name": "core_stencil_100_r4", "op": "core", "matrix": "stencil27", "n": 100, "r": 4, "vt": "f64"},
        # a new irregular matrix: conversion and its first product
        {"name": "convert_powerlaw_1m_r1", "op": "convert", "matrix": "powerlaw", "n": 1_000_000, "r": 1, "vt": "f64"},
        # the request loop at saturation: power-law (r = 1) and stencil (r = 4) matrices, Zipf choice
        {"name": "serve_48", "op": "serve", "matrix": "pool", "n": 300_000, "r": 0, "vt": "f64", "k": 48},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["spmv"] * 6 + ["spmm", "spmm", "core", "batch", "convert", "decode", "serve"])
    r = rng.choice([1, 2, 4, 8])
    if op == "batch":
        return {"op": op, "matrix": "banded", "n": _log(rng, 20_000, 200_000), "r": 0,
                "vt": rng.choice(["f64", "f64", "mixed"]), "k": _log(rng, 4, 64)}
    if op == "serve":
        return {"op": op, "matrix": "pool", "n": _log(rng, 20_000, 300_000), "r": 0,
                "vt": rng.choice(["f64", "mixed"]), "k": _log(rng, 8, 48)}
    matrix = rng.choice(["banded", "poisson", "stencil27", "stencil27", "powerlaw", "powerlaw", "powerlaw"])
    if op == "decode":  # the matrices whose number of values does not depend on the seed
        matrix = rng.choice(["poisson", "stencil27"])
    # the largest size of each op keeps a drawn case below the largest listed one
    share = {"spmv": 1.0, "spmm": 0.15, "core": 0.25, "convert": 0.25, "decode": 0.25}[op]
    case = {"op": op, "matrix": matrix}
    if matrix == "banded":
        case |= {"n": _log(rng, 2_000, 200_000), "bw": rng.randint(5, 200)}
    elif matrix == "poisson":
        case["n"] = _log(rng, 64, 1024 * math.sqrt(share))
    elif matrix == "stencil27":
        case["n"] = _log(rng, 16, 160 * share ** (1 / 3))
    else:
        case["n"] = _log(rng, 20_000, 4_000_000 * share)
    case |= {"r": r, "vt": rng.choice(["f64", "f64", "f32", "mixed"]) if op != "core" else rng.choice(["f64", "f32"])}
    if op == "spmm":
        case["k"] = rng.choice([2, 3, 4, 5, 8, 12, 16])
    return case


# ---------------------------------------------------------------------------
# matrices on the GPU: (nrows, rowptr, colidx, values), the generators of spc5_b200.matrices
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0


def _rowptr(counts):
    rp = torch.zeros(counts.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=rp[1:])
    return rp.to(torch.int32)


def _grid(offsets, valid, idx):
    cols = torch.stack([idx + o for o in offsets], dim=1)
    ok = torch.stack(valid, dim=1)
    return _rowptr(ok.sum(1)), cols[ok].to(torch.int32), ok


def _poisson(side):
    idx = torch.arange(side * side, device="cuda")
    iy, ix = idx // side, idx % side
    rp, ci, ok = _grid([-side, -1, 0, 1, side], [iy > 0, ix > 0, ix >= 0, ix < side - 1, iy < side - 1], idx)
    diag = torch.zeros_like(ok)
    diag[:, 2] = True
    return side * side, rp, ci, torch.where(diag[ok], 4.0, -1.0).to(torch.float64)


def _stencil27(side, g):
    n = side ** 3
    idx = torch.arange(n, device="cuda")
    iz, iy, ix = idx // (side * side), (idx // side) % side, idx % side
    offsets, valid = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                offsets.append(dz * side * side + dy * side + dx)
                valid.append((iz + dz >= 0) & (iz + dz < side) & (iy + dy >= 0) & (iy + dy < side) &
                             (ix + dx >= 0) & (ix + dx < side))
    rp, ci, ok = _grid(offsets, valid, idx)
    diag = torch.zeros_like(ok)
    diag[:, 13] = True
    vals = torch.where(diag[ok], 26.0, -1.0 + 1e-3 * _uniform(g, ci.numel()))
    return n, rp, ci, vals


def _banded(n, bw, g):
    w = 2 * bw + 1
    off = torch.arange(-bw, bw + 1, device="cuda")
    counts, cols = [], []
    step = max(1, (1 << 25) // w)
    for r0 in range(0, n, step):
        rows = torch.arange(r0, min(n, r0 + step), device="cuda")
        cc = rows[:, None] + off[None, :]
        keep = torch.rand(cc.shape, generator=g, device="cuda") < 0.1
        keep[:, bw] = True
        keep &= (cc >= 0) & (cc < n)
        counts.append(keep.sum(1))
        cols.append(cc[keep].to(torch.int32))
    ci = torch.cat(cols)
    return n, _rowptr(torch.cat(counts)), ci, _uniform(g, ci.numel())


def _powerlaw(n, g):
    # row lengths min(2000, Zipf(1.8) + 3); 70% of a row in runs of U[1, 16] near the diagonal
    # (sigma n / 100), the rest uniform; duplicates merged
    pmf = np.arange(1, 1997, dtype=np.float64) ** -1.8
    cdf = torch.from_numpy(np.cumsum(pmf) / 1.8822296181028)  # zeta(1.8)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    lens = torch.clamp(torch.searchsorted(cdf.cuda(), u) + 4, max=2000)
    n_run = torch.round(0.7 * lens).to(torch.int64)
    row_end = torch.cumsum(n_run, 0)
    total = int(row_end[-1])
    run_end = torch.cumsum(torch.randint(1, 17, (int(total / 8.5 * 1.1) + 4096,), generator=g, device="cuda"), 0)
    cuts = torch.unique(torch.cat([run_end[run_end < total], row_end]))
    start = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), cuts[:-1]])
    seg = cuts - start
    row = torch.searchsorted(row_end, start, right=True)
    centre = row + torch.round(torch.randn(seg.numel(), generator=g, device="cuda") * (0.01 * n)).to(torch.int64)
    first = torch.minimum(torch.clamp(centre, min=0), n - seg)
    key = torch.repeat_interleave(row * n + first - start, seg) + torch.arange(total, device="cuda")
    n_uni = lens - n_run
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), n_uni)
    uni = rows * n + torch.randint(0, n, (rows.numel(),), generator=g, device="cuda")
    key = torch.unique(torch.cat([key, uni]))
    rows = key // n
    return n, _rowptr(torch.bincount(rows, minlength=n)), (key - rows * n).to(torch.int32), _uniform(g, key.numel())


def _matrix(case, seed):
    g = _gen(seed)
    if case["matrix"] == "poisson":
        return _poisson(case["n"])
    if case["matrix"] == "stencil27":
        return _stencil27(case["n"], g)
    if case["matrix"] == "banded":
        return _banded(case["n"], case["bw"], g)
    return _powerlaw(case["n"], g)


def _members(case, seed):
    """The matrices of a batch or of a serving pool: (case of one, seed, k or share)."""
    rng = np.random.Generator(np.random.PCG64(5))
    if case["op"] == "batch":  # n log-uniform up to the case's, bandwidth U[5, 200], k in {1, 4, 8, 16}
        out = []
        for i in range(case["k"]):
            n = int(round(math.exp(rng.uniform(math.log(case["n"] / 100), math.log(case["n"])))))
            one = {"matrix": "banded", "n": n, "bw": int(rng.integers(5, 201)), "vt": case["vt"]}
            out.append((one, seed * 1000 + i, int(rng.choice([1, 4, 8, 16]))))
        return out
    n = case["n"]
    pool = [("powerlaw", n // 6, 1), ("stencil27", max(8, round((n / 3) ** (1 / 3))), 4), ("powerlaw", n, 1),
            ("stencil27", max(8, round(n ** (1 / 3))), 4)]
    return [({"matrix": m, "n": s, "r": r, "vt": case["vt"]}, seed * 1000 + i, 1.0 / (i + 1) ** 1.1)
            for i, (m, s, r) in enumerate(pool)]


def _requests(case):
    """Matrix of each request: Zipf(1.1) over the pool."""
    rng = np.random.Generator(np.random.PCG64(case["k"]))
    w = np.array([s for _, _, s in _members(case, 0)])
    return [int(i) for i in rng.choice(len(w), size=case["k"], p=w / w.sum())]


def _x_type(vt):
    return torch.float64 if vt == "f64" else torch.float32


def _y_type(vt):
    return torch.float32 if vt == "f32" else torch.float64


def _vectors(vt, seed, nrows, ncols, k=None):
    g = _gen(seed + 100_000_007)
    shape = () if k is None else (k,)
    x = _uniform(g, ncols, *shape).to(_x_type(vt))
    y = _uniform(g, nrows, *shape).to(_y_type(vt))
    return x, y


def _handle(vt, n, rp, ci, vals, r):
    vals = vals.to(_x_type(vt))
    m = S.csr_matrix(rp, ci, vals, n, value_type=S.F32_V8 if vt == "mixed" else None)
    r = r or S.autotune(m)["r"]
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
    return m


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def prepare(case, seed):
    op, vt = case["op"], case["vt"]
    if op in ("batch", "serve"):
        mats, xs, ys = [], [], []
        for one, s, k in _members(case, seed):
            n, rp, ci, vals = _matrix(one, s)
            mats.append(_handle(vt, n, rp, ci, vals, one.get("r", 0)))
            if op == "batch":
                x, y = _vectors(vt, s, n, n, k)
                xs.append(x)
                ys.append(y)
        if op == "batch":
            return {"op": op, "batch": S.Batch(mats, xs, ys, mixed=vt == "mixed"), "y": ys}
        server = S.Server(slots=4, max_k=16, hbm_budget=32 << 30, mixed=vt == "mixed")
        ids = [server.add_matrix(m) for m in mats]
        todo = []
        for j, i in enumerate(_requests(case)):
            n = mats[i].numberOfRows
            x, _ = _vectors(vt, seed * 1000 + 500 + j, 1, n)
            todo.append((ids[i], x, torch.empty(n, dtype=torch.float64, device="cuda")))
        torch.cuda.synchronize()  # the request loop reads x on its own streams
        return {"op": op, "server": server, "todo": todo}
    n, rp, ci, vals = _matrix(case, seed)
    if op in ("convert", "decode"):
        x, y = _vectors(vt, seed, n, n)
        return {"op": op, "vt": vt, "csr": (n, rp, ci, vals.to(_x_type(vt))), "r": case["r"], "x": x, "y": y}
    m = _handle(vt, n, rp, ci, vals, case["r"])
    x, y = _vectors(vt, seed, n, n, case.get("k"))
    if op == "core":
        arrays = tuple(torch.from_numpy(a).cuda() for a in m.arrays())
        return {"op": op, "r": case["r"], "n": n, "arrays": arrays, "x": x, "y": y}
    return {"op": op, "vt": vt, "m": m, "x": x, "y": y}


def run(state):
    op = state["op"]
    if op == "spmv":
        (S.SPC5_Spmv_mixed if state["vt"] == "mixed" else S.SPC5_Spmv)(state["m"], state["x"], state["y"])
        return state["y"]
    if op == "spmm":
        (S.SPC5_Spmm_mixed if state["vt"] == "mixed" else S.SPC5_Spmm)(state["m"], state["x"], state["y"])
        return state["y"]
    if op == "core":
        S.core_spmv(state["r"], state["n"], *state["arrays"], state["x"], state["y"])
        return state["y"]
    if op == "batch":
        state["batch"].launch()
        return state["y"]
    if op == "serve":
        for i, x, y in state["todo"]:
            state["server"].submit(i, x, y)
        state["server"].drain()
        return [y for _, _, y in state["todo"]]
    n, rp, ci, vals = state["csr"]
    m = S.csr_matrix(rp, ci, vals, n, value_type=S.F32_V8 if state["vt"] == "mixed" else None)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[state["r"]])
    if op == "decode":
        return S.decode_coo(m)
    (S.SPC5_Spmv_mixed if state["vt"] == "mixed" else S.SPC5_Spmv)(m, state["x"], state["y"])
    return state["y"]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its results in 64 bits
# ---------------------------------------------------------------------------

def _rows(one):
    return {"poisson": one["n"] ** 2, "stencil27": one["n"] ** 3}.get(one["matrix"], one["n"])


def _size(one):
    """(rows, values, bytes of the converted arrays) of one matrix."""
    n, r = _rows(one), one.get("r") or 4
    per_row = 1 + 0.2 * one["bw"] if one["matrix"] == "banded" else MEAN_ROW[one["matrix"]]
    nnz = per_row * n
    vb, mb, wide = (8, 1, 1.0) if one["vt"] == "f64" else ((4, 1, 1.0) if one["vt"] == "mixed" else (4, 2, 0.9))
    blocks = wide * nnz / FILL[one["matrix"]][r]
    return n, nnz, nnz * vb + blocks * (4 + r * mb) + 4 * (n / r + 1)


def work(case):
    op, vt = case["op"], case["vt"]
    xb, yb = (8 if vt == "f64" else 4), (4 if vt == "f32" else 8)
    if op == "batch":
        sizes = [(_size(one), k) for one, _, k in _members(case, 0)]
        return {"bytes": sum(b + k * n * (xb + 2 * yb) for (n, _, b), k in sizes),
                "flops": sum(2 * k * nnz for (_, nnz, _), k in sizes)}
    if op == "serve":  # every matrix at least once, every request's x and y
        sizes = [_size(one) for one, _, _ in _members(case, 0)]
        asked = _requests(case)
        return {"bytes": sum(sizes[i][2] for i in set(asked)) + sum(sizes[i][0] * (xb + yb) for i in asked),
                "flops": sum(2 * sizes[i][1] for i in asked)}
    n, nnz, arrays = _size(case)
    csr = nnz * (4 + xb) + 4 * n
    if op == "convert":  # CSR in, beta arrays out and in again, the product
        return {"bytes": csr + 2 * arrays + n * (xb + 2 * yb), "flops": 2 * nnz}
    if op == "decode":  # CSR in, beta arrays out and in again, COO out
        return {"bytes": csr + 2 * arrays + nnz * (8 + xb), "flops": 0}
    k = case.get("k", 1)
    return {"bytes": arrays + k * n * (xb + 2 * yb), "flops": 2 * nnz * k}


def _product(vt, n, rp, ci, vals, x):
    """A x in float64 from the values and x as the case's type holds them."""
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(rp.to(torch.int64)))
    vals = vals.to(_x_type(vt)).to(torch.float64)
    cols = ci.to(torch.int64)
    x = x.to(torch.float64)
    if x.dim() == 1:
        return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, vals * x[cols])
    out = [torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, vals * x[cols, j])
           for j in range(x.shape[1])]
    return torch.stack(out, dim=1)


def exact(case, seed):
    op, vt = case["op"], case["vt"]
    if op == "batch":
        out = []
        for one, s, k in _members(case, seed):
            n, rp, ci, vals = _matrix(one, s)
            x, y = _vectors(vt, s, n, n, k)
            out.append(y + _product(vt, n, rp, ci, vals, x))
        return out
    if op == "serve":
        mats = [_matrix(one, s) for one, s, _ in _members(case, seed)]
        return [_product(vt, *mats[i], _vectors(vt, seed * 1000 + 500 + j, 1, mats[i][0])[0])
                for j, i in enumerate(_requests(case))]
    n, rp, ci, vals = _matrix(case, seed)
    if op == "decode":
        if case["r"] != 1:  # the storage order of r > 1 is the format's own
            return None
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.diff(rp.to(torch.int64)))
        return rows.to(torch.int32), ci, vals.to(_x_type(vt)).to(torch.float64)
    x, y = _vectors(vt, seed, n, n, case.get("k"))
    return y.to(torch.float64) + _product(vt, n, rp, ci, vals, x)
