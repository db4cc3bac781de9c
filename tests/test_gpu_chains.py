"""The sorted plan's chain part (csrc/chain.cuh, plan.cu chain_rows): matrices whose
long rows are about as long as one another, and a few rows that outlast the rest.
Products and rebuilt arrays are the oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rows_of(lengths, ncols, seed, run=1):
    """Rows of the given numbers of values, in runs of neighbouring columns."""
    rng = np.random.default_rng(seed)
    cols = []
    for n in lengths:
        first = np.sort(rng.choice(ncols // (run + 1), -(-n // run), replace=False)) * (run + 1)
        cols.append((first[:, None] + np.arange(run)).reshape(-1)[:n])
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    return rowptr, np.concatenate(cols).astype(np.int32), rng.uniform(-1, 1, rowptr[-1]), ncols


CASES = {
    # all long rows are chains; chains of 1 .. 40 entries, whole steps and remainders
    "equal": rows_of([40] * 65, 3000, 1),
    "runs": rows_of([64] * 33, 4000, 2, run=8),
    "runs of 3": rows_of([51] * 40, 4000, 3, run=3),
    "some": rows_of(list(range(17, 57)) + [0, 3, 16] * 5, 2500, 4),
    # one row: its chains are the only slab, which is not full
    "one": rows_of([700] + [2] * 50, 6000, 5),
    # the longest rows are chains, the others streams and short rows
    "skewed": rows_of([1500, 900] + [24, 30, 18, 5] * 40, 9000, 6, run=3),
}


@pytest.mark.parametrize("tag", ["f64", "f32", "f32 mixed", "mixed8"])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
@pytest.mark.parametrize("name", list(CASES))
def test_chains_equal_oracle(cuda, name, r, tag):
    rowptr, colidx, vals, ncols = CASES[name]
    n = len(rowptr) - 1
    dt = np.float64 if tag == "f64" else np.float32
    yt = np.float32 if tag == "f32" else np.float64
    mixed = tag in ("f32 mixed", "mixed8")
    vals = vals.astype(dt)
    arrays = (oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta)(r, rowptr, colidx, vals)
    m = S.csr_matrix(rowptr, colidx, vals, ncols, value_type=S.F32_V8 if tag == "mixed8" else None)
    m.set_kernel(S.KERNEL_SORTED)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
    # the chains and their rows; rows of at most 16 values; streams beside chains
    assert m.spmv_launches == {"equal": 2, "runs": 2, "runs of 3": 2, "skewed": 4}.get(name, 3)
    for a, b in zip(m.arrays(), arrays):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "f32 mixed": oracle.beta_spmv_mixed,
         "mixed8": oracle.beta_spmv_mixed8}[tag]
    spmv, spmm = (S.SPC5_Spmv_mixed, S.SPC5_Spmm_mixed) if mixed else (S.SPC5_Spmv, S.SPC5_Spmm)
    X = np.stack([M.x_vector(ncols, 10 + j, dt) for j in range(17)], axis=1)
    Y = np.stack([M.x_vector(n, 40 + j, yt) for j in range(17)], axis=1)
    want = np.stack([f(r, n, *arrays, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y[:, j]).copy())
                     for j in range(17)], axis=1)
    for j in (0, 3):
        y = dev(Y[:, j])
        spmv(m, dev(X[:, j]), y)
        torch.cuda.synchronize()
        assert y.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, j]).tobytes()
    for k in (1, 2, 3, 4, 5, 8, 9, 16, 17):
        y = dev(Y[:, :k])
        spmm(m, dev(X[:, :k]), y)
        torch.cuda.synchronize()
        assert y.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, :k]).tobytes(), k
    # one and two columns of wider blocks
    Xd, Yd = dev(X[:, :6]), dev(Y[:, :6])
    spmm(m, Xd[:, 1:3], Yd[:, 1:3])
    spmm(m, Xd[:, 4:5], Yd[:, 4:5])
    torch.cuda.synchronize()
    got = Yd.cpu().numpy()
    for j in range(6):
        assert got[:, j].tobytes() == (want if j in (1, 2, 4) else Y)[:, j].tobytes(), j
    # the reference order through the other kernels and back
    m.set_kernel(S.KERNEL_GROUPS)
    y = dev(Y[:, 0])
    spmv(m, dev(X[:, 0]), y)
    torch.cuda.synchronize()
    assert y.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, 0]).tobytes()


def test_chains_in_order_and_captured(cuda):
    """Products on two streams and a captured pair: each has its own scratch, and the
    next launch on a stream sees the whole result."""
    rowptr, colidx, vals, ncols = CASES["skewed"]
    n = len(rowptr) - 1
    m = S.csr_matrix(rowptr, colidx, vals, ncols)
    m.set_kernel(S.KERNEL_SORTED)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[2])
    arrays = oracle.csr_to_beta(2, rowptr, colidx, vals)
    x0 = M.x_vector(ncols, 1)
    want = oracle.beta_spmv_f64(2, n, *arrays, x0, np.zeros(n))
    twice = oracle.beta_spmv_f64(2, n, *arrays, x0, want.copy())
    x = dev(x0)
    streams = [torch.cuda.Stream() for _ in range(3)]
    ys = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in streams]
    copies = [torch.empty_like(y) for y in ys]
    torch.cuda.synchronize()
    for _ in range(30):
        for st, y, c in zip(streams, ys, copies):
            with torch.cuda.stream(st):
                y.zero_()
                S.SPC5_Spmv(m, x, y, stream=st)
                c.copy_(y)
                S.SPC5_Spmv(m, x, y, stream=st)
    torch.cuda.synchronize()
    for y, c in zip(ys, copies):
        assert c.cpu().numpy().tobytes() == want.tobytes() and y.cpu().numpy().tobytes() == twice.tobytes()
    y, c = ys[0], copies[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y.zero_()
        S.SPC5_Spmv(m, x, y)
        c.copy_(y)
        S.SPC5_Spmv(m, x, y)
    for _ in range(3):
        y.fill_(7.0)
        graph.replay()
    torch.cuda.synchronize()
    assert c.cpu().numpy().tobytes() == want.tobytes() and y.cpu().numpy().tobytes() == twice.tobytes()
