"""The sorted plan at the edges of its layout (csrc/stream.cuh): rows of 15 to
18 values around the short/long split, of 4 to 33 row-blocks around the classes
of the long rows, dense steps that overflow a window's staging buffer, last
slabs with one row, matrices without short or without long rows.  Every result
is the oracle's bit for bit (no tolerance)."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu

VT = {"f64": S.F64, "f32": S.F32, "mixed": S.F32, "mixed8": S.F32_V8}


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rows_matrix(lengths, step, seed, ncols=9000):
    """Row i has lengths[i] values in columns start_i + step * j (step 1: dense
    runs of full blocks; step 17: one value per block in either layout)."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i, n in enumerate(lengths):
        start = int(rng.integers(0, max(1, ncols - step * max(n, 1))))
        rows += [i] * n
        cols += [start + step * j for j in range(n)]
    return M.from_coo(len(lengths), ncols, rows, cols, rng.uniform(-1, 1, len(rows)), name=f"rows_{step}_{seed}")


def cases():
    edge = [0, 1, 2, 15, 16, 17, 18, 31, 32, 33, 34, 64, 65, 200] * 3
    yield rows_matrix(edge, 17, 1)                      # one value per row-block
    yield rows_matrix([n * 8 for n in edge], 1, 2)      # full row-blocks: 32 values per step
    yield rows_matrix([3] * 33, 1, 3)                   # only short rows, two slabs, the second with one row
    yield rows_matrix([40] * 5 + [300], 1, 4)           # only long rows, rounds that are not full
    yield rows_matrix([500, 0, 1], 17, 5)               # one long row, one empty, one value
    yield M.powerlaw(3001, seed=6)


def make(csr, kind, r):
    dt = np.float64 if kind == "f64" else np.float32
    m = S.csr_matrix(csr.rowptr, csr.colidx, csr.values.astype(dt), csr.ncols,
                     value_type=S.F32_V8 if kind == "mixed8" else None)
    m.set_kernel(S.KERNEL_SORTED)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
    conv = oracle.csr_to_beta_v8 if kind == "mixed8" else oracle.csr_to_beta
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "mixed": oracle.beta_spmv_mixed,
         "mixed8": oracle.beta_spmv_mixed8}[kind]
    return m, conv(r, csr.rowptr, csr.colidx, csr.values.astype(dt)), f


@pytest.mark.parametrize("kind", list(VT))
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_streams_equal_oracle(cuda, kind, r):
    mixed = kind.startswith("mixed")
    xt = np.float64 if kind == "f64" else np.float32
    yt = np.float32 if kind == "f32" else np.float64
    for csr in cases():
        m, (ob, oh, ov), f = make(csr, kind, r)
        gb, gh, gv = m.arrays()  # the values back from the plan
        assert np.array_equal(gb, ob) and np.array_equal(gh, oh) and gv.tobytes() == ov.tobytes(), csr.name
        x, y0 = M.x_vector(csr.ncols, 3, xt), M.x_vector(csr.nrows, 4, yt)
        yo = f(r, csr.nrows, ob, oh, ov, x, y0.copy())
        y = dev(y0)
        (S.SPC5_Spmv_mixed if mixed else S.SPC5_Spmv)(m, dev(x), y)
        torch.cuda.synchronize()
        assert y.cpu().numpy().tobytes() == yo.tobytes(), csr.name
        # right-hand sides: every pass width, a ragged one, vectors of X aligned and not
        for k, pad in ((1, 0), (2, 0), (4, 1), (7, 0), (8, 0), (16, 0), (19, 2)):
            X = np.stack([M.x_vector(csr.ncols, 10 + j, xt) for j in range(k + pad)], axis=1)
            Y0 = np.stack([M.x_vector(csr.nrows, 50 + j, yt) for j in range(k + pad)], axis=1)
            Yd = dev(Y0)
            (S.SPC5_Spmm_mixed if mixed else S.SPC5_Spmm)(m, dev(X)[:, :k], Yd[:, :k])
            torch.cuda.synchronize()
            Y = Yd.cpu().numpy()
            assert Y[:, k:].tobytes() == Y0[:, k:].tobytes()
            for j in {0, k // 2, k - 1}:
                yo = f(r, csr.nrows, ob, oh, ov, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y0[:, j]))
                assert np.ascontiguousarray(Y[:, j]).tobytes() == yo.tobytes(), (csr.name, k, j)


@pytest.mark.parametrize("k", [0, 16])
def test_streams_in_order_and_captured(cuda, k):
    """The launches of one product overlap one another but not the next call
    on the stream, eagerly and replayed from a captured graph (k = 0: SpMV)."""
    csr = M.powerlaw(40_000, seed=9)
    m, (ob, oh, ov), f = make(csr, "f64", 2)
    shape = (csr.nrows,) if k == 0 else (csr.nrows, k)
    x0 = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, shape)).cuda()
    call = S.SPC5_Spmv if k == 0 else S.SPC5_Spmm

    def chain(x, y):  # y = A (A x / 4), each product reads the one before it
        t = torch.zeros_like(x)
        call(m, x, t)
        t.mul_(0.25)
        y.zero_()
        call(m, t, y)

    ref = x0.cpu().numpy() if k == 0 else np.ascontiguousarray(x0.cpu().numpy()[:, 3])
    t = f(2, csr.nrows, ob, oh, ov, ref, np.zeros(csr.nrows)) * 0.25
    want = f(2, csr.nrows, ob, oh, ov, t, np.zeros(csr.nrows))
    y = torch.empty_like(x0)
    for _ in range(5):
        chain(x0, y)
    torch.cuda.synchronize()
    got = lambda: (y if k == 0 else y[:, 3].contiguous()).cpu().numpy()  # noqa: E731
    assert got().tobytes() == want.tobytes()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain(x0, y)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        chain(x0, y)
    y.fill_(7.0)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert got().tobytes() == want.tobytes()


@pytest.mark.parametrize("r", [2, 8])
def test_values_outside_the_rows_are_kept(cuda, r):
    """Arrays of the caller's own whose last block-row has values in the rows
    past nrows: the product leaves them out, the arrays still hold them."""
    n = 40 * r
    csr = rows_matrix([3] * n, 1, 8)
    ob, oh, ov = oracle.csr_to_beta(r, csr.rowptr, csr.colidx, csr.values)
    m = S.beta_matrix(r, n - 1, csr.ncols, ob, oh, ov)
    m.set_kernel(S.KERNEL_SORTED)
    gb, gh, gv = m.arrays()
    assert np.array_equal(gb, ob) and np.array_equal(gh, oh) and gv.tobytes() == ov.tobytes()
    x = M.x_vector(csr.ncols, 3)
    y = dev(np.zeros(n - 1))
    S.SPC5_Spmv(m, dev(x), y)
    torch.cuda.synchronize()
    yo = oracle.beta_spmv_f64(r, n, ob, oh, ov, x, np.zeros(n))[:n - 1]
    assert y.cpu().numpy().tobytes() == yo.tobytes()
