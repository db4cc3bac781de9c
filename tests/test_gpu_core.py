"""The drop-in symbols' preparation (csrc/core_prep.cu) at the edges of its tiles
of 256 block-rows, with more tiles than a CTA adds up itself, without blocks,
and with the matrix deciding for each of the three kernels.  Every result is the
oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rows(n, seed, wide=False, dense_at=None):
    """About three neighbouring values per row near the diagonal (wide: eight
    of nine columns), every fifth row empty; one row of 1500 values: no row
    kernel."""
    rng = np.random.default_rng(seed)
    ncols = max(n, 2000)
    lens = np.full(n, 8 if wide else 3)
    lens[::5] = 0
    first = np.minimum(np.arange(n), ncols - 9)
    if dense_at is not None:
        lens[dense_at], first[dense_at] = 1500, 0
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colidx = np.repeat(first, lens) + np.arange(rowptr[-1]) - np.repeat(rowptr[:-1], lens)
    return rowptr, colidx.astype(np.int32), rng.uniform(-1, 1, rowptr[-1]), ncols


def check(r, csr, dt):
    rowptr, colidx, vals, ncols = csr
    n = len(rowptr) - 1
    vals = vals.astype(dt)
    ob, oh, ov = oracle.csr_to_beta(r, rowptr, colidx, vals)
    x, y0 = M.x_vector(ncols, 1, dt), M.x_vector(n, 2, dt)
    f = oracle.beta_spmv_f64 if dt == np.float64 else oracle.beta_spmv_f32
    want = f(r, n, ob, oh, ov, x, y0.copy())
    y = dev(y0)
    S.core_spmv(r, n, dev(ob), dev(oh), dev(ov), dev(x), y)
    torch.cuda.synchronize()
    assert y.cpu().numpy().tobytes() == want.tobytes(), n


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_tile_edges_equal_oracle(cuda, r, dt):
    for nbr in (1, 2, 255, 256, 257, 512, 767):
        for n in {nbr * r, nbr * r - r + 1}:
            check(r, rows(n, nbr), dt)
            check(r, rows(n, nbr, wide=True), dt)
            check(r, rows(n, nbr, dense_at=n - 1), dt)
    check(r, rows(700 * r, 3, dense_at=512 * r), dt)


@pytest.mark.parametrize("dense_at", [None, 2_000_000])
def test_many_tiles_equal_oracle(cuda, dense_at):
    check(1, rows(2_200_001, 5, dense_at=dense_at), np.float64)  # 8594 tiles


def test_calls_in_order_and_captured(cuda):
    """Calls on one stream, eagerly and replayed: each reads what the one
    before it wrote."""
    rowptr, colidx, vals, ncols = rows(3000, 8)
    ob, oh, ov = oracle.csr_to_beta(4, rowptr, colidx, vals)
    x0 = M.x_vector(ncols, 3)
    want = oracle.beta_spmv_f64(4, 3000, ob, oh, ov, x0, np.zeros(3000))
    want = oracle.beta_spmv_f64(4, 3000, ob, oh, ov, want, np.zeros(3000))
    a, x, t, y = (dev(ob), dev(oh), dev(ov)), dev(x0), dev(np.zeros(3000)), dev(np.zeros(3000))

    def chain():
        t.zero_()
        y.zero_()
        S.core_spmv(4, 3000, *a, x, t)
        S.core_spmv(4, 3000, *a, t, y)

    for _ in range(20):
        chain()
    torch.cuda.synchronize()
    assert y.cpu().numpy().tobytes() == want.tobytes()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain()
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        chain()
    y.fill_(5.0)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert y.cpu().numpy().tobytes() == want.tobytes()
