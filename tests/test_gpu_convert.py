"""Conversion kernels (csrc/convert.cu): the r = 1 windows of 32 entries, block-rows
walked by a lane or by a warp, and the plan built from them.  Arrays equal the
oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def rows_of(lengths, ncols, step, seed):
    """Rows of the given lengths; consecutive columns lie 1 .. step apart."""
    rng = np.random.default_rng(seed)
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    cols = []
    for n in lengths:
        c = np.cumsum(rng.integers(1, step + 1, n)) - 1
        c += rng.integers(0, max(1, ncols - (int(c[-1]) if n else 0)))
        cols.append(c)
    colidx = np.concatenate(cols).astype(np.int32) if cols else np.zeros(0, np.int32)
    assert colidx.size == 0 or colidx.max() < ncols
    return rowptr, colidx, rng.uniform(-1, 1, colidx.size)


EDGES = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 0, 0, 95, 96, 97, 130, 1, 1, 1, 500, 0, 33, 5, 3000, 2]


@pytest.mark.parametrize("tag", ["f64", "f32", "mixed8"])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
@pytest.mark.parametrize("step", [1, 3, 9, 40])
def test_conversion_equals_oracle(cuda, tag, r, step):
    dt = np.float64 if tag == "f64" else np.float32
    conv = oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta
    for lengths in (EDGES, [0] * 40, [1] * 33, EDGES[::-1] * 3, [31] * 70, [4000] * 3):
        rowptr, colidx, vals = rows_of(lengths, 200_000, step, len(lengths) + step)
        vals = vals.astype(dt)
        want = conv(r, rowptr, colidx, vals)
        m = S.csr_matrix(rowptr, colidx, vals, 200_000, value_type=S.F32_V8 if tag == "mixed8" else None)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        got = m.arrays()
        for a, b in zip(got, want):
            assert np.asarray(a).tobytes() == np.asarray(b).tobytes(), (len(lengths), step)


def test_release_leaves_a_relaxed_capture_alone(cuda):
    c = M.poisson2d(20)

    def make():
        m = S.csr_matrix(c.rowptr, c.colidx, c.values, c.ncols)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[1])
        return m

    z, m, side = torch.zeros(4, device="cuda"), make(), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        z += 1
        del m
        with torch.cuda.stream(side):
            make()
        z += 1
    graph.replay()
    torch.cuda.synchronize()
    assert z[0].item() == 2.0


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 4099])
def test_malformed_csr_is_refused(cuda, n):
    """Rows of two entries whose columns fall from one row to the next (allowed)
    and, one fault at a time, inside a row (not); entries on both sides of the
    quads that a thread reads, the last ones among them."""
    rowptr = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    colidx = np.tile(np.array([3, 7], np.int32), n)
    vals = np.ones(2 * n)

    def refused(rp, ci):
        try:
            S.csr_matrix(rp, ci, vals, 8)
        except S.SPC5Error:
            return True
        return False

    assert not refused(rowptr, colidx)
    single = np.concatenate([[0], np.arange(1, 2 * n + 1)]).astype(np.int32)
    assert not refused(single, colidx[::-1].copy())
    for row in {0, 1, n // 2, n - 1} & set(range(n)):
        for at, value in ((2 * row, 7), (2 * row, 8), (2 * row + 1, 3), (2 * row + 1, 8), (2 * row + 1, -1), (2 * row, -1)):
            bad = colidx.copy()
            bad[at] = value
            assert refused(rowptr, bad), (row, at, value)
        bad = rowptr.copy()
        bad[row + 1] += 2 * n + 1
        assert refused(bad, colidx)
        bad = rowptr.copy()
        bad[row] = -1
        assert refused(bad, colidx)
