"""SpMM over the sorted plan's streams with one and two right-hand sides, which run as
an SpMV each (two: from 4M values in the streams on).  Columns are the oracle's bit
for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def skewed(n, seed):
    """Rows of 30 to 90 values, every 5000th of 2500, every seventh of 9."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(30, 91, n)
    lens[::5000] = 2500
    lens[3::7] = 9
    ncols = 40_000
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    step = ncols // lens
    first = rng.integers(0, ncols - (lens - 1) * step)
    j = np.arange(rowptr[-1]) - np.repeat(rowptr[:-1], lens)
    colidx = np.repeat(first, lens) + j * np.repeat(step, lens)
    return rowptr, colidx.astype(np.int32), rng.uniform(-1, 1, rowptr[-1]), ncols


@pytest.mark.parametrize("n", [3_000, 90_000])  # about 0.16M and 4.7M values in the streams
@pytest.mark.parametrize("tag", ["f64", "f32", "mixed8"])
def test_one_and_two_columns_equal_oracle(cuda, tag, n):
    rowptr, colidx, vals, ncols = skewed(n, n)
    dt, yt = (np.float64 if tag == "f64" else np.float32), (np.float32 if tag == "f32" else np.float64)
    vals = vals.astype(dt)
    r = 2
    arrays = (oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta)(r, rowptr, colidx, vals)
    m = S.csr_matrix(rowptr, colidx, vals, ncols, value_type=S.F32_V8 if tag == "mixed8" else None)
    m.set_kernel(S.KERNEL_SORTED)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "mixed8": oracle.beta_spmv_mixed8}[tag]
    spmm = S.SPC5_Spmm_mixed if tag == "mixed8" else S.SPC5_Spmm
    X = np.stack([M.x_vector(ncols, 10 + j, dt) for j in range(5)], axis=1)
    Y = np.stack([M.x_vector(n, 40 + j, yt) for j in range(5)], axis=1)
    want = np.stack([f(r, n, *arrays, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y[:, j]).copy())
                     for j in range(5)], axis=1)
    Xd = torch.from_numpy(X).cuda()
    for a, b in ((0, 1), (0, 2), (3, 5), (1, 2)):
        Yd = torch.from_numpy(Y).cuda()
        spmm(m, Xd[:, a:b], Yd[:, a:b])  # leading dimension 5
        contiguous = torch.from_numpy(np.ascontiguousarray(Y[:, a:b])).cuda()
        spmm(m, Xd[:, a:b].contiguous(), contiguous)
        torch.cuda.synchronize()
        got = Yd.cpu().numpy()
        for j in range(5):
            assert got[:, j].tobytes() == (want if a <= j < b else Y)[:, j].tobytes(), (a, b, j)
        assert contiguous.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, a:b]).tobytes()
