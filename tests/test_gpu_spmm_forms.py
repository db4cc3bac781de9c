"""The staged SpMM's forms (csrc/spmm_rows.cu spmm_columns, spmv_columns): long rows of
full and of nearly empty blocks, where a chunk holds few sub-rows, for every number of
right-hand sides around the passes' widths, alone and batched.  Columns are the
oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def unknowns(side, d):
    """The 27-point grid with d coupled unknowns per node."""
    g = M.stencil27(side)
    n = len(g.rowptr) - 1
    rows = np.repeat(np.arange(n), np.diff(g.rowptr))
    a = np.arange(d)
    r = np.broadcast_to(rows[:, None, None] * d + a[None, :, None], (len(rows), d, d)).reshape(-1)
    c = np.broadcast_to(g.colidx[:, None, None].astype(np.int64) * d + a[None, None, :], (len(rows), d, d)).reshape(-1)
    return M.from_coo(n * d, n * d, r, c, np.random.default_rng(d).uniform(-1, 1, r.size))


def scattered(n, per_row, seed):
    rng = np.random.default_rng(seed)
    cols = np.stack([np.sort(rng.choice(6000, per_row, replace=False)) for _ in range(n)])
    return M.from_coo(n, 6000, np.repeat(np.arange(n), per_row), cols.reshape(-1), rng.uniform(-1, 1, n * per_row))


CASES = {"3 unknowns": unknowns(6, 3), "6 unknowns": unknowns(4, 6), "dense band": M.banded(400, 60, 1.0, seed=1),
         "wide band": M.banded(700, 200, 0.1, seed=2), "scattered": scattered(130, 40, 3), "long": scattered(60, 90, 4)}


@pytest.mark.parametrize("tag", ["f64", "f32", "f32 mixed", "mixed8"])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_every_form_equals_oracle(cuda, r, tag):
    dt, yt = (np.float64 if tag == "f64" else np.float32), (np.float32 if tag == "f32" else np.float64)
    mixed = "mixed" in tag
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "f32 mixed": oracle.beta_spmv_mixed,
         "mixed8": oracle.beta_spmv_mixed8}[tag]
    spmm = S.SPC5_Spmm_mixed if mixed else S.SPC5_Spmm
    for name, csr in CASES.items():
        v = csr.values.astype(dt)
        arrays = (oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta)(r, csr.rowptr, csr.colidx, v)
        m = S.csr_matrix(csr.rowptr, csr.colidx, v, csr.ncols, value_type=S.F32_V8 if tag == "mixed8" else None)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        X = np.stack([M.x_vector(csr.ncols, 10 + j, dt) for j in range(17)], axis=1)
        Y = np.stack([M.x_vector(csr.nrows, 40 + j, yt) for j in range(17)], axis=1)
        want = np.stack([f(r, csr.nrows, *arrays, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y[:, j]).copy())
                         for j in range(17)], axis=1)
        for k in (1, 2, 3, 4, 5, 8, 12, 16, 17):
            y = torch.from_numpy(np.ascontiguousarray(Y[:, :k])).cuda()
            spmm(m, torch.from_numpy(np.ascontiguousarray(X[:, :k])).cuda(), y)
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, :k]).tobytes(), (name, k)
        ks = [1, 3, 4, 16]
        xs = [torch.from_numpy(np.ascontiguousarray(X[:, :k])).cuda() for k in ks]
        ys = [torch.from_numpy(np.ascontiguousarray(Y[:, :k])).cuda() for k in ks]
        batch = S.Batch([m] * len(ks), xs, ys, mixed=mixed)
        batch.launch()
        torch.cuda.synchronize()
        for k, y in zip(ks, ys):
            assert y.cpu().numpy().tobytes() == np.ascontiguousarray(want[:, :k]).tobytes(), (name, k, "batch")
