"""The forms of the row kernel (csrc/spmv_rows.cu, rows_blocks.cuh narrow / deep):
matrices on both sides of each rule.  Results are the oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def csr(lengths, first, step, ncols, seed):
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    j = np.arange(rowptr[-1]) - np.repeat(rowptr[:-1], lengths)
    colidx = np.repeat(first, lengths) + step * j
    return rowptr, colidx.astype(np.int32), np.random.default_rng(seed).uniform(-1, 1, rowptr[-1]), ncols


def cases():
    n = 1001
    i = np.arange(n)
    yield "diagonal", csr(np.ones(n, int), i, 1, n, 1)                       # one value per block and sub-row
    yield "tridiagonal", csr(np.full(n, 3), i, 1, n + 2, 2)                  # three
    yield "far", csr(np.full(n, 2), i % 97, 400, 600, 3)                     # sub-rows alone in their blocks
    for name, m in (("poisson", M.poisson2d(37)), ("band", M.banded(900, 60, 0.1, seed=4)),
                    ("wide band", M.banded(900, 200, 0.1, seed=5)), ("dense band", M.banded(700, 40, 1.0, seed=6)),
                    ("long rows", M.banded(500, 240, 0.25, seed=7))):
        yield name, (m.rowptr, m.colidx, m.values, m.ncols)


@pytest.mark.parametrize("tag", ["f64", "f32", "f32 mixed", "mixed8"])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_every_form_equals_oracle(cuda, r, tag):
    dt, yt = (np.float64 if tag == "f64" else np.float32), (np.float32 if tag == "f32" else np.float64)
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "f32 mixed": oracle.beta_spmv_mixed,
         "mixed8": oracle.beta_spmv_mixed8}[tag]
    for name, (rowptr, colidx, vals, ncols) in cases():
        n = len(rowptr) - 1
        v = vals.astype(dt)
        arrays = (oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta)(r, rowptr, colidx, v)
        m = S.csr_matrix(rowptr, colidx, v, ncols, value_type=S.F32_V8 if tag == "mixed8" else None)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        assert m.kernel == S.KERNEL_ROWS or name == "long rows", name  # too long for r = 8
        x, y0 = M.x_vector(ncols, 1, dt), M.x_vector(n, 2, yt)
        want = f(r, n, *arrays, x, y0.copy())
        y, xd = torch.from_numpy(y0).cuda(), torch.from_numpy(x).cuda()
        (S.SPC5_Spmv_mixed if "mixed" in tag else S.SPC5_Spmv)(m, xd, y)
        torch.cuda.synchronize()
        assert y.cpu().numpy().tobytes() == want.tobytes(), name
        if "mixed" not in tag:  # the drop-in symbols choose between wide and narrow on the device
            y = torch.from_numpy(y0).cuda()
            b, h, w = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays)
            S.core_spmv(r, n, b, h, w, xd, y)
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == want.tobytes(), name
