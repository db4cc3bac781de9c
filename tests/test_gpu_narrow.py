"""The row kernel's narrow instantiation (csrc/spmv_rows.cu): matrices whose
sub-row masks span few columns, with wider masks strewn in (a step that meets
one leaves the window), windows that wrap around a block's last column at r = 8,
empty rows and last block-rows that are not full.  Every result is the oracle's
bit for bit, through the handle and through the drop-in symbols."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def strewn(n, every, seed, shift=0):
    """Three neighbouring columns per row near the diagonal and near two
    far ones; one row in `every` has a run of 11; some rows are empty."""
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i in range(n):
        if i % 37 == 5:
            continue
        take = set()
        for base in (i + shift, i // 2, n - 1 - i // 3):
            for d in (-1, 0, 1):
                if rng.random() < 0.9:
                    take.add(base + d)
        if every and i % every == 0:
            take |= set(range(i // 2, i // 2 + 11))
        take = sorted(c for c in take if 0 <= c < n)
        rows += [i] * len(take)
        cols += take
    return M.from_coo(n, n, rows, cols, rng.uniform(-1, 1, len(rows)), name=f"strewn_{n}_{every}")


def cases():
    yield M.stencil27(13)          # block-rows across grid lines
    yield M.poisson2d(61)
    yield strewn(3001, 0, 1)
    yield strewn(3001, 97, 2)      # a wide mask in some chunks only
    yield strewn(2999, 11, 3, shift=6)


@pytest.mark.parametrize("tag", ["f64", "f32", "mixed", "mixed8"])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_narrow_masks_equal_oracle(cuda, tag, r):
    mixed = tag.startswith("mixed")
    dt = np.float64 if tag == "f64" else np.float32
    yt = np.float32 if tag == "f32" else np.float64
    f = {"f64": oracle.beta_spmv_f64, "f32": oracle.beta_spmv_f32, "mixed": oracle.beta_spmv_mixed,
         "mixed8": oracle.beta_spmv_mixed8}[tag]
    conv = oracle.csr_to_beta_v8 if tag == "mixed8" else oracle.csr_to_beta
    for csr in cases():
        vals = csr.values.astype(dt)
        ob, oh, ov = conv(r, csr.rowptr, csr.colidx, vals)
        x, y0 = M.x_vector(csr.ncols, 5, dt), M.x_vector(csr.nrows, 6, yt)
        yo = f(r, csr.nrows, ob, oh, ov, x, y0.copy())
        m = S.csr_matrix(csr.rowptr, csr.colidx, vals, csr.ncols, value_type=S.F32_V8 if tag == "mixed8" else None)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        assert m.kernel == S.KERNEL_ROWS
        y = dev(y0)
        (S.SPC5_Spmv_mixed if mixed else S.SPC5_Spmv)(m, dev(x), y)
        torch.cuda.synchronize()
        assert y.cpu().numpy().tobytes() == yo.tobytes(), csr.name
        if not mixed:
            y = dev(y0)
            S.core_spmv(r, csr.nrows, dev(ob), dev(oh), dev(ov), dev(x), y)
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == yo.tobytes(), (csr.name, "drop-in")


@pytest.mark.parametrize("tag", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("r", [1, 4, 8])
def test_spmm_waves_equal_spmv(cuda, tag, r):
    """Parts of several block-rows, long and short, whose boundaries the SpMM
    kernels interpolate: every column is the SpMV's, bit for bit."""
    dt = np.float64 if tag == "f64" else np.float32
    yt = torch.float64 if tag != "f32" else torch.float32
    csr = strewn(40003, 1009, 9)
    m = S.csr_matrix(csr.rowptr, csr.colidx, csr.values.astype(dt), csr.ncols)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
    assert m.kernel == S.KERNEL_ROWS
    spmv, spmm = (S.SPC5_Spmv_mixed, S.SPC5_Spmm_mixed) if tag == "mixed" else (S.SPC5_Spmv, S.SPC5_Spmm)
    rng = np.random.default_rng(2)
    x = dev(rng.uniform(-1, 1, (csr.ncols, 7)).astype(dt))
    want = torch.zeros(csr.nrows, 7, dtype=yt, device="cuda")
    for j in range(7):
        y = torch.zeros(csr.nrows, dtype=yt, device="cuda")
        spmv(m, x[:, j].contiguous(), y)
        want[:, j] = y
    for k in (2, 3, 5, 7):
        got = torch.zeros(csr.nrows, k, dtype=yt, device="cuda")
        spmm(m, x[:, :k].contiguous(), got)
        assert torch.equal(got, want[:, :k])
