"""How the passes over block-rows are cut into parts (csrc/core_prep.cu part_rows): sizes on both sides of every cut, with long
block-rows at the edges.  Arrays and results are the oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def mixed_rows(n, seed, long_at):
    """Rows of 0 .. 3 values near the diagonal; 70 and 600 values at the given rows."""
    rng = np.random.default_rng(seed)
    ncols = max(n, 2000)
    lens = rng.integers(0, 4, n)
    lens[[a for a in long_at if a < n]] = 70
    lens[[a + 1 for a in long_at if a + 1 < n]] = 600
    first = np.minimum(np.arange(n), ncols - 600)
    rowptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    colidx = np.repeat(first, lens) + np.arange(rowptr[-1]) - np.repeat(rowptr[:-1], lens)
    return rowptr, colidx.astype(np.int32), rng.uniform(-1, 1, rowptr[-1]), ncols


@pytest.mark.parametrize("r, dt", [(1, np.float64), (8, np.float32)])
@pytest.mark.parametrize("rows", [16, 64, 256])
def test_dropin_parts_equal_oracle(cuda, rows, r, dt):
    """`rows` block-rows per part (16, 64, 256) below and above the number of block-rows
    that makes 2 * SMs of them."""
    edge = (2 * sms() - 1) * rows
    for nbr in (edge - 1, edge, edge + rows - 1):
        n = nbr * r - r // 2
        for tail in (0, 1500):  # a last row of 1500 values: no row kernel
            rowptr, colidx, vals, ncols = mixed_rows(n, nbr, [rows * r - 1, (rows + 1) * r])
            if tail:
                rowptr[-1] += tail - (rowptr[-1] - rowptr[-2])
                colidx = np.concatenate([colidx[:rowptr[-2]], np.arange(tail, dtype=np.int32)])
                vals = np.resize(vals, rowptr[-1])
            ob, oh, ov = oracle.csr_to_beta(r, rowptr, colidx, vals.astype(dt))
            x, y0 = M.x_vector(ncols, 1, dt), M.x_vector(n, 2, dt)
            f = oracle.beta_spmv_f64 if dt == np.float64 else oracle.beta_spmv_f32
            want = f(r, n, ob, oh, ov, x, y0.copy())
            b, h, v, xd, y = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (ob, oh, ov, x, y0))
            S.core_spmv(r, n, b, h, v, xd, y)
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == want.tobytes(), (nbr, tail)
