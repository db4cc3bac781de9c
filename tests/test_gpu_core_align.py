"""Headers of the drop-in symbols that are 4-byte but not 16-byte aligned: the row
kernels stage 16 bytes at a time, so the group kernel runs.  Every result is the
oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_headers_at_four_byte_offsets(cuda, r, dt):
    for csr in (M.stencil27(9), M.banded(501, 40, 0.3, seed=2), M.powerlaw(2000, seed=5), M.dense(700)):
        ob, oh, ov = oracle.csr_to_beta(r, csr.rowptr, csr.colidx, csr.values.astype(dt))
        x, y0 = M.x_vector(csr.ncols, 1, dt), M.x_vector(csr.nrows, 2, dt)
        f = oracle.beta_spmv_f64 if dt == np.float64 else oracle.beta_spmv_f32
        want = f(r, csr.nrows, ob, oh, ov, x, y0.copy())
        b, v, xd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (ob, ov, x))
        room = torch.zeros(len(oh) + 16, dtype=torch.uint8, device="cuda")
        for at in (0, 4, 8, 12):
            h = room[at:at + len(oh)]
            h.copy_(torch.from_numpy(oh))
            assert h.data_ptr() % 16 == at
            y = torch.from_numpy(y0).cuda()
            S.core_spmv(r, csr.nrows, b, h, v, xd, y)
            torch.cuda.synchronize()
            assert y.cpu().numpy().tobytes() == want.tobytes(), (csr.name, at)


def test_other_alignments_are_refused(cuda):
    z = torch.zeros(64, dtype=torch.uint8, device="cuda")
    br = torch.zeros(2, dtype=torch.int32, device="cuda")
    v = torch.zeros(4, dtype=torch.float64, device="cuda")
    for headers, values in ((z[1:], v), (z[2:], v), (z, v[1:])):
        with pytest.raises(S.SPC5Error) as e:
            S.core_spmv(1, 1, br, headers, values, v, v)
        assert e.value.status == 1
