"""Device memory of a handle with the sorted plan (csrc/plan.cu): one copy of the
values, an x index each, and little more; a batch adds exactly the reference-order
copy.  The bound is counted from the layout: what a second copy of the values would add
does not fit under it."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vt", [S.F64, S.F32, S.F32_V8])
@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_one_copy_of_the_values(cuda, r, vt):
    dt = np.float64 if vt == S.F64 else np.float32
    mixed, vbytes, vs = vt == S.F32_V8, 8 if vt == S.F64 else 4, 16 if vt == S.F32 else 8
    for csr in (M.powerlaw(60_000, seed=21), M.dense(2048)):
        m = S.csr_matrix(csr.rowptr, csr.colidx, csr.values.astype(dt), csr.ncols, value_type=S.F32_V8 if mixed else None)
        m.set_kernel(S.KERNEL_SORTED)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        assert m.kernel == S.KERNEL_SORTED
        inf = m.info()
        nbr = (csr.nrows + r - 1) // r
        conv = oracle.csr_to_beta_v8 if mixed else oracle.csr_to_beta
        brptr, headers, _ = conv(r, csr.rowptr, csr.colidx, csr.values.astype(dt))
        mb = 2 if vs == 16 else 1
        masks = np.frombuffer(headers.tobytes(), np.uint8).reshape(int(brptr[-1]), 4 + r * mb)[:, 4:]
        subrows = np.count_nonzero(np.ascontiguousarray(masks).view(f"u{mb}"))  # with a value
        # a mask word per step of 32 / vs rows (neighbours of the sorted order: nearly
        # one length), 10 bytes per row (order, key, chains), two offsets per block-row;
        # 256 KB for the slabs' offsets, their padding and the kernels' partitions
        steps = 1.25 * subrows * vs / 32
        bound = inf.header_bytes + csr.nnz * (vbytes + 4) + 4 * steps + 10 * csr.nrows + 8 * (nbr + 1) + (256 << 10)
        assert bound < inf.header_bytes + csr.nnz * (2 * vbytes + 4)
        assert inf.device_bytes <= bound, (csr.name, inf.device_bytes, bound)
        x = torch.zeros(csr.ncols, 1, dtype=torch.float64 if vt == S.F64 else torch.float32, device="cuda")
        y = torch.zeros(csr.nrows, 1, dtype=torch.float32 if vt == S.F32 else torch.float64, device="cuda")
        batch = S.Batch([m], [x], [y], mixed=mixed)
        assert m.info().device_bytes == inf.device_bytes + csr.nnz * vbytes, csr.name
        del batch
