"""Admission of matrices with the sorted plan to the request loop."""
import numpy as np
import pytest
import torch

import spc5_b200 as S
from spc5_b200 import matrices as M

from test_gpu_serve import converted, solo

pytestmark = pytest.mark.gpu


def test_plan_gives_way_to_the_budget(cuda):
    """A matrix that fits the budget only without its sorted plan is served from its
    beta arrays; one byte less and it is refused and left as it is."""
    csr = M.powerlaw(20000, seed=9)
    m = converted(csr, np.float64, 1)
    assert m.kernel == S.KERNEL_SORTED
    with_plan = m.info().device_bytes
    m.set_kernel(S.KERNEL_GROUPS)
    beta = m.info().device_bytes
    m.set_kernel(S.KERNEL_AUTO)
    assert m.kernel == S.KERNEL_SORTED and m.info().device_bytes == with_plan > beta
    staging = 2 * 4 * 8 * (csr.nrows + csr.ncols)
    tight = S.Server(slots=2, max_k=4, hbm_budget=beta + staging - 1)
    with pytest.raises(S.SPC5Error) as e:
        tight.add_matrix(m)
    assert e.value.status == 3 and m.kernel == S.KERNEL_SORTED
    tight.close()
    roomy = S.Server(slots=2, max_k=4, hbm_budget=with_plan + staging)
    roomy.add_matrix(m)
    assert m.kernel == S.KERNEL_SORTED
    roomy.close()
    xs = [torch.from_numpy(M.x_vector(csr.ncols, 50 + q)).cuda() for q in range(9)]
    want = [solo(m, x, False) for x in xs]
    fits = S.Server(slots=2, max_k=4, hbm_budget=beta + staging)
    i = fits.add_matrix(m)
    assert m.kernel == S.KERNEL_GROUPS and fits.stats()["resident_bytes"] == beta
    ys = [torch.empty(csr.nrows, dtype=torch.float64, device="cuda") for _ in xs]
    torch.cuda.synchronize()
    for rid in [fits.submit(i, x, y) for x, y in zip(xs, ys)]:
        fits.wait(rid)
    for y, w in zip(ys, want):
        assert y.cpu().numpy().tobytes() == w.cpu().numpy().tobytes()
    fits.close()
