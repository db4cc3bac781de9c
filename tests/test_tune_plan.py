"""The autotuner's model on sorted-plan matrices: the plan stores rows, so its estimate
does not depend on r, r = 1 is picked (the cheapest conversion), and the estimate is
near the measured time."""
import json

import numpy as np
import pytest

import spc5_b200 as S
from spc5_b200 import matrices as M
from spc5_b200 import tune_fit as T


def test_fit_plan_recovers_its_coefficients(tmp_path):
    rows = []
    for vt in range(3):
        for r in T.RS:
            for nnz in (1e6, 3e6, 1e7, 3e7):
                rows.append({"vt": vt, "r": r, "plan": 1, "nnz": nnz, "us": 20.0 + vt + 4e-6 * (1 + vt) * nnz})
            rows.append({"vt": vt, "r": r, "plan": 0, "nnz": 1e6, "us": 1e9})  # ignored
    path = tmp_path / "plan.jsonl"
    path.write_text("\n".join(json.dumps(p) for p in rows))
    got = T.fit_plan(str(path))
    for vt in range(3):
        assert np.allclose(got[vt], [20.0 + vt, 4e-6 * (1 + vt)], rtol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("vt", [S.F64, S.F32, S.F32_V8])
def test_plan_estimates(cuda, vt):
    import torch
    dt = np.float64 if vt == S.F64 else np.float32
    csr = M.powerlaw(1_000_000, seed=44)
    new = lambda: S.csr_matrix(csr.rowptr, csr.colidx, csr.values.astype(dt), csr.ncols,
                               value_type=S.F32_V8 if vt == S.F32_V8 else None)
    t = S.autotune(new(), S.TUNE_MODEL)
    assert t["r"] == 1 and len(set(t["est_us"].values())) == 1, t
    m = new()
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[1])
    assert m.kernel == S.KERNEL_SORTED
    x = torch.from_numpy(M.x_vector(csr.ncols, 1, dt)).cuda()
    y = torch.zeros(csr.nrows, dtype=torch.float32 if vt == S.F32 else torch.float64, device="cuda")
    f = S.SPC5_Spmv_mixed if vt == S.F32_V8 else S.SPC5_Spmv
    best = float("inf")
    for _ in range(4):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(20):
            f(m, x, y)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / 20)
    # the fit's own residual at this size is 0.8 to 1.0
    assert 0.6 <= t["est_us"][1] / best <= 1.5, (t["est_us"], best)
