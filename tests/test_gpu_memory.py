"""Handle buffers (csrc/memory.cu): a release waits for the products that still
run on other streams, also beside an open capture."""
import time

import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S
from spc5_b200 import matrices as M

pytestmark = pytest.mark.gpu

SLEEP_CYCLES = 400_000_000  # about 0.2 s


@pytest.mark.parametrize("capture", [None, "global", "relaxed"])
@pytest.mark.parametrize("csr", [M.poisson2d(40), M.powerlaw(3000, seed=3)], ids=["rows", "plan"])
def test_release_waits_for_a_running_product(cuda, csr, capture):
    ob, oh, ov = oracle.csr_to_beta(1, csr.rowptr, csr.colidx, csr.values)
    x0 = M.x_vector(csr.ncols, 1)
    want = oracle.beta_spmv_f64(1, csr.nrows, ob, oh, ov, x0, np.zeros(csr.nrows))
    x, y, z = torch.from_numpy(x0).cuda(), torch.zeros(csr.nrows, dtype=torch.float64, device="cuda"), \
        torch.zeros(4, device="cuda")
    side = torch.cuda.Stream()
    m = S.csr_matrix(csr.rowptr, csr.colidx, csr.values, csr.ncols)
    S.CSR_to_SPC5(m, S.FORMAT_OF_R[1])
    S.SPC5_Spmv(m, x, torch.zeros_like(y))  # the kernels are loaded before a capture
    torch.cuda.synchronize()
    begin = time.perf_counter()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP_CYCLES)
    side.synchronize()
    sleep = time.perf_counter() - begin

    def release():
        """Destroys the handle while its product waits behind the sleep; seconds until the return."""
        nonlocal m
        begin = time.perf_counter()
        with torch.cuda.stream(side):
            torch.cuda._sleep(SLEEP_CYCLES)
            S.SPC5_Spmv(m, x, y, stream=side)
        m = None
        return time.perf_counter() - begin

    if capture is None:
        took = release()
    else:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, capture_error_mode=capture):
            z += 1
            took = release()
            z += 1
        graph.replay()
    torch.cuda.synchronize()
    assert took > 0.8 * sleep, (took, sleep)
    assert y.cpu().numpy().tobytes() == want.tobytes()
    assert capture is None or z[0].item() == 2.0
