"""How the passes over block-rows of a conversion are cut (csrc/convert.cu
block_rows_per_warp): numbers of block-rows on both sides of every cut, with long
block-rows at the edges.  Arrays are the oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
import spc5_b200 as S

from test_gpu_split import mixed_rows, sms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [2, 4, 8])
@pytest.mark.parametrize("per", [1, 2, 8, 32])
def test_conversion_equals_oracle(cuda, r, per):
    """`per` block-rows per warp, from this many block-rows on."""
    for nbr in (32 * sms() * per - 1, 32 * sms() * per):
        n = nbr * r - 1
        rowptr, colidx, vals, ncols = mixed_rows(n, nbr + r, [0, per * r - 1, per * r, 33 * r, n // 2, n - 2])
        m = S.csr_matrix(rowptr, colidx, vals, ncols)
        S.CSR_to_SPC5(m, S.FORMAT_OF_R[r])
        for a, b in zip(m.arrays(), oracle.csr_to_beta(r, rowptr, colidx, vals)):
            assert np.asarray(a).tobytes() == np.asarray(b).tobytes(), nbr
