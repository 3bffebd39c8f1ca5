"""Generic FP64 programs whose rows leave the most points per thread with idle
rows or uneven CTAs: whichever number of rows a thread takes, UHS_ARITH_EXACT
ends bit-identical to the serial loops."""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import run_gpu, run_oracle
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu

EXACT = uhs.RunParams(arith=uhs.UHS_ARITH_EXACT)


@pytest.mark.parametrize("rank,r,kind,interior", [(2, 3, "box", (217, 2528)), (2, 2, "box", (659, 479)),
                                                  (2, 1, "star", (2601, 237)), (2, 1, "box", (130, 1926)),
                                                  (3, 2, "box", (52, 37, 213)), (3, 3, "star", (116, 77, 257)),
                                                  (3, 1, "box", (164, 21, 252)), (3, 1, "star", (41, 33, 400))])
def test_exact_on_uneven_rows(cuda, rank, r, kind, interior):
    st, a0 = random_case(rank, r, kind, interior, 2, 91)
    ra, rb = run_oracle(st, a0)
    ga, gb = run_gpu(st, a0, EXACT)
    assert np.array_equal(ga.view(np.uint64), ra.view(np.uint64))
    assert np.array_equal(gb.view(np.uint64), rb.view(np.uint64))
