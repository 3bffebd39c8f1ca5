"""Grids too small to fill the GPU: their sweeps run in chunks of a few planes
(down to 2, shorter than the halo of radius 3), each launched into the slots
of the one before.  Many dependent sweeps on extents that leave ragged last
chunks and tiles, against the oracle at the element type's bar, through the
streaming kernel (kernel = STREAM)."""
import numpy as np
import pytest

import oracle
import uxxxxxxxxh_gb300 as uhs
from gpu_util import assert_f64_close, assert_halo_exact, run_gpu, run_oracle
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("rank,r,kind,interior", [
    (2, 1, "star", (2, 3)), (2, 1, "star", (255, 257)), (2, 3, "star", (129, 511)), (2, 2, "box", (67, 300)),
    (3, 1, "star", (3, 17, 33)), (3, 1, "star", (65, 63, 66)), (3, 3, "star", (25, 31, 70)), (3, 1, "box", (13, 16, 35)),
])
def test_short_chunks_of_dependent_sweeps(cuda, rank, r, kind, interior, dtype):
    import torch
    st, a0 = random_case(rank, r, kind, interior, 24, 500 + 10 * rank + r)
    p = uhs.RunParams(kernel=uhs.UHS_KERNEL_STREAM)
    if dtype == "f32":
        st, a0 = st.with_(dtype=uhs.UHS_F32), a0.astype(np.float32)
        ra, rb = run_oracle(st, a0.astype(np.float64))
        ga, gb = run_gpu(st, a0, p, dtype=torch.float32)
        assert oracle.error(st, ra, ga.astype(np.float64))["l2_rel"] <= 1e-6
        assert oracle.error(st, rb, gb.astype(np.float64))["l2_rel"] <= 1e-6
    else:
        ra, rb = run_oracle(st, a0)
        ga, gb = run_gpu(st, a0, p)
        assert_f64_close(st, ra, ga)
        assert_f64_close(st, rb, gb)
        assert_halo_exact(st, ra, ga)
        assert_halo_exact(st, rb, gb)
