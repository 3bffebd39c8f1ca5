"""The generic kernel's points per thread (1, 2, 4; 8 in 2D) and chunk lengths
follow the grid's size: sizes on both sides of each choice, one-sided and
two-sided programs, domains at the grid's edge, EXACT against the oracle bit
for bit (FP64) and FP32 within its bar."""
import numpy as np
import pytest

import oracle
import uxxxxxxxxh_gb300 as uhs
from gpu_util import run_gpu, run_oracle
from uxxxxxxxxh_gb300.stencil import Stencil
from uxxxxxxxxh_gb300.workloads import normalised, splitmix_uniform

pytestmark = pytest.mark.gpu


def _program(rank, interior, offs, T):
    """Offsets `offs` on a grid with only the halo they need."""
    lo = [max(0, -min(o[i] for o in offs)) for i in range(3)]
    hi = [max(0, max(o[i] for o in offs)) for i in range(3)]
    inner = [1] * (3 - rank) + list(interior)
    coefs = normalised(splitmix_uniform(7, len(offs)) + 0.05)
    return Stencil(name="generic", rank=rank, sizes=tuple(n + a + b for n, a, b in zip(inner, lo, hi)), lb=tuple(lo),
                   ub=tuple(n + a for n, a in zip(inner, lo)),
                   terms=[(*o, c) for o, c in zip(offs, coefs)], iterations=T)


UP2 = [(0, 0, 0), (0, -1, 0), (0, -2, 0), (0, 0, -1), (0, 0, -2)]
UP3 = UP2 + [(-1, 0, 0), (-2, 0, 0)]
DOWN3 = [(0, 0, 0), (1, 0, 0), (0, 3, 1), (0, 0, 4), (2, -1, 0)]
SIDES = [(0, 0, 0), (-1, 2, 0), (1, 0, -3), (0, -1, 1)]


@pytest.mark.parametrize("rank,interior,offs", [
    (2, (5, 40), UP2), (2, (63, 2000), UP2), (2, (330, 2000), UP2), (2, (317, 2051), UP2),
    (3, (3, 9, 33), UP3), (3, (20, 33, 65), UP3), (3, (48, 100, 400), UP3), (3, (41, 90, 211), DOWN3),
    (3, (17, 131, 333), SIDES), (3, (8, 300, 290), DOWN3),
])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_generic_program(cuda, rank, interior, offs, dtype):
    import torch
    st = _program(rank, interior, offs, 2)
    a0 = 2.0 * splitmix_uniform(9, int(np.prod(st.sizes))) - 1.0
    b0 = 2.0 * splitmix_uniform(10, a0.size) - 1.0
    if dtype == "f64":
        ra, rb = run_oracle(st, a0, b0)
        ga, gb = run_gpu(st, a0, uhs.RunParams(arith=uhs.UHS_ARITH_EXACT), b0)
        assert np.array_equal(ra.view(np.uint64), ga.view(np.uint64))
        assert np.array_equal(rb.view(np.uint64), gb.view(np.uint64))
    else:
        st = st.with_(dtype=uhs.UHS_F32)
        a0, b0 = a0.astype(np.float32), b0.astype(np.float32)
        ra, rb = run_oracle(st, a0.astype(np.float64), b0.astype(np.float64))
        ga, gb = run_gpu(st, a0, uhs.RunParams(kernel=uhs.UHS_KERNEL_GENERIC), b0, dtype=torch.float32)
        assert oracle.error(st, ra, ga.astype(np.float64))["l2_rel"] <= 1e-6
        assert oracle.error(st, rb, gb.astype(np.float64))["l2_rel"] <= 1e-6
