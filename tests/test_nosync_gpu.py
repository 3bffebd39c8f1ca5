"""FP64 runs under UHS_ARITH_AUTO with UHS_FLAG_NO_SYNC wait for their range
scan alone: a run of many sweeps returns while the GPU is still sweeping, its
results (and a fallback to native FP64) are those of the same run with a wait."""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import to_dev
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu

QUIET = uhs.RunParams(flags=uhs.UHS_FLAG_NO_SYNC)


@pytest.mark.parametrize("rank,r,interior,T", [(3, 1, (20, 24, 37), 2), (3, 1, (20, 24, 37), 24), (2, 1, (90, 131), 1),
                                               (2, 2, (90, 131), 12), (3, 2, (129, 130, 131), 4)])
@pytest.mark.parametrize("wide", [False, True])
def test_results_without_a_wait(cuda, rank, r, interior, T, wide):
    import torch
    st, a0 = random_case(rank, r, "star", interior, T, 61)
    if wide:
        a0 = np.abs(a0) + 0.5
        a0[a0.size // 2:a0.size // 2 + 9] = 1e-60
    out = []
    for p in (None, QUIET):
        a, b = to_dev(a0, st), to_dev(a0, st)
        uhs.run(st, a, b, p)
        torch.cuda.synchronize()
        out.append((a, b))
    for x, y in zip(*out):
        assert torch.equal(x, y)


@pytest.mark.parametrize("rank,interior", [(3, (256, 256, 256)), (2, (1024, 1024))])
def test_returns_before_the_sweeps_end(cuda, rank, interior):
    import torch
    st, _ = random_case(rank, 1, "star", (4,) * rank, 800, 62)
    st = uhs.make_stencil("long", rank, interior, 1, uhs.star_offsets(rank, 1), [t[3] for t in st.terms],
                          iterations=800)
    a = torch.rand(st.shape, dtype=torch.float64, device="cuda")
    b = a.clone()
    torch.cuda.synchronize()
    uhs.run(st, a, b, QUIET)
    assert not torch.cuda.current_stream().query()
    torch.cuda.synchronize()
