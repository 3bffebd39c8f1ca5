"""Whether an FP64 run under UHS_ARITH_AUTO rounds to FP64 between its steps
depends on T and the number of points alone: a resident run, the same run
with a stated launch parameter, and the same run without a wait end bit for
bit alike on both sides of 2^21 points."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 4, 6, 8])
@pytest.mark.parametrize("r,kind", [(1, "star"), (3, "star"), (1, "box")])
def test_resident_runs_round_as_the_other_routes(cuda, r, kind, T):
    import torch
    for interior in ((1441, 1203), (1500, 1450), (1448, 1448 + 1)):
        st = random_case(2, r, kind, (8, 8), T, 90 + r)[0]
        st = uhs.make_stencil("r", 2, interior, r, [t[:3] for t in st.terms], [t[3] for t in st.terms], iterations=T)
        g = torch.Generator(device="cuda").manual_seed(7)
        data = torch.rand(st.shape, dtype=torch.float64, device="cuda", generator=g) - 0.5
        torch.cuda.synchronize()
        out = []
        for p in (None, uhs.RunParams(kernel=uhs.UHS_KERNEL_STREAM), uhs.RunParams(flags=uhs.UHS_FLAG_NO_SYNC)):
            a, b = data.clone(), data.clone()
            torch.cuda.synchronize()
            n0 = uhs.launch_count()
            uhs.run(st, a, b, p)
            if p is None:
                assert uhs.launch_count() - n0 == 1
            torch.cuda.synchronize()
            out.append((a, b))
        for x, y in out[1:]:
            assert torch.equal(x, out[0][0]) and torch.equal(y, out[0][1]), (interior, (x - out[0][0]).abs().max().item())
