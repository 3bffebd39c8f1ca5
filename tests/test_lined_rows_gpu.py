"""FP32 runs of 3D radius-1 stars on grids whose rows already start on 128-byte
lines sweep the caller's grids; the same program off the lines runs on padded
copies.  Both end bit for bit alike."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


def test_rows_on_lines_need_no_copies(cuda):
    import torch
    T = 16
    st = random_case(3, 1, "star", (6, 6, 6), T, 95)[0]
    st = uhs.make_stencil("lined", 3, (256, 256, 256), 1, [t[:3] for t in st.terms], [t[3] for t in st.terms],
                          iterations=T, dtype=uhs.UHS_F32)
    g = torch.Generator(device="cuda").manual_seed(8)
    data = torch.rand(st.shape, dtype=torch.float32, device="cuda", generator=g) - 0.5
    out = []
    for col, want in ((32, T), (4, T + 2)):  # the domain's first column, on a line or off (TMA loads both)
        prog = st.with_(sizes=(258, 258, 320), lb=(1, 1, col), ub=(257, 257, col + 256))
        a, b = (torch.zeros((258, 258, 320), dtype=torch.float32, device="cuda") for _ in range(2))
        cut = (slice(None), slice(None), slice(col - 1, col + 257))
        a[cut] = data
        b[cut] = data
        torch.cuda.synchronize()
        n0 = uhs.launch_count()
        uhs.run(prog, a, b)
        assert uhs.launch_count() - n0 == want
        out.append((a[cut].clone(), b[cut].clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
