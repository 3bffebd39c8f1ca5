"""A call without a wait that fails after its range scan is enqueued (here: one
plane a chunk, more chunks than the launch grid takes) returns once the scan's
verdict has landed in the host's words, and the thread's next calls are right."""
import time

import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


def test_a_failed_call_leaves_no_copy_in_flight(cuda):
    import torch
    terms = random_case(3, 1, "star", (6, 6, 6), 2, 3)[0].terms
    st = uhs.make_stencil("tall", 3, (70000, 94, 94), 1, [t[:3] for t in terms], [t[3] for t in terms], iterations=2)
    a = torch.rand(st.shape, dtype=torch.float64, device="cuda")
    b = torch.zeros_like(a)
    small = uhs.make_stencil("small", 3, (20, 20, 20), 1, [t[:3] for t in terms], [t[3] for t in terms], iterations=2)
    x = torch.rand(small.shape, dtype=torch.float64, device="cuda")
    want = [x.clone(), x.clone()]
    uhs.run(small, *want)
    torch.cuda.synchronize()
    with pytest.raises(uhs._lib.UhsError):  # the scan reads 5 GB: most of a millisecond
        uhs.run(st, a, b, uhs.RunParams(tile_z=1, flags=uhs.UHS_FLAG_NO_SYNC))
    time.sleep(1e-4)
    assert torch.cuda.current_stream().query()
    got = [x.clone(), x.clone()]
    torch.cuda.synchronize()
    uhs.run(small, *got)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
