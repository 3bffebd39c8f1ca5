"""A launch that the driver refuses (more chunks than the launch grid takes)
fails its own call alone: the thread's next calls run as ever."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params", [dict(), dict(kernel=uhs.UHS_KERNEL_GENERIC, arith=uhs.UHS_ARITH_FMA),
                                    dict(arith=uhs.UHS_ARITH_DF32), dict(arith=uhs.UHS_ARITH_FMA)])
@pytest.mark.parametrize("T", [1, 2, 8])
def test_the_next_call_is_not_refused(cuda, T, params):
    import torch
    terms = random_case(3, 1, "star", (6, 6, 6), 2, 3)[0].terms
    offs, coefs = [t[:3] for t in terms], [t[3] for t in terms]
    tall = uhs.make_stencil("tall", 3, (70000, 6, 6), 1, offs, coefs, iterations=T)
    small = uhs.make_stencil("small", 3, (20, 20, 20), 1, offs, coefs, iterations=T)
    a = torch.rand(tall.shape, dtype=torch.float64, device="cuda")
    b = a.clone()
    x = torch.rand(small.shape, dtype=torch.float64, device="cuda")
    want, got = [x.clone(), x.clone()], [x.clone(), x.clone()]
    uhs.run(small, *want)
    torch.cuda.synchronize()
    with pytest.raises(uhs._lib.UhsError) as ei:
        uhs.run(tall, a, b, uhs.RunParams(tile_z=1, **params))
    assert ei.value.code == uhs._lib.UHS_ECUDA
    uhs.run(small, *got)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
