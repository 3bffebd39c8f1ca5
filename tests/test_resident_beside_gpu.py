"""Resident runs beside another stream's kernel that holds some SMs for longer
than a wait inside the run may take (about a second): the cooperative launch
starts once all of its CTAs can be placed, so no wait runs out, and the result is
that of the same call made alone, bit for bit."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


def _star(rank, interior, T, dtype=uhs.UHS_F64):
    terms = random_case(rank, 1, "star", (4,) * rank, 2, 17)[0].terms
    return uhs.make_stencil("beside", rank, interior, 1, [t[:3] for t in terms], [t[3] for t in terms], iterations=T,
                            dtype=dtype)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_a_long_kernel_elsewhere(cuda, dtype):
    import torch
    # two CTAs that walk 350,000 planes each: 1.5 s; the run needs every SM's shared memory
    long = _star(3, (350000, 8, 64), 1)
    st = _star(2, (1950, 1950) if dtype == "f64" else (2800, 2880), 12, uhs.UHS_F32 if dtype == "f32" else uhs.UHS_F64)
    data = torch.rand(st.shape, dtype=torch.float32 if dtype == "f32" else torch.float64, device="cuda") - 0.5
    want, got = [data.clone(), data.clone()], [data.clone(), data.clone()]
    n0 = uhs.launch_count()
    uhs.run(st, *want)
    assert uhs.launch_count() - n0 == 1
    x = torch.rand(long.shape, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    busy, mine = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    uhs.sweep(long, x, y, uhs.RunParams(kernel=uhs.UHS_KERNEL_GENERIC, arith=uhs.UHS_ARITH_EXACT, tile_z=1 << 30,
                                        flags=uhs.UHS_FLAG_NO_SYNC), stream=busy)
    uhs.run(st, *got, stream=mine)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
