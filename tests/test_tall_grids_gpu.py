"""Domains with more rows (planes) than the launch grid's third axis takes
chunks of the class's usual length: the chunks get longer and the run is that
of native FP64 arithmetic within the oracle's bar."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,interior,dtype", [(2, (1100000, 64), "f64"), (3, (600000, 4, 5), "f64"),
                                                 (3, (700000, 4, 6), "f32")])
def test_tall_runs(cuda, rank, interior, dtype):
    import torch
    st = random_case(rank, 1, "star", (6, 6, 6)[:rank], 8, 3)[0]
    st = uhs.make_stencil("tall", rank, interior, 1, uhs.star_offsets(rank, 1), [t[3] for t in st.terms], iterations=8)
    g = torch.Generator(device="cuda").manual_seed(5)
    a64 = torch.rand(st.shape, dtype=torch.float64, device="cuda", generator=g)
    if dtype == "f32":
        a64 = a64.float().double()
    ra, rb = a64.clone(), a64.clone()
    uhs.run(st, ra, rb, uhs.RunParams(arith=uhs.UHS_ARITH_FMA))
    tdt = torch.float32 if dtype == "f32" else torch.float64
    a, b = a64.to(tdt, copy=True), a64.to(tdt, copy=True)
    uhs.run(st.with_(dtype=uhs.UHS_F32) if dtype == "f32" else st, a, b)
    torch.cuda.synchronize()
    tol = 1e-6 if dtype == "f32" else 1e-12
    assert (a.double() - ra).abs().max().item() <= tol
    assert (b.double() - rb).abs().max().item() <= tol
