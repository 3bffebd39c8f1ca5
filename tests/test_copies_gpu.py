"""Runs on the library's own copies: FP64 programs under UHS_ARITH_AUTO (T >=
8, or T >= 4 from 2^21 points on) read the caller's grid in their first sweep
and write it in their last ones, with float-pair copies in between and the
range decided on the device; FP32 programs run on padded copies where TMA
cannot load the caller's rows.  Both grids must end bit-identical to the path
with conversion passes (FP64: UHS_ARITH_DF32 explicit, on data whose scale is
immaterial) or to the sweeps launched in place (FP32: kernel = STREAM), halos
untouched, on odd widths, strided grids and halos that differ between a and b."""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import assert_f64_close, assert_halo_exact, run_gpu, run_oracle
from uxxxxxxxxh_gb300.stencil import box_offsets, make_stencil
from uxxxxxxxxh_gb300.workloads import random_case, splitmix_uniform

pytestmark = pytest.mark.gpu

DF32 = uhs.RunParams(arith=uhs.UHS_ARITH_DF32)
STREAM = uhs.RunParams(kernel=uhs.UHS_KERNEL_STREAM)
NO_RESIDENT = uhs.RunParams(prefetch=4)  # a stated launch parameter (2D: the built depth): not a resident run


def _program(rank, r, kind, interior, T):
    if kind != "sep":
        return random_case(rank, r, kind, interior, T, 300 + r)[0]
    w = [1.0 + abs(d) for d in range(-r, r + 1)]
    offs = box_offsets(rank, r)
    coefs = [np.prod([w[d + r] / sum(w) for d in o[3 - rank:]]) for o in offs]
    return make_stencil(f"sep{rank}d{r}", rank, interior, r, offs, coefs, iterations=T)


def _runs(st, params, tdt, pad=0):
    import torch
    shape = [n + pad for n in st.sizes[3 - st.rank:]]
    data = [torch.from_numpy(2.0 * splitmix_uniform(s, int(np.prod(shape))).reshape(shape) - 1.0).to(tdt).cuda()
            for s in (41, 42)]
    cut = tuple(slice(pad // 2, pad // 2 + n) for n in st.sizes[3 - st.rank:])
    out = []
    for p in params:
        full = [d.clone() for d in data]
        n0 = uhs.launch_count()
        uhs.run(st, full[0][cut], full[1][cut], p)
        torch.cuda.synchronize()
        out.append((full, uhs.launch_count() - n0))
    return out


SHAPES = [(3, r, k) for r in (1, 2, 3) for k in ("star", "sep")] + [(3, 1, "box")] + \
         [(2, r, k) for r in (1, 2, 3) for k in ("star", "sep", "box")]


@pytest.mark.parametrize("rank,r,kind", SHAPES)
def test_fp64_run_ends_match_the_conversion_passes_bitwise(cuda, rank, r, kind):
    import torch
    for interior, T, pad in (((13, 17, 36), 8, 0), ((9, 33, 65), 10, 0), ((20, 16, 31), 8, 5)) if rank == 3 else \
            (((37, 130), 8, 0), ((64, 257), 10, 0), ((50, 131), 8, 5)):
        st = _program(rank, r, kind, interior, T)
        auto = None if rank == 3 else NO_RESIDENT
        (one, n1), (two, n2) = _runs(st, (auto, DF32), torch.float64, pad)
        assert n1 == T + 2 and n2 == T + 4  # scan and shells; split x 2 and join x 2
        for x, y in zip(one, two):
            assert torch.equal(x, y), (interior, (x - y).abs().max().item())


@pytest.mark.parametrize("rank,r,kind,interior", [(3, 1, "star", (130, 129, 127)), (3, 2, "star", (128, 130, 131)),
                                                  (2, 2, "star", (2900, 1999)), (2, 1, "sep", (2100, 2601))])
def test_short_fp64_runs_of_large_grids(cuda, rank, r, kind, interior):
    """T = 4 above 2^21 points: on copies, against the oracle."""
    st = _program(rank, r, kind, interior, 4)
    a0 = 2.0 * splitmix_uniform(51, int(np.prod(st.sizes))) - 1.0
    b0 = 2.0 * splitmix_uniform(52, a0.size) - 1.0
    ra, rb = run_oracle(st, a0, b0)
    n0 = uhs.launch_count()
    ga, gb = run_gpu(st, a0, None if rank == 3 else NO_RESIDENT, b0)
    assert uhs.launch_count() - n0 == 4 + 2
    assert_f64_close(st, ra, ga)
    assert_f64_close(st, rb, gb)
    assert_halo_exact(st, ra, ga)
    assert_halo_exact(st, rb, gb)


@pytest.mark.parametrize("rank,r,kind,T", [(3, 1, "star", 8), (3, 2, "star", 16), (3, 3, "star", 8), (3, 1, "box", 8),
                                           (3, 2, "sep", 16), (2, 1, "star", 16), (2, 2, "star", 16), (2, 3, "box", 16)])
def test_fp32_runs_on_padded_copies_bitwise(cuda, rank, r, kind, T):
    import torch
    # (2D: beyond what runs resident; 3D: 2^18 or 2^20 points)
    for interior, pad in (((97, 130, 87), 0), ((107, 101, 102), 3)) if rank == 3 else (((37, 200001), 0), ((64, 150003), 3)):
        st = _program(rank, r, kind, interior, T).with_(dtype=uhs.UHS_F32)
        (one, n1), (two, n2) = _runs(st, (None, STREAM), torch.float32, pad)
        assert n1 == T + 2 and n2 == T  # padded copies: the shells, and step T - 1 twice
        for x, y in zip(one, two):
            assert torch.equal(x, y), (interior, (x - y).abs().max().item())


@pytest.mark.parametrize("T", [1, 2, 6, 8, 24])
def test_range_decided_on_the_device(cuda, T):
    """A field wider than float pairs' window, and one with an Inf: native FP64,
    bit-identical to UHS_ARITH_FMA, on every route (in place, on copies)."""
    for bad in (1e-60, np.inf):
        st, a0 = random_case(3, 1, "star", (20, 24, 37), T, 71)
        a0 = np.abs(a0) + 0.5
        a0[a0.size // 2:a0.size // 2 + 7] = bad
        ga, gb = run_gpu(st, a0)
        fa, fb = run_gpu(st, a0, uhs.RunParams(arith=uhs.UHS_ARITH_FMA))
        assert np.array_equal(ga.view(np.uint64), fa.view(np.uint64))
        assert np.array_equal(gb.view(np.uint64), fb.view(np.uint64))
