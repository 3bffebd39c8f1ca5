"""Resident runs: rank-2 programs whose domain fits in shared memory run in
one cooperative launch (UHS_ARITH_AUTO on FP64 grids; FP32 from T = 8).  Both
grids must end bit-identical to the same program launched sweep by sweep on
the streaming kernel (kernel = STREAM), whose results are held to the oracle
elsewhere: the same terms, order and roundings per point.  Sizes cover one
box, boxes thinner than the radius, ragged splits, one and several groups of
rows per box, domains inside a larger strided grid, and halos that differ
between the two grids."""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import assert_cells_close, assert_f64_close, run_gpu, run_oracle
from uxxxxxxxxh_gb300.stencil import box_offsets, make_stencil
from uxxxxxxxxh_gb300.workloads import random_case, splitmix_uniform

pytestmark = pytest.mark.gpu

STREAM = uhs.RunParams(kernel=uhs.UHS_KERNEL_STREAM)


def _program(r, kind, interior, T):
    if kind != "sep":
        return random_case(2, r, kind, interior, T, 900 + r)[0]
    w = [1.0 + abs(d) for d in range(-r, r + 1)]
    coefs = [w[dy + r] * w[dx + r] / sum(w) ** 2 for _, dy, dx in box_offsets(2, r)]
    return make_stencil(f"sep2d{r}", 2, interior, r, box_offsets(2, r), coefs, iterations=T)


def _pair_of_runs(st, tdt, pad=(0, 0)):
    """(a, b) of a default run and of the streaming sweeps, from the same data."""
    import torch
    shape = (st.sizes[1] + pad[0], st.sizes[2] + pad[1])
    n = shape[0] * shape[1]
    data = [torch.from_numpy(2.0 * splitmix_uniform(s, n).reshape(shape) - 1.0).to(tdt).cuda() for s in (31, 32)]
    out = []
    for p in (None, STREAM):
        full = [d.clone() for d in data]
        a, b = (f[pad[0] // 2:pad[0] // 2 + st.sizes[1], pad[1] // 2:pad[1] // 2 + st.sizes[2]] for f in full)
        n0 = uhs.launch_count()
        uhs.run(st, a, b, p)
        torch.cuda.synchronize()
        out.append((full, uhs.launch_count() - n0))
    return out


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("T", [2, 8, 14])
@pytest.mark.parametrize("r,kind", [(1, "star"), (2, "star"), (3, "star"), (1, "box"), (2, "box"), (3, "box"),
                                    (1, "sep"), (2, "sep"), (3, "sep")])
def test_resident_run_is_the_streaming_run_bitwise(cuda, r, kind, T, dtype):
    import torch
    for interior in ((1, 1), (2, 700), (700, 2), (33, 65), (301, 257), (1441, 1203)):
        st = _program(r, kind, interior, T)
        if dtype == "f32":
            st = st.with_(dtype=uhs.UHS_F32)
        tdt = torch.float32 if dtype == "f32" else torch.float64
        pad = (6, 10) if interior == (33, 65) else (0, 0)
        (one, n1), (many, _) = _pair_of_runs(st, tdt, pad)
        assert n1 == 1 or (dtype == "f32" and T < 8)
        for x, y in zip(one, many):
            assert torch.equal(x, y), (interior, (x - y).abs().max().item())


def test_range_outside_float_pairs_runs_native(cuda):
    """Values near 1 and near 1e-60, and a NaN: the resident launch leaves the
    grids as they were and the sweeps run in native FP64, bit-identical to
    UHS_ARITH_FMA."""
    for small in (1e-60, float("nan")):
        st, a0 = random_case(2, 1, "star", (90, 130), 10, 77)
        a0 = np.abs(a0) + 0.5
        a0[len(a0) // 2:len(a0) // 2 + 40] = small
        ga, gb = run_gpu(st, a0)
        fa, fb = run_gpu(st, a0, uhs.RunParams(arith=uhs.UHS_ARITH_FMA))
        assert np.array_equal(ga.view(np.uint64), fa.view(np.uint64))
        assert np.array_equal(gb.view(np.uint64), fb.view(np.uint64))


def test_scaled_range_and_back_to_back_runs(cuda):
    """Fields of any magnitude keep every cell (the scale comes from the
    kernel's own scan), run after run on one stream."""
    for scale in (1e-40, 1.0, 1e200):
        st, a0 = random_case(2, 2, "star", (70, 300), 8, 78)
        a0 = scale * (1.5 + a0)
        ra, rb = run_oracle(st, a0)
        ga, gb = run_gpu(st, a0)
        assert_cells_close(st, ra, ga, 1e-12)
        assert_cells_close(st, rb, gb, 1e-12)


def test_captured_and_concurrent_runs(cuda):
    """Under stream capture the sweeps are launched one by one (FP32); resident
    runs on several streams at once do not disturb one another."""
    import torch
    st, a0 = random_case(2, 1, "star", (200, 330), 12, 79, dtype=uhs.UHS_F32)
    host = torch.from_numpy(a0.reshape(st.sizes[1:]).astype(np.float32))
    want = host.cuda()
    wb = want.clone()
    uhs.run(st, want, wb)
    quiet = uhs.RunParams(flags=uhs.UHS_FLAG_NO_SYNC)
    a, b = host.cuda(), host.cuda()
    s = torch.cuda.Stream()
    uhs.run(st, a.clone(), b.clone(), stream=s)  # the stream's status word exists before the capture
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        uhs.run(st, a, b, quiet, stream=s)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b, wb)
    streams = [torch.cuda.Stream() for _ in range(4)]
    grids = [(host.cuda(), host.cuda()) for _ in streams]
    torch.cuda.synchronize()
    for _ in range(3):
        for q, (x, y) in zip(streams, grids):
            uhs.run(st, x, y, quiet, stream=q)
    torch.cuda.synchronize()
    for _ in range(2):
        uhs.run(st, want, wb)
    for x, y in grids:
        assert torch.equal(x, want) and torch.equal(y, wb)


def test_scratch_cap_falls_back_to_sweeps(cuda):
    st, a0 = random_case(2, 1, "star", (64, 80), 8, 80)
    ra, _ = run_oracle(st, a0)
    run_gpu(st, a0)
    L = uhs.lib()
    assert L.uhs_set_alloc_cap(64) == 0
    try:
        n0 = uhs.launch_count()
        ga, _ = run_gpu(st, a0)
        assert uhs.launch_count() - n0 >= 8
    finally:
        assert L.uhs_set_alloc_cap(0) == 0
    assert_f64_close(st, ra, ga)
