"""The top of the float-pair range: values up to 2^128 (unscaled: F32X2 grids,
and FP64 grids under UHS_ARITH_DF32) sum without overflow as long as the
results stay below 2^128, each cell within n^2 2^-46 of sum |c_k x_k| a sweep
for n terms; 2^128 and above returns UHS_ERANGE from FP64 grids.  The passes of
a separable box hold up to G = (sum w / max w)^(rank - 1) times the values in
between, so its values end at 2^127 / G here."""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import assert_cells_close, assert_halo_exact, run_gpu, run_oracle, to_dev
from uxxxxxxxxh_gb300.stencil import box_offsets, make_stencil, star_offsets
from uxxxxxxxxh_gb300.workloads import normalised, splitmix_uniform

pytestmark = pytest.mark.gpu

SHAPES = [(rank, r, kind) for rank in (2, 3) for r in (1, 2, 3) for kind in ("star", "sep")] + [(3, 2, "box"), (3, 3, "box")]
LEVELS = [(2.0 ** 126 * 1.3, 2.0 ** 127 * 0.99), (2.0 ** 127, 2.0 ** 128 * 0.99)]
CASES = [(rank, r, kind, level) for rank, r, kind in SHAPES for level in ((0,) if kind == "sep" else (0, 1))]


def _program(rank, r, kind, interior, T):
    offs = star_offsets(rank, r) if kind == "star" else box_offsets(rank, r)
    if kind == "sep":
        w = [1.0 + abs(d) for d in range(-r, r + 1)]
        coefs = [float(np.prod([w[d + r] / sum(w) for d in o[3 - rank:]])) for o in offs]
    else:
        coefs = normalised(splitmix_uniform(12, len(offs)) + 0.1)
    return make_stencil("top", rank, interior, r, offs, coefs, iterations=T)


def _field(st, r, kind, level, seed=33):
    lo, hi = LEVELS[level]
    gain = (sum(1.0 + abs(d) for d in range(-r, r + 1)) / (1.0 + r)) ** (st.rank - 1) if kind == "sep" else 1.0
    return (lo + (hi - lo) * splitmix_uniform(seed, int(np.prod(st.sizes)))) / gain


def _pairs(x):
    hi = x.astype(np.float32)
    lo = (x - hi.astype(np.float64)).astype(np.float32)
    return np.stack([hi, lo], axis=-1).reshape(-1).view(np.float64), hi.astype(np.float64) + lo.astype(np.float64)


def _joined(t):
    p = t.cpu().numpy().reshape(-1).view(np.float32).reshape(-1, 2).astype(np.float64)
    return p[:, 0] + p[:, 1]


@pytest.mark.parametrize("rank,r,kind,level", CASES)
def test_pair_grids(cuda, rank, r, kind, level):
    import torch
    st = _program(rank, r, kind, (12, 17, 40) if rank == 3 else (40, 300), 2)
    packed, x0 = _pairs(_field(st, r, kind, level))
    ra, rb = run_oracle(st, x0)
    for params in (uhs.RunParams(), uhs.RunParams(use_tma=-1)):
        a, b = to_dev(packed, st), to_dev(packed, st)
        uhs.run(st.with_(dtype=uhs.UHS_F32X2), a, b, params)
        torch.cuda.synchronize()
        tol = 2 * st.nterms ** 2 * 2.0 ** -46
        assert_cells_close(st, ra, _joined(a), tol)
        assert_cells_close(st, rb, _joined(b), tol)


@pytest.mark.parametrize("T,flags", [(1, 0), (2, 0), (8, 0), (8, uhs.UHS_FLAG_IN_PLACE)])
@pytest.mark.parametrize("rank,r,kind,level", CASES)
def test_fp64_grids_in_unscaled_pairs(cuda, rank, r, kind, level, T, flags):
    st = _program(rank, r, kind, (12, 17, 40) if rank == 3 else (40, 300), T)
    a0 = _field(st, r, kind, level)
    ra, rb = run_oracle(st, a0)
    ga, gb = run_gpu(st, a0, uhs.RunParams(arith=uhs.UHS_ARITH_DF32, flags=flags))
    tol = T * st.nterms ** 2 * 2.0 ** -46
    assert_cells_close(st, ra, ga, tol)
    assert_cells_close(st, rb, gb, tol)
    assert_halo_exact(st, ra, ga)


@pytest.mark.parametrize("rank,r", [(2, 2), (3, 1), (3, 3)])
def test_batched_grids_in_unscaled_pairs(cuda, rank, r):
    import torch
    st = _program(rank, r, "star", (12, 17, 40) if rank == 3 else (40, 300), 2)
    a0 = _field(st, r, "star", 0)
    ra, rb = run_oracle(st, a0)
    a, b = to_dev(a0, st), to_dev(a0, st)
    bt = uhs.Batch([st], [a], [b], uhs.RunParams(arith=uhs.UHS_ARITH_DF32))
    bt.run()
    torch.cuda.synchronize()
    bt.close()
    tol = 2 * st.nterms ** 2 * 2.0 ** -46
    assert_cells_close(st, ra, a.cpu().numpy().reshape(-1), tol)
    assert_cells_close(st, rb, b.cpu().numpy().reshape(-1), tol)


@pytest.mark.parametrize("rank,r,kind", [(2, 1, "star"), (3, 2, "star"), (3, 2, "sep"), (3, 2, "box")])
def test_results_from_2_to_the_128_on_are_refused(cuda, rank, r, kind):
    st = _program(rank, r, kind, (12, 17, 40) if rank == 3 else (40, 300), 1)
    st = st.with_(terms=[(t[0], t[1], t[2], 1.3 * t[3]) for t in st.terms])
    a0 = 2.0 ** 127.7 + (2.0 ** 127.9 - 2.0 ** 127.7) * splitmix_uniform(33, int(np.prod(st.sizes)))  # sums from 2^128.07 on
    with pytest.raises(uhs._lib.UhsError) as ei:
        run_gpu(st, a0, uhs.RunParams(arith=uhs.UHS_ARITH_DF32))
    assert ei.value.code == uhs._lib.UHS_ERANGE
