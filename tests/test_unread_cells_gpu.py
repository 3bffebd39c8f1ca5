"""Cells that a program never reads: a domain inside a larger grid leaves cells
farther from it than the radius, which tiles load all the same.  Whatever they
hold (NaN, Inf, values far above the domain's), an FP64 run under
UHS_ARITH_AUTO returns what it returns with ordinary values there, bit for
bit, on every route: one sweep, sweeps in place, copies; TMA and cp.async
layouts; with and without a wait.  (Term-by-term 3D boxes of radius 2-3 from
eight sweeps on scan whole grids and may turn to native FP64: within 1e-12.)"""
import numpy as np
import pytest

import uxxxxxxxxh_gb300 as uhs
from gpu_util import to_dev
from uxxxxxxxxh_gb300.stencil import box_offsets, make_stencil, star_offsets
from uxxxxxxxxh_gb300.workloads import normalised, splitmix_uniform

pytestmark = pytest.mark.gpu

NO_RESIDENT = dict(prefetch=4)  # 2D: a stated launch parameter (the built depth)


def _program(rank, r, kind, interior, margin, T):
    offs = star_offsets(rank, r) if kind == "star" else box_offsets(rank, r)
    if kind == "sep":
        w = [1.0 + abs(d) for d in range(-r, r + 1)]
        coefs = [float(np.prod([w[d + r] / sum(w) for d in o[3 - rank:]])) for o in offs]
    else:
        coefs = normalised(splitmix_uniform(12, len(offs)) + 0.1)
    st = make_stencil("inner", rank, interior, r, offs, coefs, iterations=T)
    axes = range(3 - rank, 3)
    grow = [margin if i in axes else 0 for i in range(3)]
    return st.with_(sizes=tuple(n + 2 * g for n, g in zip(st.sizes, grow)),
                    lb=tuple(l + g for l, g in zip(st.lb, grow)), ub=tuple(u + g for u, g in zip(st.ub, grow)))


def _grids(st, r, outer):
    """Ordinary values within r of the domain, `outer` beyond (None: ordinary too)."""
    out = []
    for seed in (21, 22):
        g = (2.0 * splitmix_uniform(seed, int(np.prod(st.sizes))) - 1.0).reshape(st.sizes)
        if outer is not None:
            keep = np.zeros(st.sizes, bool)
            keep[tuple(slice(max(0, l - r), u + r) for l, u in zip(st.lb, st.ub))] = True
            g[~keep] = outer
        out.append(g.reshape(-1))
    return out


@pytest.mark.parametrize("T,sweep", [(1, True), (1, False), (2, False), (6, False), (8, False)])
@pytest.mark.parametrize("rank,r,kind,interior,margin", [
    (3, 1, "star", (18, 19, 40), 4), (3, 2, "star", (18, 19, 37), 3), (3, 3, "star", (9, 21, 37), 2),
    (3, 1, "box", (9, 19, 37), 3), (3, 2, "box", (9, 11, 37), 3), (3, 2, "sep", (9, 19, 40), 4),
    (2, 1, "star", (37, 140), 4), (2, 3, "star", (37, 131), 3), (2, 2, "sep", (37, 140), 4), (2, 2, "box", (37, 131), 3)])
def test_cells_beyond_the_radius_do_not_count(cuda, rank, r, kind, interior, margin, T, sweep):
    import torch
    st = _program(rank, r, kind, interior, margin, T)
    out = []
    for outer in (None, np.nan, np.inf, 1e30):
        for flags in (0, uhs.UHS_FLAG_NO_SYNC):
            p = uhs.RunParams(flags=flags, **(NO_RESIDENT if rank == 2 else {}))
            a, b = (to_dev(g, st) for g in _grids(st, r, outer))
            (uhs.sweep if sweep else uhs.run)(st, a, b, p)
            if flags:
                uhs.sweep(st.with_(iterations=1), b, torch.zeros_like(a), uhs.RunParams(arith=uhs.UHS_ARITH_FMA))
            torch.cuda.synchronize()
            inner = tuple(slice(l, u) for l, u in zip(st.lb, st.ub))[3 - rank:]
            out.append((a[inner].clone(), b[inner].clone()))
    whole = rank == 3 and r > 1 and kind == "box" and T >= 8
    for got in out[1:]:
        for x, y in zip(got, out[0]):
            assert torch.allclose(x, y, rtol=0.0, atol=1e-12) if whole else torch.equal(x, y)
