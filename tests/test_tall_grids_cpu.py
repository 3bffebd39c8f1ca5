"""Automatic z-chunks never cut a domain into more than 65535 pieces (the
launch grid's limit along its third axis), whatever cap a sweep class has."""
import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case


@pytest.mark.parametrize("dtype", [uhs.UHS_F64, uhs.UHS_F32, uhs.UHS_F32X2])
@pytest.mark.parametrize("rank,r,kind", [(k, r, s) for k in (2, 3) for r in (1, 2, 3) for s in ("star", "box")])
def test_chunks_fit_the_launch_grid(rank, r, kind, dtype):
    st = random_case(rank, r, kind, (6, 6, 6)[:rank], 2, 3, dtype=dtype)[0]
    for nz in (65536, 524281, 1048561, 1100000, 1 << 24):
        lb, ub, sizes = list(st.lb), list(st.ub), list(st.sizes)
        ax = 3 - rank
        ub[ax], sizes[ax] = lb[ax] + nz, nz + 2 * r
        g = uhs.launch_geometry(st.with_(sizes=tuple(sizes), ub=tuple(ub)))
        assert g["zchunk"] >= 1 and -(-nz // g["zchunk"]) <= 65535, (nz, g)
