"""A batch cuts its grids into items as short as one plane (shorter than the
halo): one small grid of each of the 12 shapes in FP64 and FP32, on extents
that leave ragged tiles, alone in its batch and all together, against the
oracle at the element type's bar."""
import numpy as np
import pytest

import oracle
import uxxxxxxxxh_gb300 as uhs
from gpu_util import assert_f64_close, assert_halo_exact, run_oracle, to_dev
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu

SHAPES = [(rank, r, kind) for rank in (2, 3) for r in (1, 2, 3) for kind in ("star", "box")]


def _check(st, a0, a, b):
    ra, rb = run_oracle(st, a0)
    for want, got in ((ra, a), (rb, b)):
        got = got.cpu().numpy().reshape(-1)
        if st.dtype == uhs.UHS_F32:
            assert oracle.error(st, want, got.astype(np.float64))["l2_rel"] <= 1e-6
        else:
            assert_f64_close(st, want, got)
            assert_halo_exact(st, want, got)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_one_plane_items_of_every_shape(cuda, dtype):
    import torch
    parts = []
    for rank, r, kind in SHAPES:
        st, a0 = random_case(rank, r, kind, (21, 261) if rank == 2 else (9, 19, 37), 4, 600 + 10 * rank + r)
        if dtype == "f32":
            st, a0 = st.with_(dtype=uhs.UHS_F32), a0.astype(np.float32).astype(np.float64)
        parts.append((st, a0))
    tdt = torch.float32 if dtype == "f32" else torch.float64
    together = [(st, a0, to_dev(a0, st, tdt), to_dev(a0, st, tdt)) for st, a0 in parts]
    batch = uhs.Batch([p[0] for p in together], [p[2] for p in together], [p[3] for p in together])
    batch.run()
    batch.close()
    for st, a0, a, b in together:
        _check(st, a0, a, b)
    for st, a0 in parts:
        a, b = to_dev(a0, st, tdt), to_dev(a0, st, tdt)
        batch = uhs.Batch([st], [a], [b])
        batch.run()
        batch.close()
        _check(st, a0, a, b)
