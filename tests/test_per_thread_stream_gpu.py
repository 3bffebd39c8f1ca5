"""cudaStreamPerThread: one handle value, a stream of its own in each host
thread.  Threads that pass it run at the same time and share no counters:
every result is that of the same call made alone, bit for bit, for runs that
stay on chip, runs on copies and sweeps in place, with and without a wait.
Each thread waits for its stream before it ends."""
import threading

import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # the handle's value in the CUDA headers
QUIET = uhs.RunParams(flags=uhs.UHS_FLAG_NO_SYNC)

JOBS = [  # (rank, interior, T, dtype, params)
    (2, (200, 310), 40, "f64", None),
    (2, (512, 400), 60, "f32", None),
    (2, (300, 310), 60, "f32", QUIET),
    (3, (40, 50, 61), 12, "f64", None),
    (3, (40, 50, 61), 4, "f64", QUIET),
    (2, (150, 170), 2, "f64", None),
]


def _job(rank, interior, T, dtype, params):
    import torch
    st = random_case(rank, 1, "star", (4,) * rank, T, 17)[0]
    st = uhs.make_stencil("pt", rank, interior, 1, [t[:3] for t in st.terms], [t[3] for t in st.terms], iterations=T,
                          dtype=uhs.UHS_F32 if dtype == "f32" else uhs.UHS_F64)
    tdt = torch.float32 if dtype == "f32" else torch.float64
    data = torch.rand(st.shape, dtype=tdt, device="cuda") - 0.5
    want = [data.clone(), data.clone()]
    uhs.run(st, *want)
    torch.cuda.synchronize()
    return st, data, want, params


def _check(pairs):
    import torch
    torch.cuda.synchronize()
    for (a, b), want in pairs:
        assert torch.equal(a, want[0]) and torch.equal(b, want[1])


def _together(workers):
    errors = []

    def guarded(w):
        try:
            w()
        except Exception as e:  # reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=guarded, args=(w,)) for w in workers]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not errors, errors


def test_threads_at_once(cuda):
    import torch
    jobs = [_job(*j) for j in JOBS]
    sets = [[(data.clone(), data.clone()) for _ in range(15)] for _, data, _, _ in jobs]
    torch.cuda.synchronize()

    def worker(job, grids):
        st, _, _, params = job
        for a, b in grids:
            uhs.run(st, a, b, params, stream=PER_THREAD)
        spare = grids[0][0].clone()
        torch.cuda.synchronize()
        uhs.run(st.with_(iterations=0), spare, grids[0][1], stream=PER_THREAD)  # no sweeps, but the wait

    _together([lambda j=j, g=g: worker(j, g) for j, g in zip(jobs, sets)])
    _check([(g, j[2]) for j, s in zip(jobs, sets) for g in s])

