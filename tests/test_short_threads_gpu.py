"""Host threads that make one call and end leave their pinned words to the next
ones, across uhs_release_scratch as well: each result is right."""
import threading

import pytest

import uxxxxxxxxh_gb300 as uhs
from uxxxxxxxxh_gb300.workloads import random_case

pytestmark = pytest.mark.gpu


def _program(T, dtype):
    terms = random_case(3, 1, "star", (4, 4, 4), 2, 17)[0].terms
    return uhs.make_stencil("one", 3, (20, 21, 22), 1, [t[:3] for t in terms], [t[3] for t in terms], iterations=T,
                            dtype=dtype)


def _in_a_thread(f):
    errors = []

    def guarded():
        try:
            f()
        except Exception as e:  # reported below
            errors.append(repr(e))

    t = threading.Thread(target=guarded)
    t.start()
    t.join(timeout=60)
    assert not t.is_alive() and not errors, errors


def test_one_call_per_thread(cuda):
    import torch
    st = _program(4, uhs.UHS_F64)
    data = torch.rand(st.shape, dtype=torch.float64, device="cuda")
    want = [data.clone(), data.clone()]
    uhs.run(st, *want)
    sets = [(data.clone(), data.clone()) for _ in range(40)]
    torch.cuda.synchronize()
    for i, (a, b) in enumerate(sets):
        _in_a_thread(lambda: uhs.run(st, a, b))
        if i % 10 == 9:
            uhs.release_scratch()
    torch.cuda.synchronize()
    for a, b in sets:
        assert torch.equal(a, want[0]) and torch.equal(b, want[1])
