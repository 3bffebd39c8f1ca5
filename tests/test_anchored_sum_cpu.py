"""The float-pair anchored sum's arithmetic (df32.cuh: anchor_add, dfa_first,
dfa_add, dfa_end, dfa_renorm), restated in C on the host with the C library's
correctly rounded fmaf (tests/c/anchored_sum_check.c): on random stencil sums
of 3-19 float-pair terms every step that the scheme takes as exact is exact,
and the result is within n^2 2^-46 of B = sum |ch_k| |xh_k| of the exact sum
(computed in binary128)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_anchored_sum_steps_are_exact_and_the_result_within_its_bound(tmp_path):
    exe = tmp_path / "anchored_sum_check"
    r = subprocess.run(["gcc", "-O2", "-ffp-contract=off", os.path.join(HERE, "c", "anchored_sum_check.c"), "-lm",
                        "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0 and "float128" in r.stderr:
        pytest.skip("this compiler has no binary128 type")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe), "120000", "11"], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "violations=0" in out.stdout
