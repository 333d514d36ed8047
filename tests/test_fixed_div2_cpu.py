"""The two-operation division by a fixed divisor (csrc/fixed_div.cuh): every answer it gives is the IEEE quotient, for
divisors of the plane's form, powers of two and random ones, and dividends that include zeros of both signs,
infinities, NaN, the extremes of the range, the divisor's exceptional dividend and quotients next to midpoints."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_answer_is_the_rounded_quotient(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "fixed_div2")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "lmweather_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fixed_div2_test.cpp"), "-o", exe], check=True)
    divisors, qualified, exceptions, wrong, slow = (int(v) for v in subprocess.run([exe, "3000"], check=True, capture_output=True,
                                                                                  text=True).stdout.split())
    assert wrong == 0
    assert qualified == divisors  # all of them have a proof with at most one exception
    assert exceptions < divisors // 8
    assert slow < 400 * divisors // 10  # the special dividends and a few far outside the range
