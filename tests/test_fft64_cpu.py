"""The FP64 grid stage's FFT (csrc/fft64.cuh) on the host: its error against long double is no larger than that of plain radix-2
butterflies, which form the product and then two sums, also for small variations beside a large mean."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_error_is_that_of_plain_butterflies(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "fft64")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "lmweather_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fft64_test.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    lines = [line.split() for line in out.splitlines()]
    assert len(lines) == 18
    for n, kind, forward, inverse, most in lines:
        # two per cent for the scatter of 6144 values' errors
        assert float(forward) <= 1.02 and float(inverse) <= 1.02, (n, kind)
        # three roundings a stage at most, each of at most half a unit of a value of the norm's size
        assert float(most) <= 1.5 * (int(n).bit_length() - 1), (n, kind)
