"""The exact slicing behind the FP64 Legendre sums (csrc/exact_slices.cuh) on the host: every sum within the bound that the
file's users state, K 1.4 2^-55 2^(ea + eb) and one rounding, for rows flat and steep, of any magnitude down to subnormals."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sums_stay_within_their_bound(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "exact_slices")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "lmweather_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "exact_slices_test.cpp"), "-o", exe], check=True)
    _, out, past, digits, lost = (int(v) for v in subprocess.run([exe, "20000"], check=True, capture_output=True, text=True).stdout.split())
    assert out == 0
    assert past == 0  # every order fits the FP32 accumulators exactly
    assert digits == 0
    assert lost == 0
