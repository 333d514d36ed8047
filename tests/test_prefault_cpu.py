"""Faulting in a host buffer's pages ahead of a copy (csrc/prefault.cpp) is a help and no more: where memory or threads run out
the call comes back, so that the copy itself goes on."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_it_comes_back_when_memory_runs_out(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    csrc, exe = os.path.join(ROOT, "lmweather_gb300", "csrc"), str(tmp_path / "prefault")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", csrc, os.path.join(ROOT, "tests", "cpp", "prefault_test.cpp"),
                    os.path.join(csrc, "prefault.cpp"), "-o", exe], check=True)
    calls, threw, changed = (int(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert (calls, threw, changed) == (13, 0, 0)
