"""The step graphs an engine keeps (csrc/graph_slots.h): what a pattern of calls captures, and that none is used after it was
destroyed, destroyed twice or left behind."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_graphs_are_captured_where_they_are_used_again(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "graph_slots")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "lmweather_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "graph_slots_test.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    captures = {name: (int(n), int(wrong)) for name, n, wrong in (line.split() for line in out.splitlines())}
    assert captures["alternating"] == (1 + 200, 0)  # the step's graph once, each run's two chunks
    assert captures["remainders"] == (1 + 100, 0)  # the guard-sized chunk once, the remainders (4 to 63, each again after 60 runs) each time
    assert captures["short"] == (0, 0)
    assert captures["long"] == (8, 0)
