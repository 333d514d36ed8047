"""What the sphere's engines copy or set in device memory goes through their own (non-blocking) streams: a copy from pageable
memory, or a memset, on the default stream may still be under way when the kernels that read it start."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lmweather_gb300", "csrc")
# self-tests, whose kernels run on the default stream themselves
DEFAULT_STREAM = ("conversion_selftest_run", "wait_selftest_run", "division_selftest_run")


def functions(text):
    """(name, body) of every function definition at namespace level."""
    for m in re.finditer(r"^(?!#|//|namespace|struct|class|template|constexpr)[^\n;={}]*?([\w:~]+)\([^;{}]*\)[^;{}]*\{\n", text, re.M):
        end = text.find("\n}", m.end())
        yield m.group(1).split("::")[-1], text[m.end():end]


@pytest.mark.parametrize("name", ["sphere.cu", "sphere_tc64.cuh", "sphere_split.cuh", "plane.cu", "ensemble.cu"])
def test_nothing_is_written_on_the_default_stream(name):
    text = open(os.path.join(CSRC, name)).read()
    found = [f for f, body in functions(text) if f not in DEFAULT_STREAM
             and (re.search(r"cudaMemset\(", body) or re.search(r"cudaMemcpy\([^;]*HostToDevice", body))]
    assert found == []
