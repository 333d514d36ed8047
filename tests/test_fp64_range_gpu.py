"""What FP64 promises at the ends of its range: a tracer of any magnitude is carried as one of order one is (its equation is
linear)."""
import numpy as np
import pytest

from test_stage_forms_gpu import tracer
from test_tc64_gpu import initial

pytestmark = pytest.mark.gpu

# the bar of tests/test_tracer_gpu.py, of the largest value. Scaled to 2^-1000 the grid products lie 2^-1030 and above,
# where subnormal numbers still have 44 bits (2^-44 = 6e-14)
TOL = 1e-12


@pytest.mark.parametrize("T", [21, 62])
@pytest.mark.parametrize("power", [900, -880, -930, -1000])
def test_a_tracer_of_any_magnitude_is_carried(engine, T, power):
    s = engine.Sphere(T)
    state, q = initial(T, 5 * T), tracer(T, s.nlat, s.nlon, 3)

    def carried(scale):
        e = engine.Sphere(T)
        e.set_state(*state)
        e.set_tracer_grid(q * scale)
        first = e.tracer_state()
        for _ in range(3):
            e.step(20000.0 / T)
        return first / scale, e.tracer_state() / scale

    first, ref = carried(1.0)
    _, got = carried(2.0 ** power)
    assert np.abs(ref - first).max() > 1e-4 * np.abs(ref).max()  # it has moved
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
