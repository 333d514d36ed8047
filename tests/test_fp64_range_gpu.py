"""What FP64 promises at the ends of its range: a tracer of any magnitude is carried as one of order one is (its equation is
linear), and the grids handed out keep the relative accuracy of plain FP64 sums where a wavenumber is tiny."""
import numpy as np
import pytest

from oracle_lib import OracleSphere
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


@pytest.mark.parametrize("T,m", [(21, 9), (42, 20), (85, 40), (170, 80)])
def test_grids_keep_their_digits_towards_the_poles(engine, T, m):
    """A flow of one wavenumber m whose large coefficient is the first, (m, m): towards the poles P_m^m is many orders smaller
    than the P_n^m of its small coefficients. Row by row within 2^-53 of the sum's terms, of which there are T: 1e-12."""
    M = T + 1
    z, d, f = (np.zeros((M, M), complex) for _ in range(3))
    n = np.arange(m, M)
    z[m, m:] = 1e-5 * np.exp(-3.0 * (n - m)) * (1 + 0.5j)
    f[0, 0] = 8000.0 * 9.80616 * np.sqrt(2.0)
    s, o = engine.Sphere(T), OracleSphere(T)
    for x in (s, o):
        x.set_state(z.ravel(), d.ravel(), f.ravel())
    for got, ref in ((s.grid_vorticity(), o.grid_vorticity()), (s.grid_u(), o.grid_u()), (s.grid_v(), o.grid_v())):
        scale = np.abs(ref).max(axis=1)
        assert scale.min() < 1e-3 * scale.max()
        assert (np.abs(got - ref).max(axis=1) <= 1e-12 * scale).all()
