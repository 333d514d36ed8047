"""The plane's stage kernel at the edges of its arithmetic, against the oracle bit for bit."""
import numpy as np
import pytest

from oracle_lib import OraclePlane

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    """The same values with the same signs of zero; NaN in the same places."""
    a, b = np.asarray(a), np.asarray(b)
    nan = np.isnan(a)
    return np.array_equal(nan, np.isnan(b)) and np.array_equal(a[~nan].view(np.uint64), b[~nan].view(np.uint64))


@pytest.mark.parametrize("linear", [True, False])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_without_drag_a_value_that_is_not_finite_spreads_as_in_the_reference(engine, linear, bad):
    nx, ny = 40, 20
    par = dict(f0=1e-4, beta=0.0, depth=100.0, linear=linear)
    rng = np.random.default_rng(5)
    h, u, v = 100.0 + rng.standard_normal((ny, nx)), rng.standard_normal((ny, nx)), rng.standard_normal((ny + 1, nx))
    v[0] = v[ny] = 0.0
    u[7, 9], v[12, 30] = bad, bad
    o, p = OraclePlane(nx, ny, 4e5, 2e5, **par), engine.Plane(nx, ny, 4e5, 2e5, **par)
    o.set(h, u, v)
    p.set_h_from_grid(h).set_u_from_grid(u).set_v_from_grid(v)
    o.step(10.0)
    p.step(10.0)
    for a, b in zip(p.get(), o.get()):
        assert same_bits(a, b)


def test_a_rest_state_of_negative_zeros(engine):
    nx, ny = 36, 18
    par = dict(f0=0.0, beta=2e-11, depth=100.0)
    for lin in (True, False):
        o, p = OraclePlane(nx, ny, 4e5, 2e5, linear=lin, **par), engine.Plane(nx, ny, 4e5, 2e5, linear=lin, **par)
        h, u, v = np.full((ny, nx), 100.0), np.full((ny, nx), -0.0), np.full((ny + 1, nx), -0.0)
        o.set(h, u, v)
        p.set_h_from_grid(h).set_u_from_grid(u).set_v_from_grid(v)
        for _ in range(3):
            o.step(10.0)
            p.step(10.0)
        for a, b in zip(p.get(), o.get()):
            assert same_bits(a, b)
