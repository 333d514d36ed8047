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


@pytest.mark.parametrize("linear", [True, False])
@pytest.mark.parametrize("low,high", [(-322, -300), (-305, -290), (-160, -90), (-100, 0), (0, 120), (120, 160), (150, 307)])
def test_values_at_the_ends_of_the_range(engine, low, high, linear):
    """Fields of 10^low to 10^high: products that are subnormal, that vanish or that overflow round as in the reference."""
    for k, (nx, ny, kw) in enumerate([(5, 4, {}), (40, 20, dict(drag=1e-6, viscosity=30.0)), (70, 33, dict(f0=0.0)), (33, 150, dict(beta=0.0)),
                                      (410, 200, {}), (600, 300, dict(drag=1e-6))]):
        rng = np.random.default_rng(1000 * k + 400 + high)
        par = dict(f0=1e-4, beta=1e-11, depth=100.0, linear=linear)
        par.update(kw)
        ends = lambda *shape: rng.standard_normal(shape) * 10.0 ** rng.uniform(low, high, shape)
        for base in (0.0, 100.0):
            h, u, v = base + ends(ny, nx), ends(ny, nx), ends(ny + 1, nx)
            o, p = OraclePlane(nx, ny, nx * 1e4, ny * 1.1e4, **par), engine.Plane(nx, ny, nx * 1e4, ny * 1.1e4, **par)
            o.set(h, u, v)
            p.set_h_from_grid(h).set_u_from_grid(u).set_v_from_grid(v)
            for _ in range(3):
                o.step(10.0)
                p.step(10.0)
            for a, b in zip(p.get(), o.get()):
                assert same_bits(a, b)
