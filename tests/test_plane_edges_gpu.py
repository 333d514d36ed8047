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


# spacings L / n whose two-operation quotient is wrong for one fraction (csrc/fixed_div.cuh takes the IEEE division there)
EXCEPTIONAL = [(22, 5.0e5, "0x1.5c4ed08ba2e88p+0"), (26, 3.1e6, "0x1.cad18a9be5be4p+0"), (30, 1.3e6, "0x1.632798aaaaaadp+0"),
               (37, 1.1e6, "0x1.0061cc40939aep+0")]


@pytest.mark.parametrize("n,length,x", EXCEPTIONAL)
@pytest.mark.parametrize("along", ["x", "y"])
def test_the_exceptional_dividend_of_a_spacing(engine, n, length, x, along):
    """Velocity differences that are exactly the spacing's exceptional dividend, times powers of two and of both signs."""
    x = float.fromhex(x)
    nx, ny = (n, 24) if along == "x" else (24, n)
    lx, ly = (length, 2.4e5) if along == "x" else (2.4e5, length)
    par = dict(f0=0.0, beta=0.0, depth=100.0)
    for scale in (0.125, 1.0, 16.0, -2.0):
        h, u, v = np.full((ny, nx), 100.0), np.zeros((ny, nx)), np.zeros((ny + 1, nx))
        if along == "x":
            v[1:ny, ::2] = x * scale
            u[:, :] = 1.0
        else:
            u[::2, :] = x * scale
            v[1:ny, :] = 1.0
        o, p = OraclePlane(nx, ny, lx, ly, **par), engine.Plane(nx, ny, lx, ly, **par)
        o.set(h, u, v)
        p.set_h_from_grid(h).set_u_from_grid(u).set_v_from_grid(v)
        o.step(0.25)
        p.step(0.25)
        for a, b in zip(p.get(), o.get()):
            assert same_bits(a, b)


@pytest.mark.parametrize("log2", [-480, -110, -60, 60, 110, 480, 520])
@pytest.mark.parametrize("kw", [{}, dict(viscosity=3.0), dict(linear=True)])
def test_spacings_beyond_the_proven_ones(engine, log2, kw):
    """Spacings whose squares, or which themselves, leave 2^-100 .. 2^100: every division takes the general path."""
    nx, ny = 37, 21
    rng = np.random.default_rng(log2 + 600)
    s = 2.0 ** log2
    par = dict(f0=1e-4, beta=0.0, depth=100.0, **kw)
    h, u, v = 100.0 + rng.standard_normal((ny, nx)), rng.standard_normal((ny, nx)), rng.standard_normal((ny + 1, nx))
    o, p = OraclePlane(nx, ny, 1.3 * nx * s, 1.7 * ny * s, **par), engine.Plane(nx, ny, 1.3 * nx * s, 1.7 * ny * s, **par)
    o.set(h, u, v)
    p.set_h_from_grid(h).set_u_from_grid(u).set_v_from_grid(v)
    dt = 2.0 ** -4 * min(s, 1e6)
    for _ in range(2):
        o.step(dt)
        p.step(dt)
    for a, b in zip(p.get(), o.get()):
        assert same_bits(a, b)


def test_the_stencils_division_on_the_device(engine):
    """As tests/test_fixed_div2_cpu.py, on the GPU: answered, refused and exceptional dividends."""
    import ctypes as C

    rng = np.random.default_rng(9)
    spacings = np.array([length / n for n, length, _ in EXCEPTIONAL] + [1e6 / n for n in range(5, 400, 7)] + list(2.0 ** rng.uniform(-99, 99, 60)))
    x = np.concatenate([rng.standard_normal(20000) * 10.0 ** rng.uniform(-300, 300, 20000),
                        (np.outer(spacings, rng.integers(1, 2 ** 20, 100)) * 2.0 ** -10).ravel(),
                        np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7e308])])
    counts = np.zeros(2, np.int64)
    lib = engine.load_library()
    engine._check(lib.lmw_division_selftest(x.ctypes.data_as(C.POINTER(C.c_uint64)), x.size, spacings.ctypes.data_as(C.POINTER(C.c_double)),
                                            spacings.size, counts.ctypes.data_as(C.POINTER(C.c_longlong))))
    assert counts[0] == 0
