"""The FP64 Legendre sums on the tensor cores (csrc/sphere_tc64.cuh) and the FP64 grid kernel (csrc/sphere.cu) at the sizes
where their tiles end: the smallest grids (padding to 16 latitudes, transforms shorter than a warp), ragged
coefficient counts, one and two latitude slices, and member tiles that are not full."""
import numpy as np
import pytest

from oracle_lib import OracleSphere

pytestmark = pytest.mark.gpu

# the bars of tests/test_sphere_gpu.py: zeta and Phi 1e-12 of their scale; delta 1e-12, and above T106 the floor that
# the reference keeps against itself there (3e-11 of the vorticity scale: a small difference of large terms)
TOL, DELTA_HIGH = 1e-12, 3e-11


def initial(T, seed):
    """A balanced flow with a divergent part, spectral, in the reference layout; heights stay positive."""
    rng = np.random.default_rng(seed)
    o = OracleSphere(T, diffusion=1e15)
    h, u, v = o.turbulence_grids(seed, 8000.0, 30.0, max(2, T // 2))
    o.set_state_grid(h, u, v)
    z, d, f = o.get_state()
    M = T + 1
    m, n = np.divmod(np.arange(M * M), M)
    noise = rng.standard_normal(M * M) + 1j * rng.standard_normal(M * M) * (m > 0)
    d = np.where((n >= np.maximum(m, 1)) & (n <= T // 2 + 1), noise, 0) * 0.1 * np.abs(z).max()
    return z, d, f


@pytest.mark.parametrize("T", [4, 5, 6, 10, 14, 15, 16, 22, 30, 31, 33, 47, 62, 64, 86, 107, 170])
def test_steps_match_the_oracle_for_one_and_three_members(engine, T):
    states = [initial(T, 100 * T + k) for k in range(3)]
    dt = 20000.0 / T
    many = engine.Sphere(T, diffusion=1e15, members=3)
    for b, s in enumerate(states):
        many.set_state(*s, member=b)
    many.step(dt)
    many.step(dt)
    for b, s in enumerate(states):
        one = engine.Sphere(T, diffusion=1e15)
        one.set_state(*s)
        one.step(dt)
        one.step(dt)
        for x, y in zip(one.get_state(), many.get_state(member=b)):
            assert np.array_equal(x, y)  # the sums do not depend on the batch
        if b == 0 or T < 64:
            o = OracleSphere(T, diffusion=1e15)
            o.set_state(*s)
            o.step(dt)
            o.step(dt)
            got, ref = one.get_state(), o.get_state()
            wind = max(np.abs(ref[0]).max(), np.abs(ref[1]).max())
            assert np.abs(got[0] - ref[0]).max() <= TOL * wind
            assert np.abs(got[1] - ref[1]).max() <= (TOL if T <= 106 else DELTA_HIGH) * wind
            assert np.abs(got[2] - ref[2]).max() <= TOL * np.abs(ref[2]).max()


def test_a_value_that_is_not_finite_reaches_every_field(engine):
    """As with plain sums, a NaN or an infinity in one coefficient is not lost in the digits."""
    for bad in (np.nan, np.inf):
        s = engine.Sphere(21)
        s.turbulence(3)
        z, d, f = s.get_state()
        d[2 * 22 + 5] = bad
        s.set_state(z, d, f)
        s.step(60.0)
        assert all(not np.isfinite(x).all() for x in s.get_state())
        with pytest.raises(RuntimeError):
            s.run(120.0, 60.0)
