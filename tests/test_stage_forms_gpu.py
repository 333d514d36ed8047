"""Forms of the sphere's stage kernels at the sizes where their tiles end: the FP64 stage that carries the tracer with the flow
(csrc/sphere_tc64.cuh, csrc/sphere.cu) and the FP32 sums that stage one wavenumber's coefficients in shared memory."""
import numpy as np
import pytest

from oracle_lib import OracleSphere
from test_tc64_gpu import initial

pytestmark = pytest.mark.gpu

# the bar of tests/test_tracer_gpu.py for the tracer, of the largest coefficient
TOL = 1e-12


def tracer(T, nlat, nlon, seed):
    rng = np.random.default_rng(seed)
    lam = 2 * np.pi * np.arange(nlon) / nlon
    phi = np.linspace(-1, 1, nlat)[:, None]
    k = rng.integers(1, max(2, T // 3), 3)
    return 1.0 + 0.3 * np.cos(k[0] * lam) * (1 - phi ** 2) + 0.2 * np.sin(k[1] * lam + 0.3) * (1 - phi ** 2) * phi + 0.1 * np.cos(k[2] * phi)


@pytest.mark.parametrize("T", [4, 5, 10, 15, 16, 31, 33, 47, 62, 107, 170])
def test_tracer_rides_with_the_flow(engine, T):
    dt, states = 20000.0 / T, [initial(T, 100 * T + k) for k in range(3)]
    many = engine.Sphere(T, diffusion=1e15, members=3)
    grids = []
    for b, s in enumerate(states):
        many.set_state(*s, member=b)
        grids.append(tracer(T, many.nlat, many.nlon, 7 * T + b))
        many.set_tracer_grid(grids[b], member=b)
    many.step(dt)
    many.step(dt)
    for b, s in enumerate(states):
        one, bare = engine.Sphere(T, diffusion=1e15), engine.Sphere(T, diffusion=1e15)
        one.set_state(*s)
        bare.set_state(*s)
        one.set_tracer_grid(grids[b])
        for e in (one, bare):
            e.step(dt)
            e.step(dt)
        assert np.array_equal(one.tracer_state(), many.tracer_state(member=b))
        for x, y, z in zip(one.get_state(), many.get_state(member=b), bare.get_state()):
            assert np.array_equal(x, y) and np.array_equal(x, z)  # the tracer does not touch the flow
        if b == 0:
            o = OracleSphere(T, diffusion=1e15)
            o.set_state(*s)
            o.set_tracer_grid(grids[b])
            o.step(dt)
            o.step(dt)
            ref = o.get_state(with_tracer=True)[3]
            assert np.abs(one.tracer_state() - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("T", [4, 5, 42, 43, 86, 341])
def test_fp32_sums_from_staged_coefficients(engine, T):
    """FP32 against FP64 within 1e-6 of the height (the bar of tests/test_sphere_gpu.py), and the same bits in a batch."""
    dt, states = 8000.0 / T, [initial(min(T, 170), 10 * T + k) for k in range(2)]
    if T > 170:  # the same flow, its coefficients placed in the larger triangle
        big = []
        for s in states:
            z = [np.zeros((T + 1, T + 1), complex) for _ in range(3)]
            for a, x in zip(z, s):
                a[:171, :171] = np.asarray(x).reshape(171, 171)
            big.append(tuple(a.ravel() for a in z))
        states = big
    make = lambda precision, members=1: engine.Sphere(T, diffusion=0.0, precision=precision, members=members, max_truncation=341)
    many = make(engine.FP32, 2)
    for b, s in enumerate(states):
        many.set_state(*s, member=b)
    many.step(dt)
    for b, s in enumerate(states):
        one, ref = make(engine.FP32), make(engine.FP64)
        for e in (one, ref):
            e.set_state(*s)
            e.step(dt)
        for x, y in zip(one.get_state(), many.get_state(member=b)):
            assert np.array_equal(x, y)
        f, g = one.get_state()[2], ref.get_state()[2]
        assert np.linalg.norm(f - g) <= 1e-6 * np.linalg.norm(g)


@pytest.mark.parametrize("T", [5, 15, 31, 33, 42, 62, 86])
def test_batches_that_fill_the_gpu_keep_the_bits(engine, T):
    """Past 304 (wavenumber, member) pairs the FP64 analysis takes narrower CTAs and the synthesis pairs its members."""
    B, dt, states = 304 // (T + 1) + 2, 20000.0 / T, [initial(T, 100 * T + k) for k in range(2)]
    many = engine.Sphere(T, diffusion=1e15, members=B)
    for b in range(B):
        many.set_state(*states[b % 2], member=b)
    for _ in range(3):
        many.step(dt)
    for k in range(2):
        one = engine.Sphere(T, diffusion=1e15)
        one.set_state(*states[k])
        one.run(3 * dt, dt)
        for b in range(k, B, 2):
            for x, y in zip(one.get_state(), many.get_state(member=b)):
                assert np.array_equal(x, y)
