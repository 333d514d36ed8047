"""FP64 above T170 (csrc/sphere.cu, csrc/sphere_tracer.cuh): the plain Legendre sums, the grid clusters at 1024 points and the
tracer's own kernels, over several steps launched singly and as a graph."""
import numpy as np
import pytest

from oracle_lib import OracleSphere
from test_stage_forms_gpu import tracer
from test_tc64_gpu import initial

pytestmark = pytest.mark.gpu

# the bars of tests/test_sphere_gpu.py (zeta, Phi 1e-12; delta above T106 3e-11 of the vorticity) and tests/test_tracer_gpu.py
TOL, DELTA_HIGH = 1e-12, 3e-11


def widened(T, seed):
    """A T170 flow whose coefficients are placed in the triangle of T."""
    out = []
    for x in initial(170, seed):
        a = np.zeros((T + 1, T + 1), complex)
        a[:171, :171] = np.asarray(x).reshape(171, 171)
        out.append(a.ravel())
    return out


@pytest.mark.parametrize("T", [171, 213, 341])
def test_flow_and_tracer_above_t170(engine, T):
    dt, steps = 16.0, 5
    states = [widened(T, 7 * T + k) for k in range(2)]
    make = lambda members=1: engine.Sphere(T, diffusion=1e15, members=members, max_truncation=341)
    many = make(2)
    grids = [tracer(T, many.nlat, many.nlon, 11 * T + b) for b in range(2)]
    for b in range(2):
        many.set_state(*states[b], member=b)
        many.set_tracer_grid(grids[b], member=b)
    for _ in range(steps):
        many.step(dt)  # the first steps launched singly, later ones as a graph
    for b in range(2):
        one, bare = make(), make()
        one.set_state(*states[b])
        bare.set_state(*states[b])
        one.set_tracer_grid(grids[b])
        one.run(steps * dt, dt)  # one graph
        for _ in range(steps):
            bare.step(dt)
        assert np.array_equal(one.tracer_state(), many.tracer_state(member=b))
        for x, y, z in zip(one.get_state(), many.get_state(member=b), bare.get_state()):
            assert np.array_equal(x, y) and np.array_equal(x, z)
        if b == 0:
            o = OracleSphere(T, diffusion=1e15, max_truncation=341)
            o.set_state(*states[0])
            o.set_tracer_grid(grids[0])
            for _ in range(steps):
                o.step(dt)
            z, d, f, q = o.get_state(with_tracer=True)
            got = one.get_state()
            wind = max(np.abs(z).max(), np.abs(d).max())
            assert np.abs(got[0] - z).max() <= TOL * wind
            assert np.abs(got[1] - d).max() <= DELTA_HIGH * wind
            assert np.abs(got[2] - f).max() <= TOL * np.abs(f).max()
            assert np.abs(one.tracer_state() - q).max() <= TOL * np.abs(q).max()
