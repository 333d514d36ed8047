"""A tensor-core wait of the FP64 sums that ran out (its code written on the host): every call that ends such a launch reports
it once, and the engine then serves the next state; grids, which take plain sums, are not touched by it."""
import ctypes as C

import numpy as np
import pytest

from test_tc64_gpu import initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["step", "run", "stable_dt", "kernel_times"])
def test_a_timed_out_wait_is_reported_once(engine, call):
    lib, state = engine.load_library(), initial(21, 4)
    s, fresh = engine.Sphere(21, diffusion=1e16), engine.Sphere(21, diffusion=1e16)
    for x in (s, fresh):
        x.set_state(*state)
    grid = s.grid_vorticity()
    engine._check(lib.lmw_sphere_inject_fp64_error(s._h, 12))
    assert np.array_equal(s.grid_vorticity(), grid)  # plain sums
    with pytest.raises(engine.DeviceError, match="a wait on the tensor cores timed out"):
        {"step": lambda: s.step(600.0), "run": lambda: s.run(3600.0, 600.0), "stable_dt": s.stable_dt,
         "kernel_times": lambda: engine._check(lib.lmw_sphere_kernel_times(s._h, C.c_double(600.0), 2, (C.c_double * 3)()))}[call]()
    s.set_state(*state)
    for x in (s, fresh):
        x.step(600.0)
        x.run(3600.0, 600.0)
    for a, b in zip(s.get_state(), fresh.get_state()):
        assert np.array_equal(a, b)


def test_only_engines_with_such_waits_take_the_code(engine):
    lib = engine.load_library()
    for s in (engine.Sphere(21, precision=engine.FP32), engine.Sphere(171, max_truncation=341)):
        with pytest.raises(ValueError, match="does not use the FP64 sums"):
            engine._check(lib.lmw_sphere_inject_fp64_error(s._h, 12))
