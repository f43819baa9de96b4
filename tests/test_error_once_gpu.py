"""A call that CUDA refuses (memory nobody has) is reported by that call and by no later
one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["host", "field"])
def test_refused_allocation_does_not_fail_the_next_call(gpu, what):
    from tsl_array_n_gb300 import _lib, fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    lib = _lib.load()
    shape, h = (16, 12, 8), (1.0 / 16,) * 3
    active = np.zeros(16 * 12 * 8, np.uint8)
    active[0] = 1
    s = ff.create_grid_pressure_solver3(shape, h, dirichlet=(active, np.zeros(active.size, np.float32)))
    rng = np.random.default_rng(0)
    vel = [rng.standard_normal(int(np.prod([m + (a == b) for b, m in enumerate(shape)]))).astype(np.float32) for a in range(3)]
    grid, out = ff.FaceCenteredGrid3(shape, h).set(*vel), ff.FaceCenteredGrid3(shape, h)
    if what == "host":
        p = C.c_void_p()
        assert lib.ff_host_alloc(C.c_size_t(1 << 50), C.byref(p)) != 0
    else:
        f = C.c_void_p()
        assert lib.ff_field_create(gpu.handle, 0, 3, (C.c_int * 3)(1 << 16, 1 << 16, 1 << 10), C.byref(f)) == -3
    assert s.project(grid, out)()["iterations"] > 0
    Field("float", shape).fill(1.0)
