"""The solve in one launch against one launch per pass with variable density: every
cell's couplings its own, cells beside Dirichlet cells, couplings kept in shared memory
and (more cells than there is room for) read from memory.  The same operations in the
same order, so the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((32, 12, 8), 2, "direct"), ((36, 44, 42), 2, "sweeps"), ((64, 32, 32), 4, "sweeps"), ((96, 64, 1), 3, "direct"),
         ((256, 192, 1), 4, "sweeps"), ((64, 64, 48), 4, "sweeps"), ((320, 240, 1), 5, "sweeps"), ((64, 48, 40), 3, "direct")]


@pytest.mark.parametrize("collider", [False, True])
@pytest.mark.parametrize("shape,levels,coarse", CASES)
def test_variable_density_is_the_same_solve(gpu, shape, levels, coarse, collider):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(sum(shape))
    nx, ny, nz = shape
    dims = 3 if nz > 1 else 2
    fs = [(nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1)]
    fw, cw = {}, {}
    for a, f in enumerate(fs):
        v = np.where(rng.random((f[2], f[1], f[0])) < 0.5, 1.0, 0.001).astype(np.float32)
        fw["uvw"[a]] = Field("float", f).from_array((v * rng.uniform(0.5, 1.0, v.shape).astype(np.float32)).ravel())
        w = np.ones((f[2], f[1], f[0]), np.float32)
        w[: max(1, nz // 4), : ny // 3, : nx // 3] = 0.0
        w[: max(1, nz // 4), : ny // 3, nx // 3] = 0.4
        cw["uvw"[a]] = Field("float", f).from_array(w.ravel())
    active = rng.random((nz, ny, nx)) < 0.02
    active[:, :, nx - 1] = True
    make = ff.create_grid_pressure_solver3 if dims == 3 else ff.create_grid_pressure_solver2
    h = (1.0 / nx,) * 3
    s = make(shape[:dims], h[:dims], face_weights=fw, collider_weights=cw if collider else None,
             multigrid={"numberOfLevels": levels, "coarseSolve": coarse},
             dirichlet=(active.ravel().astype(np.uint8), rng.standard_normal(active.size).astype(np.float32)),
             precision="mixed", tolerance=1e-6, max_iterations=60)
    vel = [0.3 * rng.standard_normal(int(np.prod(f))).astype(np.float32) for f in fs]
    grid, out = ff.FaceCenteredGrid3(shape, h).set(*vel), ff.FaceCenteredGrid3(shape, h)
    got = []
    for one in (True, False):
        s.settings.useGraph = one
        s.pressure.fill(0.0)
        d = dict(s.project(grid, out)())
        got.append((d["iterations"], d["residual"], s.pressure.to_array().copy(), [np.array(v) for v in out.get()]))
    a, b = got
    assert a[0] == b[0] and a[1] == b[1] and np.all(np.isfinite(a[2]))
    np.testing.assert_array_equal(a[2], b[2])
    for v, w in zip(a[3], b[3]):
        np.testing.assert_array_equal(v, w)
