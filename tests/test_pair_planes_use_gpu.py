"""When the sweeps read couplings as planes: a solve in one launch asks for no memory for
them, and a solver of separate launches goes over to them with face weights, back
without, and over again, each time with the results of a solver that never changed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def faces(shape):
    nx, ny, nz = shape
    return [(nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1)]


def weights(shape, seed):
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(seed)
    w = {}
    for a, f in enumerate(faces(shape)):
        v = rng.uniform(0.2, 1.0, (f[2], f[1], f[0])).astype(np.float32)
        v[:, : f[1] // 2] = 1.0
        w["uvw"[a]] = Field("float", f).from_array(v.ravel())
    return w


def solver(shape, levels, **kw):
    from tsl_array_n_gb300 import fluxflow as ff
    nx, ny, nz = shape
    dims = 3 if nz > 1 else 2
    active = np.zeros((nz, ny, nx), np.uint8)
    active[:, :, nx - 1] = 1
    make = ff.create_grid_pressure_solver3 if dims == 3 else ff.create_grid_pressure_solver2
    h = (1.0 / nx,) * 3
    s = make(shape[:dims], h[:dims], multigrid={"numberOfLevels": levels, "coarseSolve": "sweeps"},
             dirichlet=(active.ravel(), np.full(active.size, 0.25, np.float32)), precision="mixed", tolerance=1e-6,
             max_iterations=300, **kw)
    rng = np.random.default_rng(4)
    vel = [0.3 * rng.standard_normal(int(np.prod(f))).astype(np.float32) for f in faces(shape)]
    return s, ff.FaceCenteredGrid3(shape, h).set(*vel), ff.FaceCenteredGrid3(shape, h)


def solve(s, grid, out):
    s.pressure.fill(0.0)
    d = s.project(grid, out)()
    assert d["converged"]
    return d["iterations"], s.pressure.to_array().copy()


def test_one_launch_takes_no_planes(gpu):
    torch = pytest.importorskip("torch")
    shape, w = (96, 96, 64), weights((96, 96, 64), 1)
    pair = [solver(shape, 4, face_weights=w) for _ in range(2)]
    gpu.synchronize()
    for first, (s, grid, out) in zip((True, False), pair):   # (the first loads the kernels)
        before = torch.cuda.mem_get_info(0)[0]
        s.settings.maxIterations = 2
        s.project(grid, out)()
        gpu.synchronize()
        assert first or torch.cuda.mem_get_info(0)[0] == before


@pytest.mark.parametrize("shape,levels", [((36, 48, 20), 2), ((64, 64, 1), 3), ((132, 34, 6), 2), ((128, 96, 96), 4)])
def test_planes_come_and_go(gpu, shape, levels):
    s, grid, out = solver(shape, levels)
    s.settings.useGraph = False
    a, b = weights(shape, 1), weights(shape, 2)
    got = []
    for fw in (None, a, b, None, a):
        s.set_face_weights(fw)
        got.append(solve(s, grid, out))
    for i, fw in enumerate((None, a, b, None, a)):
        r, g, o = solver(shape, levels, face_weights=fw)
        r.settings.useGraph = False
        ref = solve(r, g, o)
        assert got[i][0] == ref[0]
        np.testing.assert_array_equal(got[i][1], ref[1])


@pytest.mark.parametrize("shape,levels", [((32, 16, 8), 2), ((68, 20, 12), 2), ((132, 34, 6), 2), ((64, 64, 64), 4),
                                          ((96, 64, 1), 3), ((36, 48, 1), 2)])
def test_same_operator_both_forms(gpu, shape, levels):
    """The same weights as face weights (planes) and as collider weights (per cell)
    make the same operator: one application of the preconditioner and a solve by
    separate launches are equal."""
    from tsl_array_n_gb300.tsl_array_n import Field
    w = weights(shape, 5)
    n = int(np.prod(shape))
    rf = Field("float", shape).from_array(np.random.default_rng(7).standard_normal(n).astype(np.float32))
    z, p = [], []
    for kind in ("face_weights", "collider_weights"):
        s, grid, out = solver(shape, levels, **{kind: w})
        s.settings.useGraph = False   # (before the prepare that chooses the form)
        s.prepare(grid)
        zf = Field("float", shape)
        s.apply_preconditioner(rf, zf)
        z.append(zf.to_array())
        s.pressure.fill(0.0)
        s.solve(rf)
        p.append(s.pressure.to_array())
    assert np.all(np.isfinite(z[0])) and np.all(np.isfinite(p[0]))
    np.testing.assert_array_equal(z[0], z[1])
    np.testing.assert_array_equal(p[0], p[1])
