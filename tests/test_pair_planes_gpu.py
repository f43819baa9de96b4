"""The sweep that reads its couplings as planes (solvers with face weights) against
the one that reads them per cell: the same positive weights given as collider
weights make the same operator, so an application of the preconditioner and a solve
are equal.  Rows of one tile and of a partial one, one quad past a tile, one plane."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels", [((32, 16, 8), 2), ((68, 20, 12), 2), ((132, 34, 6), 2), ((64, 64, 64), 4),
                                          ((96, 64, 1), 3), ((36, 48, 1), 2)])
def test_same_operator_same_result(gpu, shape, levels):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(sum(shape))
    nx, ny, nz = shape
    dims = 3 if nz > 1 else 2
    fs = [(nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1)]
    # 1 in two thirds of the domain (plain cells beside general ones), else 0.2 .. 1
    w = {}
    for a, f in enumerate(fs):
        v = rng.uniform(0.2, 1.0, (f[2], f[1], f[0])).astype(np.float32)
        v[:, : 2 * f[1] // 3] = 1.0
        w["uvw"[a]] = v.ravel()
    active = np.zeros((nz, ny, nx), np.uint8)
    active[:, :, nx - 1] = 1
    h = (1.0 / nx,) * 3
    vel = [0.3 * rng.standard_normal(int(np.prod(f))).astype(np.float32) for f in fs]
    rf = Field("float", shape).from_array(rng.standard_normal(nx * ny * nz).astype(np.float32))
    make = ff.create_grid_pressure_solver3 if dims == 3 else ff.create_grid_pressure_solver2
    got = []
    for kind in ("face_weights", "collider_weights"):
        s = make(shape[:dims], h[:dims], **{kind: {k: Field("float", f).from_array(w[k]) for k, f in zip("uvw", fs)}},
                 multigrid={"numberOfLevels": levels, "coarseSolve": "sweeps"},
                 dirichlet=(active.ravel(), np.full(active.size, 0.25, np.float32)), precision="mixed", tolerance=1e-6,
                 max_iterations=300)
        grid, out = ff.FaceCenteredGrid3(shape, h).set(*vel), ff.FaceCenteredGrid3(shape, h)
        s.prepare(grid)
        s.settings.useGraph = False   # the sweeps themselves, not the one-launch solve
        zf = Field("float", shape)
        s.apply_preconditioner(rf, zf)
        got.append(zf.to_array())
    assert np.all(np.isfinite(got[0]))
    np.testing.assert_array_equal(got[0], got[1])
