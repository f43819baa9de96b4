"""The whole-array sums beside a solve (the start's norm of reportNoiseFloor, the
residuals that a warm start compares) on solvers with fewer sums of their own than
those have blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(shape, levels=1):
    from tsl_array_n_gb300 import fluxflow as ff
    dims = 3 if shape[2] > 1 else 2
    make = ff.create_grid_pressure_solver3 if dims == 3 else ff.create_grid_pressure_solver2
    n = int(np.prod(shape))
    active = np.zeros(n, np.uint8)
    active[0] = 1
    return make(shape[:dims], (0.25,) * dims, dirichlet=(active, np.zeros(n, np.float32)),
                multigrid={"numberOfLevels": levels}, precision="mixed", tolerance=1e-5)


@pytest.mark.parametrize("shape", [(2, 2, 1), (4, 4, 4), (32, 3, 1), (13, 11, 9), (64, 32, 1), (32, 16, 16)])
def test_noise_floor_of_small_solvers(gpu, shape):
    from tsl_array_n_gb300.tsl_array_n import Field
    n = int(np.prod(shape))
    rng = np.random.default_rng(n)
    s = solver(shape)
    x0, b = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    x0[0] = b[0] = 0.0
    s.settings.reportNoiseFloor = True
    s.pressure.from_array(x0)
    d = s.solve(Field("float", shape).from_array(b))
    expected = 2.0 ** -24 * (3 if shape[2] > 1 else 2) * 2.0 / 0.0625 * np.linalg.norm(x0.astype(np.float64))
    assert abs(d["noiseFloor"] / expected - 1) < 1e-6


@pytest.mark.parametrize("shape", [(8, 4, 4), (12, 8, 4)])
def test_warm_start_of_small_solvers(gpu, shape):
    """An untrained network's guess is compared with the previous pressure, and the
    solve converges from the better one."""
    pytest.importorskip("torch")
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.warmstart import UNetWarmStart, attach
    rng = np.random.default_rng(3)
    s = solver(shape, 2)
    attach(s, UNetWarmStart(seed=5))
    sizes = [(shape[0] + 1) * shape[1] * shape[2], shape[0] * (shape[1] + 1) * shape[2], shape[0] * shape[1] * (shape[2] + 1)]
    grid = ff.FaceCenteredGrid3(shape, (0.25,) * 3).set(*[rng.standard_normal(k).astype(np.float32) for k in sizes])
    d = s.project(grid, ff.FaceCenteredGrid3(shape, (0.25,) * 3))()
    assert d["converged"] and d["warmStart"] in (0, 1)
