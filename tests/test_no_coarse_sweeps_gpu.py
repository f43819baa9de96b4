"""A V-cycle whose coarsest level is swept zero times leaves zero there, also where that
level is level 0, whose x another preconditioner has just written, and whichever way
the coarsest sweeps would run."""
import numpy as np
import pytest
from test_resident_gpu import solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [True, False])
@pytest.mark.parametrize("shape", [(8, 4, 4), (32, 3, 1), (6, 5, 7), (64, 16, 8), (90, 10, 6)])
def test_one_level_and_no_sweeps_is_zero(gpu, shape, tail):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    _, grid, _ = solver_for(shape, 1, "sweeps", "fp32", 3)
    dims = 3 if shape[2] > 1 else 2
    make = ff.create_grid_pressure_solver3 if dims == 3 else ff.create_grid_pressure_solver2
    n = int(np.prod(shape))
    active = np.zeros(n, np.uint8)
    active[-1] = 1
    s = make(shape[:dims], (1.0 / shape[0],) * dims, dirichlet=(active, np.zeros(n, np.float32)),
             multigrid={"numberOfLevels": 1, "numberOfCoarsestIterations": 0})
    s.prepare(grid)
    s.settings.coarseTail = tail
    r = Field("float", shape).from_array(np.random.default_rng(2).standard_normal(n).astype(np.float32))
    z = Field("float", shape)
    s.settings.preconditioner = "jacobi"
    s.apply_preconditioner(r, z)
    assert np.any(z.to_array() != 0)
    s.settings.preconditioner = "multigrid"
    s.apply_preconditioner(r, z)
    np.testing.assert_array_equal(z.to_array(), np.zeros(n, np.float32))
