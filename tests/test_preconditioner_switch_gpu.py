"""Multigrid with a direct coarsest solve chosen after prepares with another
preconditioner, which make no factorisation: for the first time, and after the operator
has changed meanwhile.  The results are those of a solver that had multigrid all along."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solver(shape, levels, weights, preconditioner):
    from tsl_array_n_gb300 import fluxflow as ff
    n = int(np.prod(shape))
    active = np.zeros(n, np.uint8)
    active[n // 2] = 1
    return ff.create_grid_pressure_solver3(shape, (1.0 / shape[0],) * 3, face_weights=weights, preconditioner=preconditioner,
                                           dirichlet=(active, np.zeros(n, np.float32)), precision="mixed", tolerance=1e-6,
                                           multigrid={"numberOfLevels": levels, "coarseSolve": "direct"}, max_iterations=400)


@pytest.mark.parametrize("shape,levels", [((16, 12, 8), 2), ((48, 24, 24), 3), ((18, 12, 10), 2), ((128, 96, 96), 4)])
def test_direct_coarsest_after_another_preconditioner(gpu, shape, levels):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(1)
    fs = [tuple(m + (a == b) for b, m in enumerate(shape)) for a in range(3)]
    w1, w2 = ([rng.uniform(lo, 1.0, int(np.prod(f))).astype(np.float32) for f in fs] for lo in (0.5, 0.01))
    vel = [rng.standard_normal(int(np.prod(f))).astype(np.float32) for f in fs]
    grid, out = ff.FaceCenteredGrid3(shape, (1.0 / shape[0],) * 3).set(*vel), ff.FaceCenteredGrid3(shape, (1.0 / shape[0],) * 3)

    def fields(w):
        return {k: Field("float", f).from_array(v) for k, f, v in zip("uvw", fs, w)}

    def solve(s):
        s.pressure.fill(0.0)
        d = s.project(grid, out)()
        return d["converged"], d["iterations"], s.pressure.to_array().copy()

    fw = fields(w1)
    s = solver(shape, levels, fw, "jacobi")
    s.settings.maxIterations = 1
    s.project(grid, out)()
    s.settings.maxIterations = 400
    for w in (w1, w2):
        for k, v in zip("uvw", w):
            fw[k].from_array(v)
        s.settings.preconditioner = "none"
        s.settings.maxIterations = 1
        s.project(grid, out)()
        s.settings.maxIterations = 400
        s.settings.preconditioner = "multigrid"
        got = solve(s)
        ref = solve(solver(shape, levels, fields(w), "multigrid"))
        assert got[0] and got[:2] == ref[:2]
        np.testing.assert_array_equal(got[2], ref[2])
