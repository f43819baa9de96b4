"""kernelLaunches of a solve by separate launches: what one iteration more adds is the
two CG kernels, the loop's control kernel, the V-cycle's kernels as they are enqueued,
and r.z where no sweep forms it."""
import numpy as np
import pytest
from test_resident_gpu import solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels,tail,expect", [
    # two launches a sweep, residual, restriction, prolongation; the coarsest level's
    # 20 sweeps (45 x 27 x 33) on one cluster, or 40 colour passes
    ((90, 54, 66), 2, True, 3 + (8 + 3) + 1 + 1), ((90, 54, 66), 2, False, 3 + (8 + 3) + 40 + 1),
    # one launch a sweep, two for residual and restriction; levels 1 to 3 in one launch,
    # or by themselves with the coarsest in one block
    ((128, 96, 96), 4, True, 3 + (4 + 3) + 1), ((128, 96, 96), 4, False, 3 + 3 * (4 + 3) + 1),
    # rows too short for the staged sweep: one kernel for residual and restriction
    ((28, 20, 12), 2, True, 3 + (4 + 2) + 1),
    # one level: its sweeps and r.z
    ((20, 12, 8), 1, True, 3 + 1 + 1)])
def test_launches_of_one_iteration(gpu, shape, levels, tail, expect):
    s, grid, out = solver_for(shape, levels, "sweeps", "mixed", 3)
    s.settings.coarseTail = tail
    s.settings.tolerance = 1e-30
    got = []
    for n in (1, 2, 4):
        s.settings.maxIterations = n
        s.pressure.fill(0.0)
        d = s.project(grid, out)()
        assert d["iterations"] == n
        got.append(d["kernelLaunches"])
    assert got[1] - got[0] == expect and got[2] - got[1] == 2 * expect
