"""The PCG solve in one launch, on one cluster and over the grid, against one launch
per pass: the same operations in the same order, sums included, so the results are
equal.  Extents where the distribution over the blocks can go wrong: fewer rows than
blocks, rows that do not divide, one tile and several in x with a narrow last one,
the most cells and the most rows a block takes, a spread coarsest level with odd
extents, a direct coarsest solve on either side of its limit, work items of several
planes."""
import numpy as np
import pytest
from test_resident_gpu import solver_for

pytestmark = pytest.mark.gpu

CASES = [((32, 4, 2), 2, "sweeps"), ((36, 6, 1), 2, "sweeps"), ((32, 26, 22), 2, "sweeps"), ((66 * 2, 20, 6), 2, "sweeps"),
         ((64, 32, 32), 4, "sweeps"), ((256, 192, 1), 4, "sweeps"), ((256, 256, 1), 5, "sweeps"), ((32, 2048, 1), 4, "sweeps"), ((68, 70, 1), 2, "sweeps"),
         ((32, 12, 8), 2, "direct"), ((32, 24, 24), 2, "direct"), ((48, 24, 16), 3, "direct"), ((96, 64, 1), 3, "direct"),
         ((64, 64, 48), 4, "sweeps"), ((320, 240, 1), 5, "sweeps"), ((64, 48, 40), 3, "direct"), ((36, 44, 42), 2, "sweeps")]


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("shape,levels,coarse", CASES)
def test_one_launch_is_the_same_solve(gpu, shape, levels, coarse, precision):
    s, grid, out = solver_for(shape, levels, coarse, precision, 7)
    got = []
    for one in (True, False):
        s.settings.useGraph = one
        s.pressure.fill(0.0)
        runs = []
        for _ in range(2):   # from zero, then from the first solve's pressure
            d = dict(s.project(grid, out)())
            runs.append((d["iterations"], d["residual"], s.pressure.to_array().copy(), [np.array(v) for v in out.get()]))
        got.append(runs)
    for a, b in zip(*got):
        assert a[0] == b[0] and a[1] == b[1]
        np.testing.assert_array_equal(a[2], b[2])
        for v, w in zip(a[3], b[3]):
            np.testing.assert_array_equal(v, w)
