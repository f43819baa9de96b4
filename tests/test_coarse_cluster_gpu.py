"""The coarsest level's sweeps on one cluster against one launch a colour pass (or
one block): the same operations, so the results are equal.  Coarsest levels with odd
extents, fewer rows than blocks, one block's cells and one more pair, a length that
the blocks do not divide, the most cells a cluster takes and more than that."""
import numpy as np
import pytest
from test_resident_gpu import solver_for

pytestmark = pytest.mark.gpu

CASES = [((6, 10, 14), 2), ((90, 6, 1), 2), ((18, 16, 14), 2), ((34, 36, 34), 2), ((16, 16, 32), 2), ((34, 16, 32), 2),
         ((90, 54, 66), 2), ((74, 70, 1), 2), ((512, 512, 1), 2), ((514, 512, 1), 2), ((128, 64, 64), 2), ((36, 20, 28), 3)]


@pytest.mark.parametrize("shape,levels", CASES)
def test_preconditioner_is_the_same(gpu, shape, levels):
    from tsl_array_n_gb300.tsl_array_n import Field
    s, grid, _ = solver_for(shape, levels, "sweeps", "fp32", 5)
    s.prepare(grid)
    n = int(np.prod(shape))
    rf = Field("float", shape).from_array(np.random.default_rng(7).standard_normal(n).astype(np.float32))
    z = []
    for one in (True, False):
        s.settings.coarseTail = one
        zf = Field("float", shape)
        s.apply_preconditioner(rf, zf)
        z.append(zf.to_array())
    assert np.all(np.isfinite(z[0]))
    np.testing.assert_array_equal(z[0], z[1])
