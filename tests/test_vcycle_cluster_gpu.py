"""The coarse V-cycle on one cluster (a first coarse level of up to 65536 cells) and
over the grid (one row more) against one launch per pass, with the sweeps of the
levels above in work items of one plane and more.  The two sides round the same sums
in different orders: one FP32 application of a few sweeps a level, so 1e-5."""
import numpy as np
import pytest
from test_resident_gpu import rel, solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,levels,coarse", [((128, 64, 64), 4, "sweeps"), ((136, 64, 64), 4, "sweeps"),
                                                 ((512, 512, 1), 5, "sweeps"), ((512, 544, 1), 5, "sweeps"),
                                                 ((256, 128, 40), 4, "sweeps"), ((96, 48, 48), 4, "direct"),
                                                 ((64, 32, 4), 2, "sweeps"), ((256, 64, 64), 4, "direct")])
def test_preconditioner(gpu, shape, levels, coarse):
    from tsl_array_n_gb300.tsl_array_n import Field
    s, grid, _ = solver_for(shape, levels, coarse, "mixed", 5)
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
    assert rel(z[0], z[1]) < 1e-5
