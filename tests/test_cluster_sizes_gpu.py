"""The forms for devices that run smaller clusters or none: the one-launch solve, the
coarse V-cycle and the coarsest sweeps on 8 blocks and without a cluster (over the grid,
or level by level), against the separate launches.  Extents at which 8 blocks have every
level, some of them, and too little room."""
import numpy as np
import pytest
from test_resident_gpu import rel, solver_for

pytestmark = pytest.mark.gpu

SOLVES = [((32, 4, 2), 2, "sweeps"), ((32, 26, 22), 2, "sweeps"), ((64, 32, 32), 4, "sweeps"), ((256, 192, 1), 4, "sweeps"),
          ((32, 2048, 1), 4, "sweeps"), ((68, 70, 1), 2, "sweeps"), ((32, 24, 24), 2, "direct"), ((48, 24, 16), 3, "direct"),
          ((96, 64, 1), 3, "direct"), ((36, 44, 42), 2, "sweeps"), ((128, 128, 1), 4, "sweeps")]


@pytest.mark.parametrize("blocks", [8, 0])
@pytest.mark.parametrize("shape,levels,coarse", SOLVES)
def test_solve(gpu, shape, levels, coarse, blocks):
    s, grid, out = solver_for(shape, levels, coarse, "mixed", 7)
    got = []
    for one in (True, False):
        s.settings.clusterBlocks = blocks
        s.settings.useGraph = one
        s.pressure.fill(0.0)
        d = dict(s.project(grid, out)())
        got.append((d["iterations"], d["residual"], s.pressure.to_array().copy()))
    assert got[0][:2] == got[1][:2]
    np.testing.assert_array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("blocks", [8, 0])
@pytest.mark.parametrize("shape,levels,exact", [((90, 54, 66), 2, True), ((90, 6, 1), 2, True), ((34, 36, 34), 2, True),
                                                ((74, 70, 1), 2, True), ((36, 20, 28), 3, True), ((128, 64, 64), 4, False),
                                                ((512, 512, 1), 5, False), ((96, 48, 48), 4, False)])
def test_preconditioner(gpu, shape, levels, exact, blocks):
    """Coarsest sweeps alone are equal; whole coarse V-cycles round as level by level
    within the 1e-5 of one FP32 application."""
    from tsl_array_n_gb300.tsl_array_n import Field
    s, grid, _ = solver_for(shape, levels, "sweeps", "fp32", 5)
    s.prepare(grid)
    s.settings.clusterBlocks = blocks
    n = int(np.prod(shape))
    rf = Field("float", shape).from_array(np.random.default_rng(7).standard_normal(n).astype(np.float32))
    z = []
    for one in (True, False):
        s.settings.coarseTail = one
        zf = Field("float", shape)
        s.apply_preconditioner(rf, zf)
        z.append(zf.to_array())
    assert np.all(np.isfinite(z[0]))
    if exact:
        np.testing.assert_array_equal(z[0], z[1])
    else:
        assert rel(z[0], z[1]) < 1e-5


def test_more_blocks_than_the_device_runs_are_refused(gpu):
    from tsl_array_n_gb300._lib import FFError
    s, _, _ = solver_for((32, 4, 2), 2, "sweeps", "mixed", 7)
    for bad in (1, 4, 12, 32, -8):
        with pytest.raises(FFError):
            s.settings.clusterBlocks = bad
