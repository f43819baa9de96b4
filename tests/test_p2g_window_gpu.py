"""P2G through shared-memory windows against the FP32 oracle, bit for bit:
particle lists in cell order, shuffled, and in one cell; one and several runs
a block; grids whose windows are cut to the capacity or cover the domain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert a.shape == b.shape
    bad = a != b
    assert not bad.any(), f"{bad.sum()} of {a.size} differ"


@pytest.mark.parametrize("shape,n,order", [((7, 5, 3), 1, "cells"), ((7, 5, 3), 513, "shuffled"),
                                           ((260, 6, 4), 60000, "cells"), ((64, 40, 33), 500000, "cells"),
                                           ((64, 40, 33), 500000, "shuffled"), ((300, 3, 2), 20000, "one cell")])
def test_p2g_windows(gpu, oracle, shape, n, order):
    from tsl_array_n_gb300 import fluxflow as ff
    rng = np.random.default_rng(17)
    h, o = (0.25, 0.125, 0.25), (0.5, 0.0, -1.0)
    cell = np.sort(rng.integers(0, np.prod(shape), n)) if order != "one cell" else np.full(n, shape[0] - 1)
    idx = np.stack([cell % shape[0], cell // shape[0] % shape[1], cell // (shape[0] * shape[1])], 1)
    pos = ((idx + rng.random((n, 3))) * h + o).astype(np.float32)
    if order == "shuffled":
        pos = pos[rng.permutation(n)]
    pos[0] = [-5.0, 1e9, 2.0]     # far outside: clamped to the nearest faces
    vel = (3 * rng.standard_normal((n, 3))).astype(np.float32)
    grid = ff.FaceCenteredGrid3(shape, h, o)
    s = ff.create_grid_flip_solver3(velocity_grid=grid, max_particles=n, dt=0.01)
    s.positions.from_array(pos.ravel())
    s.velocities.from_array(vel.ravel())
    s.stage("p2g")
    ref = oracle.flip_p2g(shape, h, o, pos, vel)
    for g, r in zip(grid.get(), ref[0]):
        same(g, r)
