"""The trace and the advection where their short forms begin and end: points
within a cell of every end of the arrays and past it, grids one and two cells
thick, rows shorter than a warp and with odd remainders, spacings that are and
are not powers of two, paths of up to three substeps, a collider cutting them.
Every operation rounds as the oracle's does, so the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [((5, 4, 3), (0.25, 0.25, 0.25)), ((33, 9, 1), (0.1, 0.1, 0.1)), ((64, 8, 2), (0.125, 0.25, 0.5)),
         ((31, 17, 11), (0.07, 0.11, 0.13)), ((97, 3, 5), (1.0 / 97, 1.0 / 3, 0.2)), ((40, 36, 1), (2.0, 2.0, 2.0))]


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("with_collider", [False, True])
@pytest.mark.parametrize("shape,h", GRIDS)
def test_advect_and_trace(gpu, oracle, shape, h, with_collider, order):
    from tsl_array_n_gb300 import fluxflow as ff
    rng = np.random.default_rng(sum(shape) + order)
    nx, ny, nz = shape
    o, dt = (0.0, 0.0, 0.0), 0.5
    sizes = [(nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1)]
    u, v, w = ((rng.uniform(-6, 6, n) * (rng.random(n) < 0.9) * min(h)).astype(np.float32) for n in sizes)
    vel = ff.FaceCenteredGrid3(shape, h, o).set(u, v, w)
    mark = tuple(np.full_like(x, -3.0) for x in (u, v, w))
    out = ff.FaceCenteredGrid3(shape, h, o).set(*mark)
    col = phi = None
    if with_collider:
        col = ff.create_sdf_static_collider3(*shape, *h)
        col.add_shapes([{"type": "sphere", "center": [0.5 * nx * h[0], 0.4 * ny * h[1], 0.5 * nz * h[2]],
                         "radius": 0.3 * ny * h[1]}])
        phi = col.phi.to_array()
    adv = ff.create_semi_lagrangian_advection_solver3(velocity_grid=vel, collider=col, dt=dt, order=order)
    adv.advect_face_centered3(vel, out)()
    for g, r in zip(out.get(), oracle.advect_faces(shape, h, o, u, v, w, phi, dt, order=order, out=mark)):
        np.testing.assert_array_equal(np.asarray(g, np.float32).ravel(), np.asarray(r, np.float32).ravel())
