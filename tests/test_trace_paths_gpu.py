"""The trace and the advection where their short forms begin and end: points
within a cell of every end of the arrays and past it, grids one and two cells
thick, rows shorter than a warp and with odd remainders, grids below and above the
size from which the short form is taken, spacings that are and are not powers of two, paths of up to three substeps, a collider cutting them.
Every operation rounds as the oracle's does, so the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [((5, 4, 3), (0.25, 0.25, 0.25)), ((33, 9, 1), (0.1, 0.1, 0.1)), ((64, 8, 2), (0.125, 0.25, 0.5)),
         ((31, 17, 11), (0.07, 0.11, 0.13)), ((97, 3, 5), (1.0 / 97, 1.0 / 3, 0.2)), ((40, 36, 1), (2.0, 2.0, 2.0)),
         ((130, 90, 92), (0.01, 0.02, 0.01)), ((1050, 1001, 1), (0.5, 0.5, 0.5)), ((104, 101, 103), (0.25, 0.25, 0.25))]


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


def test_output_over_another_components_input(gpu):
    """A cube's face fields have one length, so an output may lie over another
    component's input: the components are then advected one after the other."""
    from tsl_array_n_gb300 import fluxflow as ff
    n = 20
    rng = np.random.default_rng(4)
    u, v, w = (rng.uniform(-1, 1, (n + 1) * n * n).astype(np.float32) for _ in range(3))
    shape, h, o = (n, n, n), (0.1,) * 3, (0.0,) * 3

    def grid(*f):
        return ff.FaceCenteredGrid3(shape, h, o).set(*f)

    adv = ff.create_semi_lagrangian_advection_solver3(velocity_grid=grid(u, v, w), dt=0.05)

    def apart(*f):
        out = grid(u * 0, v * 0, w * 0)
        adv.advect_face_centered3(grid(*f), out)()
        return [np.array(x) for x in out.get()]

    inp, out = grid(u, v, w), grid(u * 0, v * 0, w * 0)
    out.data_u = inp.data_v
    adv.advect_face_centered3(inp, out)()
    first = apart(u, v, w)
    second = apart(u, first[0], w)   # component 1 reads component 0's result
    np.testing.assert_array_equal(out.data_u.to_array(), first[0])
    np.testing.assert_array_equal(out.data_v.to_array(), second[1])
    np.testing.assert_array_equal(out.data_w.to_array(), first[2])
