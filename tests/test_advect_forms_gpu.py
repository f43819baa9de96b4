"""The two forms of the trace and the advection on either side of the sizes that choose
between them.  Advection in the short form (a grid of a million cells with power-of-two
spacings, of two million with others, most of its rows away from the ends) and, with one
row or plane less, in the straightforward one, against the FP32 oracle.  Lists of 2^23
points take the short form, their halves the straightforward one: equal, for points
inside, past every end and not finite.  Every operation rounds as the oracle's does, so
the results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((196, 73, 74), (0.25, 0.125, 0.25), 1, True), ((196, 73, 74), (0.25, 0.125, 0.25), 2, False),
         ((196, 73, 73), (0.25, 0.125, 0.25), 1, True), ((226, 100, 93), (0.1, 0.07, 0.1), 1, True),
         ((226, 100, 93), (0.1, 0.07, 0.1), 2, False), ((226, 99, 93), (0.1, 0.07, 0.1), 1, False),
         ((128, 2048, 4), (0.5, 0.5, 0.5), 1, True)]


def field(shape, h, rng, cells):
    nx, ny, nz = shape
    sizes = [(nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1)]
    return [(rng.uniform(-cells, cells, n) * (rng.random(n) < 0.9) * min(h)).astype(np.float32) for n in sizes]


def collider_for(shape, h):
    from tsl_array_n_gb300 import fluxflow as ff
    col = ff.create_sdf_static_collider3(*shape, *h)
    col.add_shapes([{"type": "sphere", "center": [0.5 * n * x for n, x in zip(shape, h)],
                     "radius": 0.3 * shape[1] * h[1]}])
    return col


@pytest.mark.parametrize("shape,h,order,with_collider", CASES)
def test_advection_at_the_line(gpu, oracle, shape, h, order, with_collider):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(sum(shape) + order)
    o, dt = (0.0, 0.0, 0.0), 0.5
    u, v, w = field(shape, h, rng, 5)
    vel = ff.FaceCenteredGrid3(shape, h, o).set(u, v, w)
    out = ff.FaceCenteredGrid3(shape, h, o).set(u, v, w)
    col = collider_for(shape, h) if with_collider else None
    phi = col.phi.to_array() if col else None
    adv = ff.create_semi_lagrangian_advection_solver3(velocity_grid=vel, collider=col, dt=dt, order=order)
    adv.advect_face_centered3(vel, out)()
    for g, r in zip(out.get(), oracle.advect_faces(shape, h, o, u, v, w, phi, dt, order=order)):
        np.testing.assert_array_equal(np.asarray(g, np.float32).ravel(), np.asarray(r, np.float32).ravel())
    s = rng.standard_normal(int(np.prod(shape))).astype(np.float32)
    a, b = Field("float", shape).from_array(s), Field("float", shape).from_array(s)
    adv.advect_scalar3(a, b)()
    np.testing.assert_array_equal(b.to_array(), oracle.advect_scalar(shape, h, o, u, v, w, phi, s, dt, order=order))


N = 1 << 23


def points(shape, h, rng, lo, hi):
    p = rng.random((N, 3), dtype=np.float32) * np.float32(hi - lo) + np.float32(lo)
    return p * (np.array(shape) * np.array(h)).astype(np.float32)


@pytest.mark.parametrize("shape,h", [((40, 24, 18), (0.25, 0.25, 0.5)), ((40, 24, 18), (0.1, 0.07, 0.11)),
                                     ((9, 70, 2), (0.1, 0.1, 0.1)), ((33, 40, 1), (0.25, 0.25, 0.25))])
@pytest.mark.parametrize("with_collider", [False, True])
def test_trace_of_many_points(gpu, oracle, shape, h, with_collider):
    from tsl_array_n_gb300 import fluxflow as ff
    from tsl_array_n_gb300.tsl_array_n import Field
    rng = np.random.default_rng(5)
    u, v, w = field(shape, h, rng, 4)
    vel = ff.FaceCenteredGrid3(shape, h).set(u, v, w)
    col = collider_for(shape, h) if with_collider else None
    adv = ff.create_semi_lagrangian_advection_solver3(velocity_grid=vel, collider=col, dt=0.6)
    p = points(shape, h, rng, -0.15, 1.15)
    p[:3] = [[np.nan, 0.1, 0.1], [np.inf, -np.inf, 0.0], [1e30, -1e30, 1e9]]
    whole, out = Field("vec3", (N,)).from_array(p.ravel()), Field("vec3", (N,))
    part, pout = Field("vec3", (N // 2,)), Field("vec3", (N // 2,))
    for direction in (1, -1):
        adv.trace(whole, out, direction)
        got = out.to_array().reshape(N, 3)
        for half in range(2):
            sl = slice(half * N // 2, (half + 1) * N // 2)
            part.from_array(p[sl].ravel())
            adv.trace(part, pout, direction)
            np.testing.assert_array_equal(got[sl], pout.to_array().reshape(-1, 3))
        ref = oracle.trace(shape, h, (0.0, 0.0, 0.0), u, v, w, col.phi.to_array() if col else None, p[3:100000], 0.6,
                           direction=direction)
        np.testing.assert_array_equal(got[3:100000], np.asarray(ref, np.float32).reshape(-1, 3))


@pytest.mark.parametrize("h", [(0.125,) * 3, (0.1, 0.12, 0.1)])
def test_flip_advection_of_many_particles(gpu, h):
    from tsl_array_n_gb300 import fluxflow as ff
    shape = (40, 24, 18)
    rng = np.random.default_rng(6)
    u, v, w = field(shape, h, rng, 4)
    p = points(shape, h, rng, 0.0, 1.0)
    col = collider_for(shape, h)
    got = []
    for count in (N, N // 2):
        s = ff.create_grid_flip_solver3(velocity_grid=ff.FaceCenteredGrid3(shape, h).set(u, v, w), max_particles=count,
                                        dt=0.4, collider=col, collider_push_thresh=0.02, collider_push_shift=0.01)
        parts = []
        for at in range(0, N, count):
            s.positions.from_array(p[at:at + count].ravel())
            s.stage("advectParticles")
            parts.append(s.positions.to_array().copy())
        got.append(np.concatenate(parts))
    np.testing.assert_array_equal(got[0], got[1])
