"""The in-place layered extension: the velocity constraint over its face
lists against the FP32 oracle, and the FLIP extension against Jacobi steps in
numpy, bit for bit, at extents that are not multiples of the four faces a
thread takes and at depths past the layer bytes' range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = np.asarray(a, np.float32).ravel(), np.asarray(b, np.float32).ravel()
    assert a.shape == b.shape
    bad = ~((a == b) | (np.isnan(a) & np.isnan(b)))
    assert not bad.any(), f"{bad.sum()} of {a.size} differ"


def jacobi(d, valid, depth):
    """createExtrapolateToRegion3 (array_utils3.js:88-150) on (nz, ny, nx)
    float32 arrays, neighbours in the order +x -x +y -y +z -z."""
    d, valid = d.copy(), valid.copy()
    for _ in range(depth):
        tot, cnt = np.zeros_like(d), np.zeros(d.shape, np.float32)
        for ax in (2, 1, 0):
            for by in (1, -1):
                n = d.shape[ax]
                to = [slice(None)] * 3
                fr = [slice(None)] * 3
                to[ax], fr[ax] = (slice(0, n - 1), slice(1, n)) if by == 1 else (slice(1, n), slice(0, n - 1))
                v = valid[tuple(fr)]
                tot[tuple(to)] = np.where(v, tot[tuple(to)] + d[tuple(fr)], tot[tuple(to)])
                cnt[tuple(to)] += v
        new = ~valid & (cnt > 0)
        d = np.where(new, tot / np.maximum(cnt, np.float32(1)), d).astype(np.float32)
        valid |= new
    return d


@pytest.mark.parametrize("weights", [False, True])
@pytest.mark.parametrize("shape,depth", [((1, 1, 1), 5), ((2, 3, 1), 1), ((5, 4, 7), 5), ((33, 18, 9), 0),
                                         ((31, 6, 5), 3), ((600, 2, 2), 300), ((66, 35, 12), 5)])
def test_constrain_lists(gpu, oracle, shape, depth, weights):
    from tsl_array_n_gb300 import fluxflow as ff
    rng = np.random.default_rng(3)
    h, o = (0.1,) * 3, (0.0,) * 3
    faces = [np.float32(40) * rng.standard_normal(int(np.prod([shape[b] + (a == b) for b in range(3)]))).astype(np.float32)
             for a in range(3)]
    faces[0][0] = np.inf
    col = ff.create_sdf_static_collider3(*shape, *h)
    mid = [0.05 * n for n in shape]
    # everything beyond a corner of the domain is solid: several layers deep
    col.add_shapes([{"type": "box", "center": [2 * c for c in mid], "halfExtents": [1.1 * c for c in mid]}])
    fw = col.compute_face_weights() if weights else None
    vel = ff.FaceCenteredGrid3(shape, h, o).set(*faces)
    bc = ff.create_grid_blocked_boundary_condition_solver3(vel, *shape, *h, collider=col, collider_face_weights=fw)
    bc.closed_domain_boundary_flag = 63 & ~8
    bc.constrain_velocity(depth)
    ref = oracle.constrain_velocity(shape, h, o, *faces, phi=col.phi.to_array(), depth=depth, closed=63 & ~8,
                                    face_weights=tuple(fw[k].to_array() for k in "uvw") if weights else None)
    for g, r in zip(vel.get(), ref):
        same(g, r)


@pytest.mark.parametrize("shape,depth", [((5, 4, 3), 1), ((16, 9, 7), 5), ((37, 21, 6), 0), ((330, 3, 2), 320)])
def test_flip_extension(gpu, shape, depth):
    from tsl_array_n_gb300 import fluxflow as ff
    rng = np.random.default_rng(5)
    h = (0.25,) * 3
    n = 40
    grid = ff.FaceCenteredGrid3(shape, h)
    s = ff.create_grid_flip_solver3(velocity_grid=grid, max_particles=n, dt=0.01, extrapolation_depth=depth)
    # a few particles near one end: one component of most faces stays invalid
    pos = (rng.random((n, 3)) * [0.2 * shape[0], 0.25 * shape[1], 0.25 * shape[2]]).astype(np.float32)
    s.positions.from_array(pos.ravel())
    s.velocities.from_array(rng.standard_normal(3 * n).astype(np.float32))
    s.stage("p2g")
    before = [f.to_numpy() for f in (grid.data_u, grid.data_v, grid.data_w)]
    # a face is valid where its weight sum (in 1/65536ths) exceeds 1e-4
    valid = []
    for a, f in enumerate(before):
        cnt = np.zeros(f.size, np.int64)
        g = [(pos[:, b] - np.float32(0.0 if a == b else 0.125)) / np.float32(0.25) for b in range(3)]
        lo = [np.floor(x).astype(int) for x in g]
        fr = [(x - l.astype(np.float32)) for x, l in zip(g, lo)]
        for c in range(8):
            w, idx = None, []
            for b in range(3):
                wb = fr[b] if c >> b & 1 else np.float32(1) - fr[b]
                w = wb if w is None else w * wb
                idx.append(np.clip(lo[b] + (c >> b & 1), 0, f.shape[2 - b] - 1))
            np.add.at(cnt, idx[0] + f.shape[2] * (idx[1] + f.shape[1] * idx[2]), np.rint(w * np.float32(65536)).astype(np.int64))
        valid.append(((cnt.astype(np.float32) / np.float32(65536)) > np.float32(1e-4)).reshape(f.shape))
    s.stage("extrapolateWeight")
    for f, b, v in zip((grid.data_u, grid.data_v, grid.data_w), before, valid):
        same(f.to_numpy(), jacobi(b, v, depth))
