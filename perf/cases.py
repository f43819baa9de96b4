"""The work a fluid simulation has this framework do, as cases that can be timed.

Every case runs through the public Python API (fluxflow.py, warmstart.py):
pressure projections in 3D and 2D, the grid-solver step, advection, the
velocity constraint, the FLIP transfers and step, and the warm-start network's
forward pass and training step.  Inputs are synthetic, made on the GPU from a
seed: separable Fourier velocities, a spherical obstacle, wavy free surfaces,
jittered particles in a partly mixed order.

``exact`` restates a case in plain torch, in 64 bits.
"""
import math

import numpy as np
import torch

from tsl_array_n_gb300 import fluxflow as ff
from tsl_array_n_gb300.tsl_array_n import Field, init
from tsl_array_n_gb300.warmstart import UNetWarmStart

DEV = "cuda"
WEIGHTS = "tsl_array_n_gb300/weights/unet_warmstart.npy"      # the trained network of this repository


def listed():
    return [
        # the headline benchmark's projection: a 256^3 MAC grid around a sphere
        # of radius 24 cells, mixed precision to 1e-6, closed walls and one
        # pinned cell, as one frame of an offline smoke simulation has it
        dict(name="project_sphere_256", kind="project", nx=256, ny=256, nz=256, levels=6, coarse="direct",
             scene="sphere", precision="mixed", tol=1e-6),
        # an interactive-sized grid (the resolution of the reference's stored
        # frames) in the default single precision: launches and latency
        dict(name="project_small_48", kind="project", nx=48, ny=24, nz=24, levels=3, coarse="sweeps", scene="sphere",
             precision="fp32", tol=1e-4),
        # a grid fitted to a scene rather than to a power of two: odd coarse
        # extents, rows not a multiple of four cells, two levels only
        dict(name="project_ragged_90", kind="project", nx=90, ny=54, nz=66, levels=2, coarse="sweeps", scene="sphere",
             precision="mixed", tol=1e-6),
        # a variable-density projection at 1000:1 (liquid under gas) on the
        # dam break's grid, open at the top
        dict(name="project_two_phase_256", kind="project", nx=256, ny=128, nz=128, levels=5, coarse="sweeps",
             scene="two_phase", precision="mixed", tol=1e-6),
        # the 2D cylinder flow's projection: a small 2D solve, many iterations
        dict(name="project_2d_128", kind="project", nx=128, ny=128, nz=1, levels=4, coarse="sweeps", scene="sphere",
             precision="mixed", tol=1e-6),
        # one whole step of the Karman channel (viscosity, projection,
        # constraint, advection), the 2D solver as a user drives it
        dict(name="step_channel_1024", kind="step", nx=1024, ny=256, nz=1, levels=5),
        # advection of the three face components at the benchmark's size
        dict(name="advect_256", kind="advect", nx=256, ny=256, nz=256, order=1),
        # the velocity constraint around an obstacle at the benchmark's size
        dict(name="constrain_256", kind="constrain", nx=256, ny=256, nz=256),
        # particle-grid transfers of the dam break: particles to grid, valid
        # faces extended, grid to particles
        dict(name="transfer_256", kind="transfer", nx=256, ny=128, nz=128, fill=0.4),
        # one whole step of the FLIP dam break (13M particles), resampling and
        # the free-surface projection included
        dict(name="flip_step_256", kind="flip_step", nx=256, ny=128, nz=128, fill=0.4),
        # the warm-start network: a guess for one 256^3 frame, and a training
        # step at the size it is trained at
        dict(name="unet_forward_256", kind="unet", nx=256, ny=256, nz=256, train=False),
        dict(name="unet_train_128", kind="unet", nx=128, ny=128, nz=128, train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["project", "project", "project", "project", "step", "advect", "constrain", "transfer",
                       "flip_step", "unet"])
    if kind == "project":
        scene = rng.choice(["sphere", "sphere", "two_phase", "2d"])
        size = [_log_int(rng, 64, 768) for _ in range(2)] if scene == "2d" else [_log_int(rng, 24, 128 if scene == "two_phase" else 224) for _ in range(3)]
        levels = max(2, min(6, int(math.log2(min(size) / 5)) + rng.randint(0, 1)))
        q = 1 << (levels - 1)
        nx, ny, nz = ([q * max(2, a // q) for a in size] + [1])[:3]
        coarse = "direct" if (nx // q) * (ny // q) * max(1, nz // q) <= 1024 and rng.random() < 0.5 else "sweeps"
        return dict(kind="project", nx=nx, ny=ny, nz=nz, levels=levels, coarse=coarse,
                    scene="sphere" if scene == "2d" else scene, precision="mixed", tol=1e-6)
    if kind == "step":
        q = 16
        return dict(kind="step", nx=q * max(6, _log_int(rng, 96, 1024) // q), ny=q * max(5, _log_int(rng, 80, 256) // q),
                    nz=1, levels=rng.randint(3, 5))
    if kind in ("advect", "constrain"):
        nx, ny, nz = (_log_int(rng, 20, 256) for _ in range(3))
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
        if kind == "advect":
            c["order"] = rng.choice([1, 1, 2])
        return c
    if kind in ("transfer", "flip_step"):
        nx, ny, nz = (16 * max(2, _log_int(rng, 32, b) // 16) for b in (256, 128, 128))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, fill=rng.uniform(0.25, 0.4))
    train = rng.random() < 0.5
    nx, ny, nz = (4 * _log_int(rng, 8, 32 if train else 64) for _ in range(3))
    return dict(kind="unet", nx=nx, ny=ny, nz=nz, train=train)


# ------------------------------------------------------------------ inputs --
class _Raw:
    """A library field's memory for torch (no copy); keeps its owner alive."""

    def __init__(self, field, shape, owner):
        self.keep = (field, owner)
        kinds = {"float": "<f4", "int": "<i4", "uint8": "|u1", "vec3": "<f4"}
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=kinds[field.type], version=3, strides=None,
                                             data=(field.device_ptr(), False))


def _view(field, owner=None):
    shape = tuple(reversed(field.shape)) + ((3,) if field.type == "vec3" else ())
    return torch.as_tensor(_Raw(field, shape, owner), device=DEV)


def _field(values, kind="float"):
    """A field (shape reversed: x fastest) holding a torch array."""
    shape = tuple(reversed(values.shape))
    if kind == "vec3":
        shape = (values.shape[0],)
    f = Field(kind, shape)
    _view(f).copy_(values)
    return f


def _h(case):
    return 1.0 / case["ny"] if case["nz"] > 1 or case["kind"] == "step" else 1.0 / max(case["nx"], case["ny"])


def _axis(n, off, h):
    return (torch.arange(n, dtype=torch.float64, device=DEV) + off) * h


def _fourier(case, gen, modes, amplitude):
    """Three float32 face components, each a sum of separable modes."""
    n, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    out = []
    for a in range(3):
        shp = [n[b] + (a == b) for b in range(3)]
        tot = torch.zeros(shp[2], shp[1], shp[0], device=DEV)
        for _ in range(modes):
            amp = torch.randn(1, generator=gen).item() * amplitude
            k = torch.randint(1, 5, (3,), generator=gen).tolist()
            ph = (torch.rand(3, generator=gen) * 2 * math.pi).tolist()
            f = [torch.sin(2 * math.pi * k[b] * _axis(shp[b], 0.0 if a == b else 0.5, h) + ph[b]).float()
                 for b in range(3)]
            if n[2] == 1:
                f[2] = torch.ones_like(f[2])
            tot += amp * (f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :])
        out.append(tot)
    return out


def _close_walls(vel, skip=()):
    for a, f in enumerate(vel):
        if a not in skip:
            f.select(2 - a, 0).zero_()
            f.select(2 - a, f.shape[2 - a] - 1).zero_()
    return vel


def _sphere(case, gen):
    """Signed distance (float32, cell centres) of a sphere (a disc in 2D) off
    the middle by a few cells, and the open fractions of the faces."""
    n, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    two = n[2] == 1
    r = 0.094 * min(n[0], n[1], *(() if two else (n[2],))) * h
    off = ((torch.rand(3, generator=gen) - 0.5) * 0.1).tolist()
    cen = [n[a] * h * ((0.3 if a == 0 else 0.5) + off[a]) for a in range(3)]

    def dist(shp, offs):
        d2 = 0.0
        for b in range(2 if two else 3):
            x = _axis(shp[b], offs[b], h) - cen[b]
            d2 = d2 + (x * x).reshape([-1 if 2 - b == q else 1 for q in range(3)])
        return (d2.sqrt() - r).expand(shp[2], shp[1], shp[0])

    phi = dist(n, (0.5, 0.5, 0.5)).float().contiguous()
    ws = []
    for a in range(3):
        shp = [n[b] + (a == b) for b in range(3)]
        w = (0.5 + dist(shp, [0.0 if a == b else 0.5 for b in range(3)]) / h).clamp(0.0, 1.0)
        ws.append(torch.where(w < 0.01, torch.zeros_like(w), w).float().contiguous())
    return phi, ws


def _surface(case, gen, mean, amp):
    """Height of a wavy surface over (z, x), in units of the domain height."""
    n, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    y = torch.full((n[2], n[0]), mean, dtype=torch.float64, device=DEV)
    for _ in range(6):
        k, ph = torch.randint(1, 6, (2,), generator=gen).tolist(), (torch.rand(2, generator=gen) * 6.28).tolist()
        y = y + amp * torch.randn(1, generator=gen).item() * (
            torch.sin(2 * k[1] * _axis(n[2], 0.5, h) + ph[1])[:, None] * torch.sin(2 * k[0] * _axis(n[0], 0.5, h) + ph[0])[None, :])
    return y.clamp(0.05, 0.95)


def _project_inputs(case, seed):
    gen = torch.Generator().manual_seed(seed)
    n = (case["nx"], case["ny"], case["nz"])
    vel = _fourier(case, gen, 16, 0.3)
    active = torch.zeros(n[2], n[1], n[0], dtype=torch.uint8, device=DEV)
    cw = beta = None
    if case["scene"] == "two_phase":
        _close_walls(vel)
        top = _surface(case, gen, 0.5, 0.05)[:, None, :] * n[1]
        frac = (top - torch.arange(n[1], dtype=torch.float64, device=DEV)[None, :, None]).clamp(0.0, 1.0)
        frac = (frac * 8).round() / 8          # eight particles a cell
        rho = (0.001 + 0.999 * frac).float()
        beta = []
        for a in range(3):
            lo = torch.cat([rho.narrow(2 - a, 0, 1), rho], 2 - a)
            hi = torch.cat([rho, rho.narrow(2 - a, n[a] - 1, 1)], 2 - a)
            beta.append((1.0 / ((lo + hi) * 0.5)).contiguous())
        active[:, n[1] - 1, :] = 1
    else:
        if n[2] == 1:
            vel[0] += 1.0
            vel[2].zero_()
            _close_walls(vel, skip=(0, 2))
            vel[0][:, :, 0] = 1.0
        else:
            _close_walls(vel)
        if n[2] == 1:
            active[:, :, n[0] - 1] = 1             # an outflow column
        else:
            active[0, 0, 0] = 1                    # closed walls and one pinned cell
        cw = _sphere(case, gen)[1]
    return vel, active, cw, beta


def _channel_inputs(case, seed):
    gen = torch.Generator().manual_seed(seed)
    phi, cw = _sphere(case, gen)
    vel = _fourier(case, gen, 8, 0.05)
    vel[0] += 1.0
    vel[2].zero_()
    active = torch.zeros(1, case["ny"], case["nx"], dtype=torch.uint8, device=DEV)
    active[:, :, -1] = 1
    h = _h(case)
    dt = 0.5 * h
    nu = 2 * 0.094 * min(case["nx"], case["ny"]) * h / 200.0      # Re 200 on the diameter
    # the inflow: a layer one and a half cells thick along the left wall
    inflow = ((_axis(case["nx"], 0.5, h) - 1.5 * h).float()).expand(1, case["ny"], -1).contiguous()
    return vel, phi, cw, active, inflow, dt, nu


def _grid_inputs(case, seed):
    gen = torch.Generator().manual_seed(seed)
    phi, cw = _sphere(case, gen)
    return _fourier(case, gen, 32, 1.0), phi, cw


def _particles(case, seed):
    """Particles below a wavy surface, eight a cell, jittered; an eighth of
    them moved within the liquid's list and one in fifty thrown up as spray,
    as some hundred steps leave them; velocities from smooth modes.  Also the
    faces of the same velocity."""
    gen = torch.Generator().manual_seed(seed)
    n, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    top = _surface(case, gen, case["fill"], 0.03) * n[1]                              # over (z, x), in cells
    depth = (torch.arange(n[1], device=DEV)[None, :, None] - top[:, None, :]).float().reshape(-1)
    cell = depth.argsort(stable=True)[: int(n[0] * n[1] * n[2] * case["fill"])].sort()[0]
    g = torch.Generator(device=DEV).manual_seed(seed)
    ijk = torch.stack([cell % n[0], (cell // n[0]) % n[1], cell // (n[0] * n[1])], 1).float()
    sub = torch.tensor([[(s >> b & 1) * 0.5 + 0.25 for b in range(3)] for s in range(8)], device=DEV)
    pos = (ijk[:, None, :] + sub[None]).reshape(-1, 3)
    pos = pos + (torch.rand(pos.shape, generator=g, device=DEV) - 0.5) * 0.2
    m = pos.shape[0]
    moved = torch.randperm(m, generator=g, device=DEV)[: m // 8]
    pos[moved] = pos[moved[torch.randperm(moved.numel(), generator=g, device=DEV)]]
    spray = torch.randperm(m, generator=g, device=DEV)[: m // 50]
    pos[spray, 1] = (pos[spray, 1] + torch.rand(spray.numel(), generator=g, device=DEV) * 0.2 * n[1]).clamp(max=n[1] - 0.5)
    pos = (pos * h).contiguous()
    vel, faces = torch.zeros_like(pos), _fourier(case, gen, 3, 0.5)
    for a in range(3):
        for _ in range(3):
            amp, k = torch.randn(1, generator=gen).item() * 0.5, torch.randint(1, 4, (3,), generator=gen).tolist()
            vel[:, a] += amp * (torch.sin(3 * k[0] * pos[:, 0]) * torch.cos(3 * k[1] * pos[:, 1]) * torch.sin(3 * k[2] * pos[:, 2] + 1))
    return pos, vel, _close_walls(faces)


def _unet_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    shp = (case["nz"], case["ny"], case["nx"])
    b = torch.randn(shp, generator=gen, device=DEV)
    mask = (torch.rand(shp, generator=gen, device=DEV) < 0.05).to(torch.uint8)
    prev = torch.randn(shp, generator=gen, device=DEV) * 1e-3
    target = prev + torch.randn(shp, generator=gen, device=DEV) * 3e-4
    return b, mask, prev, target


def _grid3(case, vel, h):
    g = ff.FaceCenteredGrid3((case["nx"], case["ny"], case["nz"]), (h, h, h))
    for f, v in zip((g.data_u, g.data_v, g.data_w), vel):
        _view(f).copy_(v)
    return g


def _faces(grid, owner, count=3):
    return {k: _view(f, owner) for k, f in list(zip("uvw", (grid.data_u, grid.data_v, grid.data_w)))[:count]}


def _uvw(arrays):
    return dict(zip("uvw", (_field(a) for a in arrays)))


def _collider(case, phi, h):
    c = ff.create_sdf_static_collider3(case["nx"], case["ny"], case["nz"], h, h, h)
    _view(c.phi).copy_(phi)
    return c


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    init(0)
    s = {"kind": case["kind"]}
    res, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    if case["kind"] == "project":
        vel, active, cw, beta = _project_inputs(case, seed)
        make = ff.create_grid_pressure_solver2 if res[2] == 1 else ff.create_grid_pressure_solver3
        dims = 2 if res[2] == 1 else 3
        s["solver"] = make(res[:dims], (h,) * dims, collider_weights=_uvw(cw) if cw else None,
                           face_weights=_uvw(beta) if beta else None,
                           dirichlet=(active.reshape(-1).cpu().numpy(), np.zeros(active.numel(), np.float32)),
                           multigrid={"numberOfLevels": case["levels"], "coarseSolve": case["coarse"]},
                           precision=case["precision"], tolerance=case["tol"], max_iterations=400)
        s["grid"], s["out"] = _grid3(case, vel, h), ff.FaceCenteredGrid3(res, (h, h, h))
        s["project"] = s["solver"].project(s["grid"], s["out"])
        s["result"] = {**_faces(s["out"], None, dims), "pressure": _view(s["solver"].pressure, s["solver"])}
    elif case["kind"] == "step":
        vel, phi, cw, active, inflow, dt, nu = _channel_inputs(case, seed)
        s["grid"], s["start"] = _grid3(case, vel, h), _grid3(case, vel, h)
        jet = ff.create_sdf_inflow3(*res, h, h, h, velocity=(1.0, 0.0, 0.0), mode="set")
        _view(jet.phi).copy_(inflow)
        s["solver"] = ff.create_grid_solver3(
            velocity_grid=s["grid"], collider=_collider(case, phi, h), inflows=[jet], dt=dt, nu=nu,
            closed_domain_boundary_flag=ff.DIRECTION_DOWN | ff.DIRECTION_UP | ff.DIRECTION_BACK | ff.DIRECTION_FRONT,
            dirichlet=(active.reshape(-1).cpu().numpy(), np.zeros(active.numel(), np.float32)),
            pressure={"multigrid": {"numberOfLevels": case["levels"]}, "precision": "mixed", "tolerance": 1e-6,
                      "collider_weights": _uvw(cw), "max_iterations": 400})
        s["result"] = {**_faces(s["grid"], s["solver"], 2),
                       "pressure": _view(s["solver"].pressure, s["solver"].pressure_solver)}
    elif case["kind"] == "advect":
        vel, phi, _ = _grid_inputs(case, seed)
        s["grid"], s["out"] = _grid3(case, vel, h), ff.FaceCenteredGrid3(res, (h, h, h))
        s["solver"] = ff.create_semi_lagrangian_advection_solver3(s["grid"], _collider(case, phi, h), 0.25 * h,
                                                                  order=case["order"])
        s["advect"] = s["solver"].advect_face_centered3(s["grid"], s["out"])
        s["result"] = _faces(s["out"], None)
    elif case["kind"] == "constrain":
        vel, phi, cw = _grid_inputs(case, seed)
        s["grid"], s["start"] = _grid3(case, vel, h), _grid3(case, vel, h)
        s["solver"] = ff.create_grid_blocked_boundary_condition_solver3(
            s["grid"], *res, h, h, h, collider=_collider(case, phi, h), collider_face_weights=_uvw(cw))
        s["result"] = _faces(s["grid"], None)
    elif case["kind"] in ("transfer", "flip_step"):
        pos, vel, faces = _particles(case, seed)
        s["grid"] = _grid3(case, faces, h)
        q = 1
        while q < 16 and all(a % (2 * q) == 0 and a // (2 * q) >= 4 for a in res):
            q *= 2
        s["solver"] = ff.create_grid_flip_solver3(
            velocity_grid=s["grid"], max_particles=pos.shape[0], dt=0.25 * h, flip_ratio=0.95,
            pressure={"multigrid": {"numberOfLevels": int(math.log2(q)) + 1, "coarseSolve": "sweeps"},
                      "tolerance": 1e-6, "precision": "mixed", "maxPlausiblePressure": 1e6})
        sv = s["solver"]
        _view(sv.positions, sv).copy_(pos)
        _view(sv.velocities, sv).copy_(vel)
        s["result"] = {**_faces(s["grid"], sv), "positions": _view(sv.positions, sv),
                       "velocities": _view(sv.velocities, sv)}
        if case["kind"] == "flip_step":
            s["start"] = _grid3(case, faces, h)
            s["start_pos"], s["start_vel"] = _field(pos, "vec3"), _field(vel, "vec3")
        else:
            del s["result"]["positions"]          # the transfers leave them alone
    else:
        b, mask, prev, target = _unet_inputs(case, seed)
        s["net"] = UNetWarmStart(seed=1)
        s["net"].load(WEIGHTS)
        s["args"] = (res, h, _field(b), _field(mask, "uint8"), _field(prev))
        s["target"] = _field(target) if case["train"] else None
        s["out"] = Field("float", res)
        s["result"] = {"guess": _view(s["out"])}
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run --
def _restore(s):
    """A frame's state again, on the device (a pass works in place)."""
    g, o = s["grid"], s["start"]
    g.data_u.copy_from(o.data_u)
    g.data_v.copy_from(o.data_v)
    g.data_w.copy_from(o.data_w)


def run(s):
    kind = s["kind"]
    if kind == "project":
        s["solver"].pressure.fill(0.0)            # a cold start, as a first frame has
        s["project"]()
    elif kind == "step":
        _restore(s)
        s["solver"].pressure.fill(0.0)
        s["solver"].on_advance_time_step()
    elif kind == "advect":
        s["advect"]()
    elif kind == "constrain":
        _restore(s)
        s["solver"].constrain_velocity()
    elif kind == "transfer":
        for stage in ("p2g", "snapshotOld", "extrapolateWeight", "g2p"):
            s["solver"].stage(stage)
    elif kind == "flip_step":
        _restore(s)
        s["solver"].positions.copy_from(s["start_pos"])
        s["solver"].velocities.copy_from(s["start_vel"])
        s["solver"].pressure.fill(0.0)
        s["solver"].on_advance_time_step()
    elif s["target"] is None:
        s["net"].forward(*s["args"], s["out"])
    else:
        loss = s["net"].loss_backward(*s["args"], s["target"])
        grads = s["net"].grads                    # read by the training loop
        s["net"].adam_step(1e-4)
        return {"loss": loss, "grads": grads}
    return s["result"]


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    dims = 2 if case["nz"] == 1 else 3
    kind = case["kind"]
    if kind == "project":      # faces and their weights in, faces and pressure out
        return {"bytes": n * (12 * dims + 5), "flops": n * 40}
    if kind == "step":
        return {"bytes": n * (12 * dims + 9), "flops": n * 400}
    if kind == "advect":       # three components, each read once and written once
        return {"bytes": n * (8 * dims + 4), "flops": n * 3 * 800 * case["order"]}
    if kind == "constrain":    # face values and weights in, values out, the distance in
        return {"bytes": n * (12 * dims + 4), "flops": n * 10}
    if kind in ("transfer", "flip_step"):
        p = 8 * n * case["fill"]
        return {"bytes": p * (36 if kind == "transfer" else 48) + n * 24, "flops": p * 500}
    flops = 2 * 27 * n * ((3 * 16 + 16 * 16 + 48 * 16 + 16 * 16) + (16 * 32 + 32 * 32 + 96 * 32 + 32 * 32) / 8
                          + (32 * 64 + 64 * 64) / 64)
    return {"bytes": n * 13, "flops": flops * (3 if case["train"] else 1)}


# ------------------------------------------------------------------- exact --
def _shift(x, axis, by):
    """x moved along an axis (0 = x), zeros past the ends: y[i] = x[i + by]."""
    d, n = 2 - axis, x.shape[2 - axis]
    y = torch.zeros_like(x)
    if by > 0:
        y.narrow(d, 0, n - by).copy_(x.narrow(d, by, n - by))
    else:
        y.narrow(d, -by, n + by).copy_(x.narrow(d, 0, n + by))
    return y


def _solve_poisson(h, b, mask, w):
    """Cells with sum_faces w (p_nb - p) / h^2 = b and p = 0 on the mask, by
    conjugate gradients with the diagonal, to 1e-11 of b."""
    dims = 2 if b.shape[0] == 1 else 3
    free = ~mask
    k = []
    for a in range(dims):
        n = b.shape[2 - a]
        low = w[a].narrow(2 - a, 0, n).clone() if w is not None else torch.ones_like(b)
        low.narrow(2 - a, 0, 1).zero_()
        k.append(low / (h * h))
    diag = sum(q + _shift(q, a, 1) for a, q in enumerate(k))
    inv = torch.where(free & (diag > 0), 1.0 / diag, torch.zeros_like(diag))
    pair = [k[a] * free * _shift(free.double(), a, -1) for a in range(dims)]   # couplings between free cells

    def apply(p):
        y = diag * p
        for a in range(dims):
            d, n = 2 - a, p.shape[2 - a]
            lo, hi, c = p.narrow(d, 0, n - 1), p.narrow(d, 1, n - 1), pair[a].narrow(d, 1, n - 1)
            y.narrow(d, 1, n - 1).addcmul_(c, lo, value=-1.0)
            y.narrow(d, 0, n - 1).addcmul_(c, hi, value=-1.0)
        return y

    r = torch.where(free, -b, torch.zeros_like(b))
    x, z = torch.zeros_like(r), r * inv
    p, rz = z.clone(), (r * z).sum()
    stop = 1e-22 * (r * r).sum().item()
    for it in range(20000):
        q = apply(p)
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if it % 16 == 0 and (r * r).sum().item() <= stop:
            break
        z = r * inv
        new = (r * z).sum()
        p.mul_(new / rz).add_(z)
        rz = new
    return x


def _exact_project(h, vel, active, cw, beta):
    dims = 2 if active.shape[0] == 1 else 3
    vel = [v.double() for v in vel]
    c64 = [w.double() for w in cw] if cw is not None else None
    mask = active.bool()
    if c64 is not None:
        mask = mask | (sum(c64[a].narrow(2 - a, 0, active.shape[2 - a]) + c64[a].narrow(2 - a, 1, active.shape[2 - a])
                           for a in range(dims)) < 1e-6)
    div = 0.0
    for a in range(dims):
        f, n = (vel[a] * c64[a] if c64 is not None else vel[a]), active.shape[2 - a]
        div = div + (f.narrow(2 - a, 1, n) - f.narrow(2 - a, 0, n)) / h
    w = c64 if c64 is not None else ([q.double() for q in beta] if beta is not None else None)
    p = _solve_poisson(h, div, mask, w)
    out = {}
    for a in range(dims):
        d, n = 2 - a, p.shape[2 - a]
        g = (p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1)) / h
        if beta is not None:
            g = g * beta[a].narrow(d, 1, n - 1).double()
        if c64 is not None:
            g = g * (c64[a].narrow(d, 1, n - 1) > 0)
        f = vel[a].clone()
        f.narrow(d, 1, n - 1).sub_(g)
        out["uvw"[a]] = f
    out["pressure"] = p
    return out


def _off(a):
    return [0.0 if a == b else 0.5 for b in range(3)]


def _taps(x, n, off, h, reach):
    """Grid coordinate, its clamped neighbour indices and the fraction."""
    c = x / h - off
    i = torch.floor(c)
    return [(i.long() + q).clamp(0, n - 1) for q in reach], c - i


def _linear(f, off, h, pts):
    (xi, fx), (yi, fy), (zi, fz) = (_taps(pts[b], f.shape[2 - b], off[b], h, (0, 1)) for b in range(3))
    flat, nx, ny = f.reshape(-1), f.shape[2], f.shape[1]
    s = 0.0
    for c in range(8):
        w = (fx if c & 1 else 1 - fx) * (fy if c & 2 else 1 - fy) * (fz if c & 4 else 1 - fz)
        s = s + w * flat[xi[c & 1] + nx * (yi[c >> 1 & 1] + ny * zi[c >> 2])]
    return s


def _gradient(f, off, h, pts):
    flat, n = f.reshape(-1), (f.shape[2], f.shape[1], f.shape[0])
    lo, hi, t = [], [], []
    for b in range(3):
        c = pts[b] / h - off[b]
        i = torch.floor(c).long().clamp(max=n[b] - 2).clamp(min=0)
        lo.append(i)
        hi.append((i + 1).clamp(max=n[b] - 1))
        t.append((c - i).clamp(0.0, 1.0))
    v = {c: flat[(hi if c & 1 else lo)[0] + n[0] * ((hi if c & 2 else lo)[1] + n[1] * (hi if c & 4 else lo)[2])]
         for c in range(8)}
    g = []
    for b in range(3):
        o = [q for q in range(3) if q != b]
        s = 0.0
        for c in range(8):
            if not c >> b & 1:
                w = 1.0
                for q in o:
                    w = w * (t[q] if c >> q & 1 else 1 - t[q])
                s = s + w * (v[c | 1 << b] - v[c])
        g.append(s / h)
    return g


def _cubic1(f0, f1, f2, f3, t):
    d = f2 - f1
    a, b = (f2 - f0) * 0.5, (f3 - f1) * 0.5
    flat = d.abs() < 1e-12
    a = torch.where(flat | (a * d < 0), torch.zeros_like(a), a)
    b = torch.where(flat | (b * d < 0), torch.zeros_like(b), b)
    return (a + b - 2 * d) * t ** 3 + (3 * d - 2 * a - b) * t ** 2 + a * t + f1


def _cubic(f, off, h, pts):
    (xi, fx), (yi, fy), (zi, fz) = (_taps(pts[b], f.shape[2 - b], off[b], h, (-1, 0, 1, 2)) for b in range(3))
    flat, nx, ny = f.reshape(-1), f.shape[2], f.shape[1]
    zv = []
    for c in range(4):
        rows = []
        for b in range(4):
            base = nx * (yi[b] + ny * zi[c])
            rows.append(_cubic1(*(flat[base + xi[a]] for a in range(4)), fx))
        zv.append(_cubic1(*rows, fy))
    return _cubic1(*zv, fz)


def _trace(vel, phi, h, pts, dt, way):
    """Midpoint substeps of at most a cell, ended on the obstacle."""
    pts = [p.clone() for p in pts]
    left = torch.full_like(pts[0], dt)
    go = left > 1e-6
    for _ in range(32):
        if not bool(go.any()):
            break
        v0 = [_linear(vel[a], _off(a), h, pts) for a in range(3)]
        step = left / torch.ceil(sum(v * v for v in v0).sqrt() * left / h).clamp(min=1.0)
        mid = [p - v * step * 0.5 * way for p, v in zip(pts, v0)]
        nxt = [p - _linear(vel[a], _off(a), h, mid) * step * way for a, p in enumerate(pts)]
        if phi is not None:
            a, b = _linear(phi, _off(3), h, pts), _linear(phi, _off(3), h, nxt)
            hit = b <= 0
            wgt = b.abs() / (a.abs() + b.abs())
            nxt = [torch.where(hit, p * wgt + q * (1 - wgt), q) for p, q in zip(pts, nxt)]
        else:
            hit = torch.zeros_like(go)
        pts = [torch.where(go, q, p) for p, q in zip(pts, nxt)]
        left = torch.where(go, left - step, left)
        go = go & ~hit & (left > 1e-6)
    return pts


def _face_points(shape, a, h, at):
    """Positions of the faces of component a with the flat indices `at`."""
    nx, ny = shape[2], shape[1]
    o = _off(a)
    return [((at % nx).double() + o[0]) * h, ((at // nx % ny).double() + o[1]) * h, ((at // (nx * ny)).double() + o[2]) * h]


def _exact_advect(vel, phi, h, dt, order, out=None):
    vel, phi = [v.double() for v in vel], phi.double()
    res = {}
    for a in range(3):
        f, flat = vel[a], (torch.zeros_like(vel[a]) if out is None else out[a].double().clone())
        fwd, bwd = f.clone(), f.clone()
        chunks = torch.arange(f.numel(), device=DEV).split(1 << 21)
        for at in chunks:
            pts = _face_points(f.shape, a, h, at)
            at, pts = at[_linear(phi, _off(3), h, pts) > 0], None
            pts = _face_points(f.shape, a, h, at)
            fwd.reshape(-1)[at] = _cubic(f, _off(a), h, _trace(vel, phi, h, pts, dt, 1.0))
        if order == 2:
            bwd = fwd.clone()
            for at in chunks:
                at = at[_linear(phi, _off(3), h, _face_points(f.shape, a, h, at)) > 0]
                bwd.reshape(-1)[at] = _cubic(fwd, _off(a), h, _trace(vel, phi, h, _face_points(f.shape, a, h, at), dt, -1.0))
        for at in chunks:
            at = at[_linear(phi, _off(3), h, _face_points(f.shape, a, h, at)) > 0]
            val = fwd.reshape(-1)[at]
            if order == 2:
                cor = val + (f.reshape(-1)[at] - bwd.reshape(-1)[at]) * 0.5
                pts = _trace(vel, phi, h, _face_points(f.shape, a, h, at), dt, 1.0)
                idx = [_taps(pts[b], f.shape[2 - b], _off(a)[b], h, (0, 1))[0] for b in range(3)]
                mn, mx = torch.full_like(val, 1e30), torch.full_like(val, -1e30)
                for c in range(8):
                    n = idx[0][c & 1] + f.shape[2] * (idx[1][c >> 1 & 1] + f.shape[1] * idx[2][c >> 2])
                    ok = _linear(phi, _off(3), h, _face_points(f.shape, a, h, n)) > 0
                    v = f.reshape(-1)[n]
                    mn, mx = torch.where(ok, torch.minimum(mn, v), mn), torch.where(ok, torch.maximum(mx, v), mx)
                val = torch.where((cor >= mn) & (cor <= mx), cor, val)
            flat.reshape(-1)[at] = val
        res["uvw"[a]] = flat
    return res


def _extend(f, valid, depth):
    """Jacobi extension of the valid values by `depth` layers."""
    for _ in range(depth):
        tot, cnt = torch.zeros_like(f), torch.zeros_like(f)
        fv, one = f * valid, valid.double()
        for a in range(3):
            for by in (1, -1):
                tot += _shift(fv, a, by)
                cnt += _shift(one, a, by)
        new = ~valid & (cnt > 0)
        f = torch.where(new, tot / cnt.clamp(min=1.0), f)
        valid = valid | new
    return f


def _exact_constrain(vel, phi, cw, h, closed=63, inflow=None):
    phi, cw = phi.double(), [w.double() for w in cw]
    f = []
    for a in range(3):
        open_ = cw[a] > 0
        f.append(_extend(torch.where(open_, vel[a].double(), torch.zeros_like(cw[a])), open_, 5))
    new = []
    for a in range(3):
        at = (cw[a].reshape(-1) <= 0).nonzero()[:, 0]
        pts = _face_points(f[a].shape, a, h, at)
        v = [_linear(f[b], _off(b), h, pts) for b in range(3)]
        g = _gradient(phi, _off(3), h, pts)
        gl = sum(q * q for q in g).sqrt()
        nn = [q / gl.clamp(min=1e-300) for q in g]
        vn = sum(p * q for p, q in zip(v, nn))
        vt = [p - q * vn for p, q in zip(v, nn)]
        tl = sum(q * q for q in vt).sqrt()
        sc = torch.where(tl > 0, (1 - (-vn).clamp(min=0) * 0.5 / tl.clamp(min=1e-300)).clamp(min=0), torch.ones_like(tl))
        o = f[a].clone()
        o.reshape(-1)[at] = torch.where(gl > 0, vt[a] * sc, torch.zeros_like(tl))
        new.append(o)
    solid = phi < 0
    for a in range(3):
        d, n = 2 - a, phi.shape[2 - a]
        edge = solid.narrow(d, 0, n - 1) ^ solid.narrow(d, 1, n - 1)
        inner = new[a].narrow(d, 1, n - 1)
        inner.masked_fill_(edge, 0.0)
        if closed >> (2 * a) & 1:
            new[a].select(d, 0).zero_()
        if closed >> (2 * a + 1) & 1:
            new[a].select(d, n).zero_()
        if inflow is not None:
            at = torch.arange(new[a].numel(), device=DEV)
            inside = _linear(inflow[0].double(), _off(3), h, _face_points(new[a].shape, a, h, at)) < 0
            new[a].reshape(-1)[inside] = inflow[1][a]
        new[a].clamp_(-100.0, 100.0)
    return new


def _exact_step(case, seed):
    vel, phi, cw, active, inflow, dt, nu = _channel_inputs(case, seed)
    h = _h(case)
    closed = ff.DIRECTION_DOWN | ff.DIRECTION_UP | ff.DIRECTION_BACK | ff.DIRECTION_FRONT
    jet = (inflow, (1.0, 0.0, 0.0))
    vis = []
    for a in range(3):
        f = vel[a].double()
        lap = torch.zeros_like(f)
        for b in range(3):
            d, n = 2 - b, f.shape[2 - b]
            up = torch.cat([f.narrow(d, 1, n - 1), f.narrow(d, n - 1, 1)], d)
            dn = torch.cat([f.narrow(d, 0, 1), f.narrow(d, 0, n - 1)], d)
            lap += (up + dn - 2 * f) / (h * h)
        o = f + dt * nu * lap
        for e in (0, f.shape[2 - a] - 1):
            o.select(2 - a, e).copy_(f.select(2 - a, e))
        vis.append(o)
    pr = _exact_project(h, vis, active, cw, None)
    con = _exact_constrain([pr["u"], pr["v"], vis[2]], phi, cw, h, closed, jet)
    adv = _exact_advect(con, phi, h, dt, 1, out=con)
    fin = _exact_constrain([adv["u"], adv["v"], adv["w"]], phi, cw, h, closed, jet)
    return {"u": fin[0], "v": fin[1], "pressure": pr["pressure"]}


def _exact_transfer(case, seed):
    pos, vel, faces = _particles(case, seed)
    h = _h(case)
    pts, out = [pos[:, b].double() for b in range(3)], {}
    new = torch.zeros(pos.shape, dtype=torch.float64, device=DEV)
    for a in range(3):
        f = faces[a]
        t = [_taps(pts[b], f.shape[2 - b], _off(a)[b], h, (0, 1)) for b in range(3)]
        num, den = (torch.zeros(f.numel(), dtype=torch.float64, device=DEV) for _ in range(2))
        for c in range(8):
            w = 1.0
            for b in range(3):
                w = w * (t[b][1] if c >> b & 1 else 1 - t[b][1])
            at = t[0][0][c & 1] + f.shape[2] * (t[1][0][c >> 1 & 1] + f.shape[1] * t[2][0][c >> 2])
            den.index_add_(0, at, w)
            num.index_add_(0, at, w * vel[:, a].double())
        ok = (den > 1e-4).reshape(f.shape)
        old = torch.where(ok, (num / den.clamp(min=1e-30)).reshape(f.shape), torch.zeros(f.shape, dtype=torch.float64, device=DEV))
        ext = _extend(old, ok, 5)
        nv = _linear(ext, _off(a), h, pts)
        fl = vel[:, a].double() + nv - _linear(old, _off(a), h, pts)
        new[:, a] = (fl * 0.95 + nv * 0.05) * 0.98
        out["uvw"[a]] = ext
    out["velocities"] = new
    return out


_CONVS = [(3, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16)]


def _conv(x, w, b):
    """3x3x3 convolution, channels last, as 27 products."""
    z, y, xx, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    out = b.expand(z * y * xx, -1).clone()
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        out = out + p[dz:dz + z, dy:dy + y, dx:dx + xx].reshape(z * y * xx, -1) @ w[t]
    return torch.nn.functional.gelu(out, approximate="tanh").reshape(z, y, xx, -1)


def _exact_unet(case, seed):
    b, mask, prev, target = (t.double() for t in _unet_inputs(case, seed))
    par = torch.from_numpy(np.load(WEIGHTS)).to(DEV).double().requires_grad_(case["train"])
    sb, sp = (b * b).mean().sqrt(), (prev * prev).mean().sqrt()
    pool = lambda x: torch.nn.functional.avg_pool3d(x.permute(3, 0, 1, 2)[None], 2)[0].permute(1, 2, 3, 0)
    up = lambda x: x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
    off, ws = 0, []
    for ci, co in _CONVS:
        ws.append((par[off:off + 27 * ci * co].reshape(27, ci, co), par[off + 27 * ci * co:off + 27 * ci * co + co]))
        off += 27 * ci * co + co
    with torch.set_grad_enabled(case["train"]):
        e0 = _conv(_conv(torch.stack([b / sb, mask, prev / sp], -1), *ws[0]), *ws[1])
        e1 = _conv(_conv(pool(e0), *ws[2]), *ws[3])
        bt = _conv(_conv(pool(e1), *ws[4]), *ws[5])
        d1 = _conv(_conv(torch.cat([up(bt), e1], -1), *ws[6]), *ws[7])
        d0 = _conv(_conv(torch.cat([up(d1), e0], -1), *ws[8]), *ws[9])
        raw = d0 @ par[off:off + 16] + par[off + 16]
        if not case["train"]:
            return {"guess": raw * sp}
        d = raw - target / sp
        p = torch.nn.functional.pad(d[None, None], (1,) * 6, mode="replicate")[0, 0]
        c = p[1:-1, 1:-1, 1:-1]
        lap = (p[1:-1, 1:-1, :-2] + p[1:-1, 1:-1, 2:] + p[1:-1, :-2, 1:-1] + p[1:-1, 2:, 1:-1] + p[:-2, 1:-1, 1:-1]
               + p[2:, 1:-1, 1:-1] - 6 * c)
        loss = (d * d).mean() + 0.25 * (lap * lap).mean()
        loss.backward()
    return {"loss": loss.item(), "grads": par.grad}


def exact(case, seed):
    h = _h(case)
    if case["kind"] == "project":
        return _exact_project(h, *_project_inputs(case, seed))
    if case["kind"] == "step":
        return _exact_step(case, seed)
    if case["kind"] == "advect":
        vel, phi, _ = _grid_inputs(case, seed)
        return _exact_advect(vel, phi, h, 0.25 * h, case["order"])
    if case["kind"] == "constrain":
        vel, phi, cw = _grid_inputs(case, seed)
        return dict(zip("uvw", _exact_constrain(vel, phi, cw, h)))
    if case["kind"] == "transfer":
        return _exact_transfer(case, seed)
    if case["kind"] == "unet":
        return _exact_unet(case, seed)
    return None     # a whole FLIP step moves particles between cells by their ranks: no value in 64 bits
