"""The work a program has this library do, as measurable cases.

Each case is one pass through the public entry points: a projection of a velocity field that sits in
device or host memory, a time step, a batch of patches in one launch, a training pass of the learned
preconditioner's network.  `listed` names the representative ones, `draw` gives more of the same
ranges, `prepare` makes what a program holds before the call, `run` is one pass, `work` the bytes and
operations a pass cannot do without and `exact` the result in 64 bits from plain torch.

Lengths are in metres, the grid is `nx` x `ny` x `nz` cubic cells of side `dx`, x fastest in memory and
z up.  Arrays below are shaped (z, y, x); u, v and w sit on the faces of their axis.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fluidisim_b200 import batch, learned
from fluidisim_b200.delta3d import STORAGE_F16, Volume3

RHO, G = 1025.0, 9.81
DT = 1.0 / 60.0      # projections: one frame
STEP_US = 2000       # time steps: 2 ms
MAX_ITERS = 4000


def listed():
    return [
        # The smallest call: one 2 ms step of the reference's wave tank (8 x 4 x 6 m, 4 m of water) at 25 cm,
        # where launches and latency are everything.
        dict(name="step_32", kind="step", nx=32, ny=16, nz=24, bump=False, wave=1.0),
        # The same tank over an uneven bottom at 6.25 cm: the ordinary time step of a running simulation.
        dict(name="step_128_bump", kind="step", nx=128, ny=64, nz=96, bump=True, wave=1.0),
        # A closed lake with eight spheres, fields in host arrays on both sides: a program that keeps its
        # velocities in host memory.
        dict(name="lake_64_host", kind="project", nx=64, ny=64, nz=64, fill=0.5, swell=0.0, solids="spheres", count=8,
             noise=0.6, multigrid=True, storage="f32", host=True),
        # The headline projection: a 128^3 basin with sixteen boxes under a wavy surface, fields in HBM.
        dict(name="basin_128", kind="project", nx=128, ny=128, nz=128, fill=0.5, swell=2.5, solids="boxes", count=16,
             noise=0.5, multigrid=True, storage="f32", host=False),
        # The same with the V-cycle's vectors stored in FP16.
        dict(name="basin_128_f16", kind="project", nx=128, ny=128, nz=128, fill=0.5, swell=2.5, solids="boxes",
             count=16, noise=0.5, multigrid=True, storage="f16", host=False),
        # The largest: a 256^3 bore running over 32 obstacles, which streams from HBM.
        dict(name="wave_256", kind="project", nx=256, ny=256, nz=256, fill=0.4, swell=0.0, solids="bore", count=32,
             noise=0.5, multigrid=True, storage="f32", host=False),
        # Odd sides, which cannot be coarsened: the default Jacobi-preconditioned CG.
        dict(name="jacobi_75x61x47", kind="project", nx=75, ny=61, nz=47, fill=0.6, swell=1.0, solids="spheres",
             count=4, noise=0.5, multigrid=False, storage="f32", host=False),
        # A ragged box: even sides whose halves soon are odd, so the hierarchy stops at a large level.
        dict(name="ragged_180x100x76", kind="project", nx=180, ny=100, nz=76, fill=0.7, swell=1.5, solids="boxes",
             count=6, noise=0.5, multigrid=True, storage="f32", host=False),
        # A shallow window of which a curved band of columns is in the sparse set.
        dict(name="sparse_256x256x32", kind="sparse", nx=256, ny=256, nz=32, fill=0.5, half_width=3, noise=0.3),
        # Many uneven patches in one launch.
        dict(name="patches_128", kind="patches", patches=128, lo=16, hi=96),
        # The fixed-lid step over an uneven bottom at 12.5 cm (about 220 Jacobi-CG iterations).
        dict(name="linear_64", kind="linear", nx=64, ny=32, nz=32, wave=1.0),
        # Training the learned preconditioner: forward and backward of four 64^3 samples.
        dict(name="unet_train_4x64", kind="unet", batch=4, nx=64, ny=64, nz=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["project", "project", "project", "project", "jacobi", "ragged", "step", "step", "sparse",
                       "patches", "linear", "unet"])
    if kind in ("project", "ragged"):
        q = rng.choice([8, 16]) if kind == "project" else 2  # sides 2 x anything stop coarsening early
        hi = 224 if kind == "project" else 140
        nx, ny, nz = (max(24, q * round(_log(rng, 24, hi) / q)) for _ in range(3))
        return dict(kind="project", nx=nx, ny=ny, nz=nz, fill=rng.uniform(0.35, 0.75), swell=rng.uniform(0.0, 2.0),
                    solids=rng.choice(["spheres", "boxes"]), count=rng.randint(0, 16), noise=rng.uniform(0.4, 0.8),
                    multigrid=True, storage="f16" if kind == "project" and rng.random() < 0.25 else "f32",
                    host=rng.random() < 0.2)
    if kind == "jacobi":
        nx, ny, nz = (round(_log(rng, 17, 90)) for _ in range(3))
        return dict(kind="project", nx=nx, ny=ny, nz=nz, fill=rng.uniform(0.4, 0.7), swell=rng.uniform(0.0, 0.5),
                    solids="spheres", count=rng.randint(0, 4), noise=rng.uniform(0.2, 0.8), multigrid=False,
                    storage="f32", host=False)
    if kind == "step":
        nx = 4 * round(_log(rng, 24, 160) / 4)
        return dict(kind="step", nx=nx, ny=nx // 2, nz=3 * nx // 4, bump=rng.random() < 0.5,
                    wave=rng.uniform(0.3, 1.0))
    if kind == "sparse":
        nx, ny = (16 * round(_log(rng, 64, 320) / 16) for _ in range(2))
        return dict(kind="sparse", nx=nx, ny=ny, nz=rng.choice([16, 24, 32, 48]), fill=rng.uniform(0.4, 0.7),
                    half_width=rng.randint(1, 4), noise=rng.uniform(0.1, 0.5))
    if kind == "patches":
        return dict(kind="patches", patches=rng.randint(8, 128), lo=16, hi=rng.choice([48, 64, 80, 96]))
    if kind == "linear":
        nx = 2 * round(_log(rng, 24, 128) / 2)
        return dict(kind="linear", nx=nx, ny=nx // 2, nz=nx // 2, wave=rng.uniform(0.3, 1.0))
    nx, ny, nz = (4 * round(_log(rng, 16, 64) / 4) for _ in range(3))
    return dict(kind="unet", batch=rng.randint(1, 4), nx=nx, ny=ny, nz=nz)


# ------------------------------------------------------------------------------------------ scenes
# Everything is made on the device from the seed; the library takes geometry and surfaces from host
# arrays, as its reference does.

def _shapes(nx, ny, nz):
    return (nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _dx(value):
    return float(np.float32(value))


def _nodes(nx, ny, nz, dx):
    ax = [torch.arange(n + 1, dtype=torch.float32, device="cuda") * dx for n in (nx, ny, nz)]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _sdf_spheres(nx, ny, nz, dx, centres, radii, out=None):
    x, y, z = _nodes(nx, ny, nz, dx)
    if out is None:
        out = torch.full((nz + 1, ny + 1, nx + 1), 1e3, device="cuda")
    for (a, b, c), r in zip(centres, radii):
        out = torch.minimum(out, torch.sqrt((x - a) ** 2 + (y - b) ** 2 + (z - c) ** 2) - r)
    return out


def _sdf_boxes(nx, ny, nz, dx, centres, halves, out=None):
    x, y, z = _nodes(nx, ny, nz, dx)
    if out is None:
        out = torch.full((nz + 1, ny + 1, nx + 1), 1e3, device="cuda")
    for c, h in zip(centres, halves):
        q = [(p - m).abs() - s for p, m, s in zip((x, y, z), c, h)]
        outside = torch.sqrt(sum(p.clamp(min=0.0) ** 2 for p in q))
        out = torch.minimum(out, outside + torch.maximum(torch.maximum(q[0], q[1]), q[2]).clamp(max=0.0))
    return out


def _background(nx, ny, nz, dx, rng):
    """A divergence-free field: the discrete curl of a smooth vector potential on the cell edges."""
    def potential(shape, sx, sy, sz):
        k, j, i = (torch.arange(n, dtype=torch.float64, device="cuda") for n in shape)
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for _ in range(4):
            fx, fy, fz = (rng.uniform(0.5, 3.0) * 2 * math.pi / n for n in (nx, ny, nz))
            amp, ph = rng.uniform(0.5, 1.5) * min(nx, ny, nz) * dx / (6 * math.pi), rng.uniform(0, 2 * math.pi)
            out += amp * torch.sin((fx * (i + sx))[None, None, :] + (fy * (j + sy))[None, :, None]
                                   + (fz * (k + sz))[:, None, None] + ph)
        return out
    ax = potential((nz + 1, ny + 1, nx), 0.5, 0.0, 0.0)
    ay = potential((nz + 1, ny, nx + 1), 0.0, 0.5, 0.0)
    az = potential((nz, ny + 1, nx + 1), 0.0, 0.0, 0.5)
    u = (az[:, 1:, :] - az[:, :-1, :]) - (ay[1:] - ay[:-1])
    v = (ax[1:] - ax[:-1]) - (az[:, :, 1:] - az[:, :, :-1])
    w = (ay[:, :, 1:] - ay[:, :, :-1]) - (ax[:, 1:] - ax[:, :-1])
    return [(f / dx).float() for f in (u, v, w)]


def _project_scene(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = _dx(0.1)
    rng, gen = np.random.default_rng(seed), _generator(seed)
    i, j = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5, indexing="xy")
    h = np.full((ny, nx), case["fill"] * nz)
    if case["solids"] == "bore":  # a front across the middle, steep over eight cells
        h = h + 0.25 * case["fill"] * nz * np.tanh((i - nx / 2) / 8.0) * (
            1 + 0.1 * np.sin(j / 5.0 + rng.uniform(0, 6)))
    for _ in range(6):
        kx, ky = rng.uniform(-3, 3) * 2 * np.pi / nx, rng.uniform(-3, 3) * 2 * np.pi / ny
        h = h + case["swell"] * rng.uniform(0.4, 1.6) * np.sin(kx * i + ky * j + rng.uniform(0, 2 * np.pi))
    h = np.clip(h, 4.0, nz - 2.0)
    top = float(h.min()) - 3.0
    sdf, taken = None, []
    for q in range(case["count"]):
        r = rng.uniform(2.0, 8.0, size=3)
        sphere = case["solids"] == "spheres" or (case["solids"] == "bore" and q % 2 == 0)
        r = np.minimum(r, [(nx - 3.0) / 4, (ny - 3.0) / 4, (top - 4.5) / 2])
        if sphere:
            r[:] = r.min()
        if r.min() < 1.0:
            continue
        for _ in range(50):  # the obstacles stand two cells apart: no water is shut in between them
            c = np.array([rng.uniform(r[a] + 2.0, n - r[a] - 2.0) for a, n in enumerate((nx, ny, top))])
            if all((np.abs(c - b) > r + a + 2.0).any() for a, b in taken):
                break
        else:
            continue
        taken.append((r, c))
        c, r = [float(x) * dx for x in c], [float(x) * dx for x in r]
        sdf = (_sdf_spheres(nx, ny, nz, dx, [c], [r[0]], sdf) if sphere
               else _sdf_boxes(nx, ny, nz, dx, [c], [r], sdf))
    vel = _background(nx, ny, nz, dx, rng)
    if case["solids"] == "bore":  # the crest runs at 4 m/s
        vel = [torch.zeros(s, device="cuda") for s in _shapes(nx, ny, nz)]
        crest = torch.from_numpy(h > 1.1 * case["fill"] * nz).cuda()
        under = torch.arange(nz, device="cuda")[:, None, None] + 0.5 < torch.from_numpy(h).cuda()
        vel[0][:, :, :-1] += 4.0 * (crest & under)
    vel = [f + case["noise"] * torch.randn(f.shape, generator=gen, device="cuda") for f in vel]
    return dict(nx=nx, ny=ny, nz=nz, dx=dx, rho=RHO, bottom=None,
                sdf=sdf, eta=(h * dx).astype(np.float32), rest=_dx(case["fill"] * nz * dx),
                vel=[f.contiguous() for f in vel], mask=None, dt=DT)


def _tank_scene(case, seed, linear):
    """The reference's 8 m x 4 m tank: 4 m of water 6 m high with a few modes of at most 6 mm (a free
    surface), or a lid at 4 m.  The gentle flow of a wave train."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = _dx(8.0 / nx)
    rng, gen = np.random.default_rng(seed), _generator(seed)
    x, y = np.meshgrid((np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny, indexing="xy")
    wave = case["wave"] * sum(rng.uniform(0.002, 0.006) * np.cos(np.pi * rng.integers(1, 5) * x)
                              * np.cos(np.pi * rng.integers(0, 3) * y) for _ in range(3))
    rest = _dx(nz * dx) if linear else 4.0
    bottom = None
    if linear or case["bump"]:
        bx, by = rng.uniform(2.5, 3.5), rng.uniform(1.1, 1.5)
        bottom = (0.4 + 0.6 * np.exp(-(((8 * x - bx) / 1.2) ** 2 + ((4 * y - by) / 0.9) ** 2))).astype(np.float32)
    vel = [0.05 * f + 0.01 * torch.randn(f.shape, generator=gen, device="cuda")
           for f in _background(nx, ny, nz, dx, rng)]
    return dict(nx=nx, ny=ny, nz=nz, dx=dx, rho=RHO, bottom=bottom, sdf=None,
                eta=(rest + wave).astype(np.float32), rest=rest, vel=[f.contiguous() for f in vel], mask=None,
                dt=STEP_US * 1e-6)


def _sparse_scene(case, seed):
    """A window at rest outside the blocks of 8 x 8 columns along a curved path."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = _dx(0.25)
    rng, gen = np.random.default_rng(seed), _generator(seed)
    bx, by, hw = nx // 8, ny // 8, case["half_width"]
    jj, ii = np.mgrid[0:by, 0:bx]
    blocks = np.zeros((by, bx), bool)
    i, j = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5, indexing="xy")
    bumps, phase = np.zeros((ny, nx)), rng.uniform(0, 2 * np.pi)
    for t in np.linspace(0.0, 1.0, 4 * max(bx, by)):
        px, py = (0.15 + 0.7 * t) * bx, (0.5 + 0.3 * math.sin(2 * math.pi * t + phase)) * by
        blocks |= (np.abs(ii + 0.5 - px) <= hw) & (np.abs(jj + 0.5 - py) <= hw)
        if rng.random() < 0.1:
            bumps += 0.05 * np.exp(-((i - 8 * px) ** 2 + (j - 8 * py) ** 2) / 32.0)
    mask = np.kron(blocks, np.ones((8, 8), bool))
    rest = _dx(case["fill"] * nz * dx)
    eta = np.where(mask, rest + bumps, rest).astype(np.float32)
    vel = [case["noise"] * torch.randn(s, generator=gen, device="cuda") for s in _shapes(nx, ny, nz)]
    return dict(nx=nx, ny=ny, nz=nz, dx=dx, rho=1000.0, bottom=None, sdf=None, eta=eta, rest=rest, vel=vel, mask=mask,
                dt=0.02)


def _patch_scenes(case, seed):
    """Patches with sides log-uniform in [lo, hi] (multiples of 8; the same sides for every seed), spheres in
    5 to 15 % of the cells."""
    rng, gen, sides = np.random.default_rng(seed), _generator(seed), np.random.default_rng(case["patches"])
    out = []
    for _ in range(case["patches"]):
        nx, ny, nz = (int(max(8, 8 * round(_log(sides, case["lo"], case["hi"]) / 8))) for _ in range(3))
        dx = _dx(0.1)
        centres, radii, solid, target = [], [], 0.0, rng.uniform(0.05, 0.15) * nx * ny * nz
        while solid < target and len(radii) < 400:
            r = min(rng.uniform(2.0, 6.0), (min(nx, ny) - 2.5) / 2, (nz - 3.5) / 2)
            c = [rng.uniform(r + 1.0, n - r - 1.0) for n in (nx, ny, nz - 1)]
            centres.append([a * dx for a in c])
            radii.append(r * dx)
            solid += 4.0 / 3.0 * math.pi * r ** 3
        fill = rng.uniform(0.3, 0.8)
        eta = np.full((ny, nx), np.float32(fill * nz * dx), np.float32)
        vel = [2.0 * torch.rand(s, generator=gen, device="cuda") - 1.0 for s in _shapes(nx, ny, nz)]
        out.append(dict(nx=nx, ny=ny, nz=nz, dx=dx, rho=RHO, bottom=None,
                        sdf=_sdf_spheres(nx, ny, nz, dx, centres, radii), eta=eta, rest=float(eta[0, 0]), vel=vel,
                        mask=None, dt=DT))
    return out


# Channels of the network's layers in execution order; a layer's parameters are w[27][out][in], b[out].
LAYERS = [(3, 16), (16, 32), (32, 64), (96, 32), (48, 16), (16, 1)]


def _unet_scene(case, seed):
    gen, rng = _generator(seed), np.random.default_rng(seed)
    n, cells = case["batch"], case["nx"] * case["ny"] * case["nz"]
    params = np.concatenate([np.concatenate([
        rng.normal(0.0, math.sqrt(2.0 / (27 * cin)), 27 * cin * cout), rng.normal(0.0, 0.02, cout)])
        for cin, cout in LAYERS]).astype(np.float32)
    x = torch.randn((n, cells, 3), generator=gen, device="cuda")
    solid = torch.rand((n, cells), generator=gen, device="cuda") < 0.1
    liquid = (torch.arange(cells, device="cuda") < cells // 2) & ~solid
    x[..., 0] *= liquid * 40.0  # a residual's scale; the network sees it over its rms
    x[..., 1], x[..., 2] = solid.float(), liquid.float()
    rms = x[..., 0].double().square().mean(dim=1).sqrt().cpu().numpy()
    gout = torch.randn((n, cells), generator=gen, device="cuda") / cells
    return dict(params=params, x=x.reshape(-1), gout=gout.reshape(-1), in_scale=(1.0 / rms).astype(np.float32),
                out_scale=(rms * 0.01).astype(np.float32))


def _scenes(case, seed):
    if case["kind"] == "project":
        return [_project_scene(case, seed)]
    if case["kind"] in ("step", "linear"):
        return [_tank_scene(case, seed, case["kind"] == "linear")]
    if case["kind"] == "sparse":
        return [_sparse_scene(case, seed)]
    return _patch_scenes(case, seed)


# ------------------------------------------------------------------------------------------ a pass
def _scalars(scene):
    return float(np.float32(-scene["rho"] / scene["dt"])), float(np.float32(scene["dt"] / scene["rho"]))


class _Field:
    """n floats of a volume at a device address, which keep the volume alive."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (address, False), "version": 3}


def _volume(scene, multigrid=True, storage="f32"):
    nx, ny, nz = scene["nx"], scene["ny"], scene["nz"]
    if scene["sdf"] is not None:
        v = Volume3.configure_with_solid(nx, ny, nz, scene["dx"], scene["rho"], G, np.zeros(nx * ny, np.float32),
                                         scene["sdf"].reshape(-1).cpu().numpy())
    elif scene["bottom"] is not None:
        v = Volume3.configure_with_bottom(nx, ny, nz, scene["dx"], scene["rho"], G, scene["bottom"].reshape(-1))
    else:
        v = Volume3.configure(nx, ny, nz, scene["dx"], scene["rho"], G)
    if storage == "f16":
        v.set_options(storage=STORAGE_F16)
    if multigrid:
        v.enable_multigrid()
    if scene["mask"] is not None:
        v.set_free_surface(np.full(nx * ny, scene["rest"], np.float32), scene["rest"])
        v.enable_sparse()
        v.set_active_columns(scene["mask"])
    v.set_free_surface(scene["eta"].reshape(-1), scene["rest"])
    return v


def _fields(v):
    return dict(zip("puvw", (torch.as_tensor(_Field(v, a, n), device="cuda")
                             for a, n in zip(v.device_fields(), (v.cells, v.nu, v.nv, v.nw)))))


def prepare(case, seed):
    if case["kind"] == "unet":
        s = _unet_scene(case, seed)
        net = learned.UNet(case["batch"], case["nz"], case["ny"], case["nx"])
        net.set_params(s["params"])
        s.update(case=case, net=net, y=torch.empty_like(s["gout"]))
    elif case["kind"] == "patches":
        scenes = _patch_scenes(case, seed)
        vols = [_volume(x) for x in scenes]
        scale, k1 = _scalars(scenes[0])
        fields, inputs = [_fields(v) for v in vols], []
        for v, x, f in zip(vols, scenes, fields):  # the batch takes fields whose closed faces are at rest
            v.set_velocity_device(*[a.data_ptr() for a in x["vel"]])
            inputs.append([f[q].clone() for q in "uvw"])
        s = dict(case=case, vols=vols, fields=fields, vel=inputs, scale=[scale] * len(vols), k1=[k1] * len(vols),
                 inputs=[tuple(a.data_ptr() for a in x) for x in inputs], batch=batch.PersistentBatch(vols))
    else:
        scene, = _scenes(case, seed)
        v = _volume(scene, case.get("multigrid", case["kind"] != "linear"), case.get("storage", "f32"))
        scale, k1 = _scalars(scene)
        s = dict(case=case, vol=v, fields=_fields(v), vel=scene["vel"], eta=scene["eta"].reshape(-1),
                 rest=scene["rest"], scale=scale, k1=k1)
        if case.get("host"):
            s["vel"] = [f.reshape(-1).cpu().numpy() for f in scene["vel"]]
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "unet":
        net = s["net"]
        net.forward(case["batch"], case["nz"], case["ny"], case["nx"], s["x"].data_ptr(), s["in_scale"],
                    s["out_scale"], s["y"].data_ptr())
        net.backward(s["gout"].data_ptr())
        return dict(y=s["y"], grads=net.grads())
    if kind == "patches":
        s["batch"].project(s["scale"], s["k1"], MAX_ITERS, reset_pressure=True, inputs=s["inputs"])
        return {q: torch.cat([f[q] for f in s["fields"]]) for q in "puvw"}  # gathered for the next stage
    v = s["vol"]
    if kind in ("step", "linear"):
        v.set_free_surface(s["eta"], s["rest"])
        v.set_velocity_device(*[f.data_ptr() for f in s["vel"]])
        (v.step_surface_linear if kind == "linear" else v.step_surface_mobile)(STEP_US, MAX_ITERS)
        return dict(s["fields"], eta=v.surface())
    if case.get("host"):
        v.set_velocity(*s["vel"])
        v.reset_pressure()
        v.project_mobile3(s["scale"], s["k1"], MAX_ITERS)
        return dict(zip("uvw", v.velocity()), p=v.pressure())
    v.set_velocity_device(*[f.data_ptr() for f in s["vel"]])
    v.reset_pressure()
    v.project_mobile3(s["scale"], s["k1"], MAX_ITERS)
    return s["fields"]


def work(case):
    if case["kind"] == "unet":
        cells = case["batch"] * case["nx"] * case["ny"] * case["nz"]
        level = [1.0, 1 / 8, 1 / 64, 1 / 8, 1.0, 1.0]
        macs = sum(f * 27 * a * b for f, (a, b) in zip(level, LAYERS)) * cells
        params = sum(27 * a * b + b for a, b in LAYERS)
        # in: 3 channels and the output's gradient; out: y and the parameters' gradients; each product
        # once forward and twice backward, less the input's own gradient
        return dict(bytes=4.0 * (cells * 5 + 2 * params), flops=2.0 * (3 * macs - 27 * 3 * 16 * cells))
    if case["kind"] == "patches":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])  # of a log-uniform side
        cells, cut = case["patches"] * mean ** 3, True
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        cut = case["kind"] == "linear" or bool(case.get("bump")) or case.get("count", 0) > 0
    # three velocity components read and written, the pressure written, and the cut's fraction and three
    # apertures read where there is one; a divergence, one application of the operator, one correction
    return dict(bytes=4.0 * cells * (7 + (4 if cut else 0)), flops=40.0 * cells)


# ------------------------------------------------------------------------------------ 64-bit results
F64 = torch.float64


def _split(a, axis):
    """The entries before and after each interior face of an axis."""
    n = a.shape[axis]
    return a.narrow(axis, 0, n - 1), a.narrow(axis, 1, n - 1)


def _prism_below(v, d):
    """Share of {0 < z < d} that lies under a surface linear on a triangle with corner heights v (..., 3),
    averaged over the triangle."""
    v = v.sort(dim=-1).values
    v0, v1, v2 = v.unbind(-1)

    def area(s):  # integral over (-inf, s) of the share of the triangle whose height is below s
        a, b, span = ((q - p).clamp(min=1e-100) for p, q in ((v0, v1), (v1, v2), (v0, v2)))
        low = (torch.minimum(s, v1) - v0).clamp(min=0.0) ** 3 / (3 * a * span)
        m = torch.minimum(s, v2)
        high = (m - v1).clamp(min=0.0) - (b ** 3 - (v2 - m).clamp(min=0.0).clamp(max=b) ** 3) / (3 * span * b)
        return torch.where(s <= v0, 0.0, low + torch.where(s > v1, high, torch.zeros_like(high))
                           + (s - v2).clamp(min=0.0))
    return ((area(torch.full_like(v0, d)) - area(torch.zeros_like(v0))) / d).clamp(0.0, 1.0)


def _below(v, s):
    """Share of a simplex's area (3 corners) or length (2) where a linear function is below s."""
    v = v.sort(dim=-1).values
    if v.shape[-1] == 2:
        a, b = v.unbind(-1)
        return torch.where(b > a, ((s - a) / (b - a).clamp(min=1e-300)).clamp(0.0, 1.0), (a < s).to(F64))
    a, b, c = v.unbind(-1)
    low = (s - a) ** 2 / ((b - a) * (c - a)).clamp(min=1e-300)
    high = 1.0 - (c - s) ** 2 / ((c - a) * (c - b)).clamp(min=1e-300)
    return torch.where(s <= a, 0.0, torch.where(s >= c, 1.0, torch.where(s <= b, low, high)))


def _bottom_cut(bottom, nx, ny, nz, dx):
    b = torch.as_tensor(bottom, dtype=F64, device="cuda")
    e = torch.cat([b[:, :1], 0.5 * (b[:, :-1] + b[:, 1:]), b[:, -1:]], dim=1)
    c = torch.cat([e[:1], 0.5 * (e[:-1] + e[1:]), e[-1:]], dim=0)  # heights at the column corners
    quad = torch.stack([c[:-1, :-1], c[:-1, 1:], c[1:, 1:], c[1:, :-1]], dim=-1)
    mid = quad.mean(dim=-1)
    tri = torch.stack([torch.stack([quad[..., a], quad[..., (a + 1) % 4], mid], dim=-1) for a in range(4)], dim=-2)
    frac = torch.stack([_prism_below(tri - k * dx, dx).mean(dim=-1) for k in range(nz)])
    def side(p, q):  # share of a face under its edge from height p to height q: a wall of zero thickness
        low, high = torch.minimum(p, q), torch.maximum(p, q)
        mean = lambda s: torch.where(high > low, (s - low).clamp(min=0.0).minimum(high - low) ** 2
                                     / (2 * (high - low).clamp(min=1e-300)) + (s - high).clamp(min=0.0),
                                     (s - low).clamp(min=0.0))
        return torch.stack([((mean(torch.full_like(p, (k + 1) * dx)) - mean(torch.full_like(p, k * dx))) / dx)
                            for k in range(nz)])
    au, av = side(c[:-1, :], c[1:, :]), side(c[:, :-1], c[:, 1:])
    au[..., 0] = au[..., -1] = 0.0
    av[:, 0] = av[:, -1] = 0.0
    aw = torch.stack([torch.zeros_like(mid)] + [
        torch.stack([_below(tri[..., a, :], k * dx) for a in range(4)]).mean(dim=0) for k in range(1, nz + 1)])
    return frac, au, av, aw


def _negative(v):
    """Share of a simplex (3 or 4 corners, values v (..., m)) where a linear function is negative."""
    m = v.shape[-1]
    v = v.sort(dim=-1).values
    out = (v[..., -1] < 0).to(F64)
    tiny = 1e-300
    a = -v[..., 0]
    out = torch.where((v[..., 0] < 0) & (v[..., 1] >= 0),
                      a ** (m - 1) / torch.stack([a + v[..., q] for q in range(1, m)]).prod(dim=0).clamp(min=tiny), out)
    d = v[..., -1]
    out = torch.where((v[..., -2] < 0) & (d >= 0),
                      1 - d ** (m - 1) / torch.stack([d - v[..., q] for q in range(m - 1)]).prod(dim=0).clamp(min=tiny),
                      out)
    if m == 4:
        b, c = -v[..., 1], v[..., 2]
        two = (c * d * (a * a + a * b + b * b) + (c + d) * a * b * (a + b) + a * a * b * b) / (
            (c + a) * (d + a) * (c + b) * (d + b)).clamp(min=tiny)
        out = torch.where((v[..., 1] < 0) & (c >= 0), two, out)
    return out


def _solid_cut(sdf, nx, ny, nz, geo):
    """Takes a solid out of the fractions and apertures: 24 tetrahedra a cell, four triangles a face."""
    s = sdf.to(F64)
    frac, au, av, aw = geo

    def quad(c):
        m = (c[0] + c[1] + c[2] + c[3]) / 4
        return [torch.stack([c[a], c[(a + 1) % 4], m], dim=-1) for a in range(4)]
    def face(c):
        return sum(_negative(t) for t in quad(c)) / 4
    lo, hi = slice(0, -1), slice(1, None)
    cut = lambda ap, neg: torch.where(neg > 0, 1.0 - neg, ap)
    au[..., 1:-1] = cut(au[..., 1:-1], face([s[a, b, 1:-1] for a, b in ((lo, lo), (lo, hi), (hi, hi), (hi, lo))]))
    av[:, 1:-1] = cut(av[:, 1:-1], face([s[a, 1:-1, b] for a, b in ((lo, lo), (lo, hi), (hi, hi), (hi, lo))]))
    aw[1:] = cut(aw[1:], face([s[1:][:, a, b] for a, b in ((lo, lo), (lo, hi), (hi, hi), (hi, lo))]))
    n = {(a, b, c): s[hi if c else lo, hi if b else lo, hi if a else lo] for a in (0, 1) for b in (0, 1) for c in (0, 1)}
    near = torch.stack(list(n.values())).amin(dim=0) < 0  # the rest is untouched
    n = {k: x[near] for k, x in n.items()}
    centre = sum(n.values()) / 8
    neg = torch.zeros_like(centre)
    for ax in range(3):
        for side in (0, 1):
            ring = [(0, 0), (1, 0), (1, 1), (0, 1)]
            for t in quad([n[p[:ax] + (side,) + p[ax:]] for p in ring]):
                neg += _negative(torch.cat([t, centre[..., None]], dim=-1))
    frac[near] = cut(frac[near], neg / 24)
    return frac, au, av, aw


class _Problem:
    """The rows of one projection in 64 bits: couplings c* of the interior faces between two rows, and the
    ghost coefficient and value of each side of a face that has a row on one side only."""

    def __init__(self, s, linear):
        nx, ny, nz, dx = s["nx"], s["ny"], s["nz"], s["dx"]
        self.dx, self.linear, self.nz = dx, linear, nz
        ones = [torch.ones(x, dtype=F64, device="cuda") for x in [(nz, ny, nx), *_shapes(nx, ny, nz)]]
        geo = _bottom_cut(s["bottom"], nx, ny, nz, dx) if s["bottom"] is not None else ones
        geo[1][..., 0] = geo[1][..., -1] = 0.0
        geo[2][:, 0] = geo[2][:, -1] = 0.0
        geo[3][0] = 0.0
        if s["sdf"] is not None:
            geo = _solid_cut(s["sdf"], nx, ny, nz, geo)
        frac, au, av, aw = geo
        if s["mask"] is not None:
            m = torch.as_tensor(s["mask"], device="cuda")
            frac = frac * m
            au[..., 1:-1] *= m[:, 1:] & m[:, :-1]
            av[:, 1:-1] *= m[1:] & m[:-1]
            aw = aw * m
        sealed = (au[..., :-1] + au[..., 1:] + av[:, :-1] + av[:, 1:] + aw[:-1] + aw[1:]) == 0
        frac = torch.where(sealed, 0.0, frac)
        self.frac, self.ap = frac, (au, av, aw)
        eta32 = torch.as_tensor(s["eta"], device="cuda")
        k32 = (torch.arange(nz, device="cuda", dtype=torch.float32) + 0.5)[:, None, None] * np.float32(dx)
        fluid = frac > 0
        self.row = fluid if linear else fluid & (k32 < eta32)
        self.eta = eta32.to(F64)
        zc = (torch.arange(nz, device="cuda", dtype=F64) + 0.5)[:, None, None] * dx
        rho_g = s["rho"] * G
        self.face, self.diag, self.ghost = [], torch.zeros_like(frac), torch.zeros_like(frac)
        for axis, a in ((2, au[..., 1:-1]), (1, av[:, 1:-1]), (0, aw[1:-1])):
            l, r = _split(self.row, axis)
            fl, fr = _split(fluid, axis)
            live = (a > 0) & fl & fr
            both = torch.where(live & l & r, a, 0.0)
            dl, dr = _split(self.diag, axis)
            dl += both
            dr += both
            entry = dict(axis=axis, both=both, pair=live & l & r)
            if not linear and axis != 0:  # the surface between two columns
                h = self.eta.expand_as(frac)
                hl, hr = _split(h, axis)
                z = _split(zc.expand_as(frac), axis)[0]
                value = rho_g * (z - s["rest"])
                gl, gr = _split(self.ghost, axis)
                for name, on, hc, hn, d, g in (("left", live & l & ~r, hl, hr, dl, gl),
                                               ("right", live & r & ~l, hr, hl, dr, gr)):
                    it = torch.where(on, 1.0 / torch.where(on, ((hc - z) / torch.where(on, hc - hn, 1.0)), 1.0)
                                     .clamp(min=float(np.float32(1e-3))), 0.0)
                    d += a * it
                    g += a * it * value
                    entry[name] = (it, value)
            self.face.append(entry)
        # the face above a row: the surface over its column, or the lid half a cell away
        up = aw[1:]
        if linear:
            on = torch.zeros_like(self.row)
            on[-1] = self.row[-1] & (up[-1] > 0)
            self.up_it = torch.where(on, 2.0, 0.0)
            self.up_value = (rho_g * (self.eta - nz * dx)).expand_as(frac)
        else:
            above = torch.zeros_like(self.row)
            above[:-1] = self.row[1:]
            on = self.row & (up > 0) & ~above
            self.up_it = torch.where(on, 1.0 / ((self.eta - zc) / dx).clamp(min=float(np.float32(1e-3))), 0.0)
            self.up_value = (rho_g * (self.eta - s["rest"])).expand_as(frac)
        self.diag += up * self.up_it
        self.ghost += up * self.up_it * self.up_value

    def close(self, vel):
        """Walls and closed faces carry no velocity."""
        u, v, w = (f.to(F64) * (a > 0) for f, a in zip(vel, self.ap))
        return u, v, w

    def divergence(self, vel):
        u, v, w = (f * a for f, a in zip(vel, self.ap))
        d = (u[..., 1:] - u[..., :-1] + w[1:] - w[:-1] + v[:, 1:] - v[:, :-1]) / self.dx
        return torch.where(self.frac > 0, d, 0.0)

    def apply(self, x):
        out = self.diag * x
        for f in self.face:
            lx, rx = _split(x, f["axis"])
            lo, ro = _split(out, f["axis"])
            lo -= f["both"] * rx
            ro -= f["both"] * lx
        return out / self.dx ** 2

    def solve(self, vel, scale):
        b = torch.where(self.row, scale * self.divergence(vel) + self.ghost / self.dx ** 2, 0.0)
        m = torch.where(self.diag > 0, self.dx ** 2 / self.diag.clamp(min=1e-300), 0.0) * self.row
        x, r = torch.zeros_like(b), b.clone()
        z = m * r
        d, rz = z.clone(), (r * z).sum()
        stop = float((b * b).sum()) * 1e-26
        for it in range(20000):
            q = self.apply(d)
            a = rz / (d * q).sum()
            x += a * d
            r -= a * q
            if it % 20 == 19 and float((r * r).sum()) <= stop:
                break
            z = m * r
            rz, old = (r * z).sum(), rz
            d = z + (rz / old) * d
        return x

    def correct(self, vel, p, k1):
        u, v, w = (f.clone() for f in vel)
        inner = {2: u[..., 1:-1], 1: v[:, 1:-1], 0: w[1:-1]}
        for f in self.face:
            l, r = _split(p, f["axis"])
            grad = torch.where(f["pair"], r - l, 0.0)
            if "left" in f:
                it, value = f["left"]
                grad += (value - l) * it
                it, value = f["right"]
                grad += (r - value) * it
            inner[f["axis"]] -= k1 * grad / self.dx
        w[1:] -= k1 * torch.where(self.up_it > 0, (self.up_value - p) * self.up_it, 0.0) / self.dx
        return u, v, w


def _advect(pb, vel, dt):
    """Centred advection of every open interior face."""
    u, v, w = vel
    h = 0.5 / pb.dx

    def pad(a, axis):  # a neighbour outside the box reads as the face itself
        return torch.cat([a.narrow(axis, 0, 1), a, a.narrow(axis, a.shape[axis] - 1, 1)], dim=axis)

    def slope(a, axis):
        e = pad(a, axis)
        return (e.narrow(axis, 2, a.shape[axis]) - e.narrow(axis, 0, a.shape[axis])) * h

    def mean(a, own, other):  # `a`, on the faces of `other`, at the interior faces of `own`
        l, r = _split(a, own)
        p, q = _split(l + r, other)
        return 0.25 * (p + q)
    nu, nv, nw = u.clone(), v.clone(), w.clone()
    i = lambda a, axis: a.narrow(axis, 1, a.shape[axis] - 2)
    for f, new, own, (o1, a1), (o2, a2) in ((u, nu, 2, (v, 1), (w, 0)), (v, nv, 1, (u, 2), (w, 0)),
                                            (w, nw, 0, (u, 2), (v, 1))):
        ap = pb.ap[{2: 0, 1: 1, 0: 2}[own]]
        rate = (i(f, own) * i(slope(f, own), own) + mean(o1, own, a1) * i(slope(f, a1), own)
                + mean(o2, own, a2) * i(slope(f, a2), own))
        i(new, own).sub_(torch.where(i(ap, own) > 0, dt * rate, 0.0))
    return nu, nv, nw


def _extrapolate(pb, vel):
    """Above the surface, the open faces of a column take its last solved face."""
    wet, fluid = pb.row, pb.frac > 0
    for f, ap, axis in zip(vel, pb.ap, (2, 1, 0)):
        if axis == 0:
            solved = torch.zeros_like(ap, dtype=torch.bool)
            solved[1:] = (ap[1:] > 0) & wet
        else:
            solved = torch.zeros_like(ap, dtype=torch.bool)
            (a, b), (c, d) = _split(wet, axis), _split(fluid, axis)
            solved.narrow(axis, 1, ap.shape[axis] - 2).copy_((a | b) & c & d)
            solved &= ap > 0
        last, has = torch.zeros_like(f[0]), torch.zeros_like(f[0], dtype=torch.bool)
        for k in range(f.shape[0]):
            take = has & ~solved[k] & (ap[k] > 0)
            f[k] = torch.where(take, last, f[k])
            last = torch.where(solved[k], f[k], last)
            has |= solved[k]
    return vel


def _transport(pb, vel, dt):
    eta, (u, v, _), (au, av, _) = pb.eta, vel, pb.ap
    k = torch.arange(pb.nz, device="cuda", dtype=F64)[:, None, None] * pb.dx

    def flux(f, a, axis):
        out = torch.zeros_like(f[0])
        inner = (f * a).narrow(axis + 1, 1, f.shape[axis + 1] - 2) * pb.dx
        if not pb.linear:
            l, r = _split(eta, axis)
            inner = inner * ((0.5 * (l + r) - k) / pb.dx).clamp(0.0, 1.0)
        out.narrow(axis, 1, out.shape[axis] - 2).copy_(inner.sum(dim=0))
        return out
    x, y = flux(u, au, 1), flux(v, av, 0)
    return eta - dt / pb.dx * ((x[:, 1:] - x[:, :-1]) + (y[1:] - y[:-1]))


def _unet_exact(case, seed):
    s = _unet_scene(case, seed)
    n, dims = case["batch"], (case["nz"], case["ny"], case["nx"])
    flat = torch.as_tensor(s["params"], device="cuda").to(F64)
    layers, at = [], 0
    for cin, cout in LAYERS:
        w = flat[at:at + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2).contiguous()
        at += 27 * cin * cout
        layers.append((w.requires_grad_(), flat[at:at + cout].clone().requires_grad_()))
        at += cout
    x = s["x"].to(F64).reshape(n, *dims, 3).permute(0, 4, 1, 2, 3).clone()
    x[:, 0] *= torch.as_tensor(s["in_scale"], device="cuda").to(F64)[:, None, None, None]

    def conv(a, q, relu=True):
        w, b = layers[q]
        a = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
        z, y, xx = (d - 2 for d in a.shape[2:])
        out = b[None, :, None, None, None]
        for t in range(27):  # one tap at a time: a product over the channels
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            out = out + torch.einsum("oc,nczyx->nozyx", w[:, :, dz, dy, dx],
                                     a[:, :, dz:dz + z, dy:dy + y, dx:dx + xx])
        return out.relu() if relu else out
    pool = lambda a: torch.nn.functional.avg_pool3d(a, 2)
    up = lambda a: a.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    e0 = conv(x, 0)
    e1 = conv(pool(e0), 1)
    b = conv(pool(e1), 2)
    d1 = conv(torch.cat([up(b), e1], dim=1), 3)
    d0 = conv(torch.cat([up(d1), e0], dim=1), 4)
    y = conv(d0, 5, relu=False) * torch.as_tensor(s["out_scale"], device="cuda").to(F64)[:, None, None, None, None]
    y = y.reshape(-1)
    y.backward(s["gout"].to(F64))
    grads = torch.cat([torch.cat([w.grad.permute(2, 3, 4, 0, 1).reshape(-1), b.grad]) for w, b in layers])
    return dict(y=y.detach(), grads=grads)


def exact(case, seed):
    if case["kind"] == "unet":
        return _unet_exact(case, seed)
    if case["kind"] != "patches" and case["nx"] * case["ny"] * case["nz"] > 6_000_000:
        return None  # a minute of conjugate gradients in 64 bits
    parts = []
    for s in _scenes(case, seed):
        scale, k1 = _scalars(s)
        linear = case["kind"] == "linear"
        pb = _Problem(s, linear)
        vel = pb.close(s["vel"])
        if case["kind"] == "step":
            vel = _advect(pb, vel, float(np.float32(s["dt"])))
        p = pb.solve(vel, scale)
        vel = pb.correct(vel, p, k1)
        if case["kind"] == "step":
            vel = _extrapolate(pb, vel)
        out = dict(zip("puvw", (f.reshape(-1) for f in (p, *vel))))
        if case["kind"] in ("step", "linear"):
            out["eta"] = _transport(pb, vel, s["dt"]).reshape(-1)
        parts.append(out)
    return {q: torch.cat([x[q] for x in parts]) for q in parts[0]}
