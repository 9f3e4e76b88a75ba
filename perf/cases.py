"""Performance cases of the framework: the work its users have it do, through the public entry points.

The sizes come from the repository's own configurations (the 96x48x48 sphere, the 128x64x64 vehicle and
its x2 and x4 scalings, the batched tunnels' size table, the 200,000-triangle voxelizer mesh, the closure's
65,536-sample minibatch, the tracer counts of the frame loop) and odd sizes between them.

Kinds:
  step    one solver domain advanced by `steps` steps, its drag read (and, with `field`, its velocity field
          read to the host): the runner's loop {step 8, encode force, read force}, a frame of the interactive
          loop, or a longer run; all storages, both operators, LES and wall model, halfway, interpolated and
          free-slip boundaries, and the learned closure attached;
  batch   many uneven tunnels advanced together, each one's drag read;
  train   Adam steps of the learned closure (forward, backward, update);
  load    a new body: voxelize the mesh, create the domain;
  links   voxelize with measured link fractions, the packed geometry read back;
  tracers particles and 3-D streaklines advanced through a field and read for drawing.
"""
import math

import numpy as np
import torch

from pocketwind_gb300.batch import Batch
from pocketwind_gb300.closure import Closure
from pocketwind_gb300.geometry import grid_from_arrays, voxelize
from pocketwind_gb300.solver import GpuSolver, SolverParams
from pocketwind_gb300.tracers import Particles, Streaks

FLUID, SOLID, FLOOR, EQ = 0, 1, 3, 4
ELEM = {"f32": 4, "f16": 2, "bf16": 2}
# the batched-tunnel case's size table
TUNNELS = ((64, 32, 32), (96, 48, 48), (128, 64, 64), (192, 96, 96))


def _step(name, nx, ny, nz, precision, operator, les, body, floor=False, lateral="periodic", walls="bb", steps=8,
          warm=64, field=False, closure=False):
    return {"name": name, "kind": "step", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "operator": operator,
            "les": les, "body": body, "floor": floor, "lateral": lateral, "walls": walls, "steps": steps, "warm": warm,
            "field": field, "closure": closure}


def listed():
    return [
        # the laminar validation sphere, the smallest run: its drag read every 8 steps by the runner
        _step("sphere_96", 96, 48, 48, "f32", "trt", False, "sphere", lateral="free-slip"),
        # the turbulent vehicle at the interactive size: a frame of 8 steps with macros written and the drag read
        _step("vehicle_128", 128, 64, 64, "f32", "reg", True, "vehicle", floor=True),
        # a user-chosen size that is odd in every direction, half-precision storage
        _step("ragged_203", 203, 101, 67, "f16", "trt", False, "sphere"),
        # an ordinary unattended run: 64 steps, the drag, then the velocity field to the host
        _step("vehicle_256_run", 256, 128, 128, "bf16", "reg", True, "vehicle", floor=True, steps=64, warm=16,
              field=True),
        # the full-size vehicle, half-precision storage: the headline configuration, drag read every 8 steps
        _step("vehicle_512", 512, 256, 256, "f16", "reg", True, "vehicle", floor=True, warm=8),
        # curved walls: interpolated bounce-back on measured fractions
        _step("bouzidi_160", 160, 80, 80, "f32", "trt", False, "sphere", walls="bouzidi"),
        # the coarse grid of the learned closure, the network fused into the step
        _step("closure_128", 128, 64, 64, "f32", "reg", True, "vehicle", floor=True, closure=True),
        # a sweep of independent tunnels of uneven size and Reynolds number
        {"name": "batch_32", "kind": "batch", "members": 32, "precision": "f16", "operator": "trt", "les": False,
         "steps": 50},
        # training the closure: minibatches drawn from a dataset on the GPU
        {"name": "train_65536", "kind": "train", "batch": 65536, "samples": 1 << 20, "steps": 20},
        # a new body dropped into the tunnel: the 200,000-triangle mesh, voxelized, and its domain created
        {"name": "load_200k", "kind": "load", "nx": 256, "ny": 128, "nz": 128, "lon": 400, "lat": 251, "floor": False},
        # geometry for interpolated walls on a ragged grid over a floor, read back packed
        {"name": "links_150", "kind": "links", "nx": 150, "ny": 75, "nz": 61, "lon": 96, "lat": 65, "floor": True},
        # one drawing frame's tracers on the interactive grid
        {"name": "tracers_128", "kind": "tracers", "nx": 128, "ny": 64, "nz": 64, "particles": 16384, "rake": 8,
         "slots": 512},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 6 + ["batch", "train", "load", "links", "tracers"])
    if kind == "step":
        nx = log(64, 400)
        ny, nz = max(24, int(nx * rng.uniform(0.4, 0.6))), max(24, int(nx * rng.uniform(0.4, 0.6)))
        if rng.random() < 0.6:
            nx -= nx % 2
        form = rng.choice(["plain", "plain", "floor", "free-slip", "bouzidi", "closure"])
        steps = rng.choice([1, 4, 8, 8, 16, 20, 64, 100]) if nx <= 192 else rng.choice([1, 4, 8, 8, 16])
        les = form in ("floor", "closure") or (form == "plain" and rng.random() < 0.5)
        return {k: v for k, v in _step(
            "", nx, ny, nz, rng.choice(["f32", "f16", "bf16"]), rng.choice(["trt", "reg"]), les,
            rng.choice(["sphere", "vehicle"]) if form in ("plain", "floor") else "sphere",
            floor=form in ("floor", "closure"), lateral="free-slip" if form == "free-slip" else "periodic",
            walls="bouzidi" if form == "bouzidi" else "bb", steps=steps, warm=16,
            field=rng.random() < 0.2, closure=form == "closure").items() if k != "name"}
    if kind == "batch":
        precision = rng.choice(["f32", "f16", "bf16"])
        return {"kind": "batch", "members": rng.randint(3, 15 if precision == "f32" else 32), "precision": precision,
                "operator": rng.choice(["trt", "reg"]), "les": False, "steps": rng.randint(8, 50)}
    if kind == "train":
        return {"kind": "train", "batch": log(500, 65536), "samples": log(1 << 17, 1 << 20), "steps": rng.randint(2, 20)}
    if kind in ("load", "links"):
        nx = log(64, 256)
        return {"kind": kind, "nx": nx, "ny": nx // 2 + rng.randint(0, 5), "nz": nx // 2 - rng.randint(0, 5),
                "lon": log(32, 400), "lat": log(20, 251), "floor": rng.random() < 0.5}
    nx = log(64, 200)
    return {"kind": "tracers", "nx": nx, "ny": nx // 2 + 1, "nz": nx // 2, "particles": log(1000, 65536),
            "rake": rng.randint(4, 16), "slots": log(64, 512)}


# ---------------------------------------------------------------- inputs
C19 = ((0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
       (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1))
W19 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [0] + [i + 1 if i % 2 else i - 1 for i in range(1, 19)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Buffer:
    """A domain's device buffer as torch reads one; a tensor of it keeps the domain alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _view(solver, ptr, shape, typestr):
    return torch.as_tensor(_Buffer(solver, ptr, shape, typestr), device="cuda")


def _setup(case, seed):
    """The body and flow of a step case: sizes, place, speed and Reynolds number jittered by the seed."""
    r = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    s = nx / 128 * (1 + 0.05 * r.uniform(-1, 1))
    at = np.array([nx / 4, ny / 2, nz / 2]) + r.uniform(-1, 1, 3)
    u = 0.05 * (1 + 0.05 * r.uniform(-1, 1))
    if case["body"] == "vehicle":
        length, re = 40 * s, 320 * (1 + 0.1 * r.uniform(-1, 1))
    else:
        length, re = 16 * s, 100 * (1 + 0.1 * r.uniform(-1, 1))
    return {"at": at, "s": s, "u": float(np.float32(u)), "tau0": 0.5 + 3 * max(u * length / re, 0.004)}


def _flags(case, setup, device):
    """Cell kinds and pull-direction wall links of a sphere, or of a slanted block over the ground, cell by cell."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = torch.meshgrid(*(torch.arange(n, device=device, dtype=torch.float64) for n in (nz, ny, nx)), indexing="ij")
    ax, ay, az = setup["at"]
    s = setup["s"]
    if case["body"] == "vehicle":
        tail = torch.clamp(x - (ax + 28 * s), min=0.0) * math.tan(math.radians(25))
        solid = (x >= ax) & (x <= ax + 40 * s) & ((y - ay).abs() <= 8 * s) & (z >= 3 * s) & (z <= 15 * s - tail)
    else:
        solid = (x - ax) ** 2 + (y - ay) ** 2 + (z - az) ** 2 < (8 * s) ** 2
    kind = torch.where(solid, SOLID, FLUID)
    kind[:, :, 0] = EQ
    kind[:, :, nx - 1] = EQ
    if case["floor"]:
        kind[nz - 1] = EQ
        kind[0] = FLOOR
    wall = (kind >= SOLID) & (kind <= FLOOR)
    flags, body = kind.clone(), torch.zeros_like(wall)
    for i, (cx, cy, cz) in enumerate(C19[1:], 1):
        link = torch.roll(wall, (cz, cy, cx), (0, 1, 2)) & (kind == FLUID)
        flags += link * (1 << (3 + i))
        body |= link & (torch.roll(kind, (cz, cy, cx), (0, 1, 2)) == SOLID)
    return flags, body


def _fractions(case, setup, flags, exact_dtype=torch.float32):
    """Per link (cells ascending, links in direction order) how far along it the wall lies; 1/2 for halfway walls."""
    nx, ny = case["nx"], case["ny"]
    f = flags.reshape(-1)
    cells = torch.nonzero(f >> 3).reshape(-1)
    bits = torch.stack([(f[cells] >> (3 + i)) & 1 for i in range(1, 19)], 1).bool()
    q = torch.full(bits.shape, 0.5, dtype=torch.float64, device=f.device)
    if case["walls"] == "bouzidi":
        o = torch.stack([cells % nx, cells // nx % ny, cells // (nx * ny)], 1).double() - torch.tensor(
            setup["at"], device=f.device)
        d = -torch.tensor(C19[1:], dtype=torch.float64, device=f.device)
        b, a, c = o @ d.T, (d * d).sum(1), (o * o).sum(1, keepdim=True) - (8 * setup["s"]) ** 2
        t = (-b - torch.sqrt(torch.clamp(b * b - a * c, min=0.0))) / a
        q = torch.clamp(t, 1e-3, 1.0)
    return cells, bits, q[bits].to(exact_dtype)


def _grid(case, setup):
    dev = _device()
    flags, body = _flags(case, setup, dev)
    cells, bits, q = _fractions(case, setup, flags)
    n = flags.numel()
    off = torch.full((n,), 0xFFFFFFFF, dtype=torch.int64, device=dev)
    count = bits.sum(1)
    off[cells] = torch.cumsum(count, 0) - count
    packed = np.concatenate([torch.cat([flags.reshape(-1), off]).cpu().numpy().astype(np.uint32),
                             q.cpu().numpy().view(np.uint32)])
    boundary = torch.nonzero(body.reshape(-1)).reshape(-1).cpu().numpy().astype(np.uint32)
    return grid_from_arrays((case["nx"], case["ny"], case["nz"]), packed, boundary)


def _params(seed):
    """A network in mid-training: hidden layers at their usual scale, a small output layer."""
    r = np.random.default_rng(seed + 77)
    w1, w2 = r.uniform(-0.38, 0.38, (32, 9)), r.uniform(-0.3, 0.3, (32, 32))
    return np.concatenate([w1.ravel(), r.uniform(-0.1, 0.1, 32), w2.ravel(), r.uniform(-0.1, 0.1, 32),
                           r.uniform(-0.15, 0.15, 32), [0.05]]).astype(np.float32)


def _samples(case, seed):
    """Closure inputs over their usual ranges and targets in [-1, 3] that depend on them."""
    r = np.random.default_rng(seed + 5)
    n = case["samples"]
    x = r.standard_normal((n, 9), np.float32)
    x *= np.array([0.5, 0.3, 0.3, 0.3, 0.4, 0.3, 0.4, 0.5, 0.1], np.float32)
    x += np.array([0.6, 0.0, 0.5, 1.0, 0.9, 0.1, 0.7, 0.6, 2.0], np.float32)
    y = np.tanh(x[:, 0] - x[:, 7]) + 0.5 * x[:, 2] * x[:, 6] + 0.3 * r.standard_normal(n, np.float32)
    return x, np.clip(y, -1, 3).astype(np.float32)


def _mesh(case, seed):
    """A closed latitude-longitude ellipsoid of 2 * lon * (lat - 1) triangles, as a float32 triangle soup."""
    r = np.random.default_rng(seed + 3)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    at = np.array([nx / 4, ny / 2, nz / 2])
    if case["kind"] == "links":  # whole cells: the packed geometry keeps its length
        at[:2] += r.integers(-3, 4, 2)
        rad = nx / 10 * np.array([1.1037, 0.9041, 0.8273])
    else:
        at += r.uniform(-1, 1, 3)
        rad = nx / 10 * r.uniform(0.8, 1.2, 3)
    lon, lat = case["lon"], case["lat"]
    p = np.arange(lon + 1) % lon * (2 * np.pi / lon)
    t = np.arange(lat + 1) * (np.pi / lat)
    g = np.stack([np.sin(t)[:, None] * np.cos(p), np.sin(t)[:, None] * np.sin(p),
                  np.cos(t)[:, None] * np.ones_like(p)], 2)
    g[0], g[-1] = (0, 0, 1), (0, 0, -1)
    g = g * rad + at
    a, b, c, d = g[:-1, :-1], g[1:, :-1], g[1:, 1:], g[:-1, 1:]
    tri = np.concatenate([np.stack([a, b, c], 2)[:-1].reshape(-1, 9), np.stack([a, c, d], 2)[1:].reshape(-1, 9)])
    return tri.astype(np.float32).reshape(-1)


def _tunnels(case, seed):
    """Uneven tunnels drawn from the batch's size table, each with its own sphere, speed and Reynolds number."""
    r = np.random.default_rng(1)  # the sizes are the case's; the seed moves bodies and flows
    out = []
    for k in range(case["members"]):
        nx, ny, nz = TUNNELS[int(r.integers(len(TUNNELS)))]
        t = {"nx": nx, "ny": ny, "nz": nz, "body": "sphere", "floor": False, "walls": "bb", "lateral": "periodic",
             "les": case["les"], "operator": case["operator"], "closure": False}
        out.append((t, _setup(t, seed * 1000 + k)))
    return out


def _field(case, seed):
    """A smooth shear flow with swirls past a sphere (rho, u) and the sphere's geometry."""
    r = np.random.default_rng(seed + 9)
    c = dict(case, body="sphere", floor=False, walls="bb")
    setup = _setup(c, seed)
    dev = _device()
    z, y, x = torch.meshgrid(*(torch.arange(n, device=dev, dtype=torch.float64) for n in (c["nz"], c["ny"], c["nx"])),
                             indexing="ij")
    m = torch.ones((c["nz"], c["ny"], c["nx"], 4), dtype=torch.float64, device=dev)
    for k in range(3):
        a, b, d = r.uniform(1, 3, 3) * 2 * np.pi
        ph = r.uniform(0, 6, 3)
        m[..., 1 + k] = (0.05 if k == 0 else 0.0) + 0.02 * torch.sin(a * x / c["nx"] + ph[0]) * torch.cos(
            b * y / c["ny"] + ph[1]) * torch.sin(d * z / c["nz"] + ph[2])
    return c, setup, m.float().cpu().numpy()


def _particles(case, seed):
    r = np.random.default_rng(seed + 13)
    rec = np.zeros((case["particles"], 8), np.float32)
    hi = np.array([case["nx"], case["ny"], case["nz"]]) - 3.0
    rec[:, :3] = r.uniform(2.0, hi, (case["particles"], 3))
    rec[:, 4:7] = rec[:, :3]
    return rec


def _rake(case):
    return (4.0, 0.2 * case["ny"], 0.8 * case["ny"], 0.2 * case["nz"], 0.8 * case["nz"])


H = 8.0         # solver steps between frames
FRAMES = 96     # frames that have passed before the measured one


# ---------------------------------------------------------------- prepare, run
def _solver(case, setup, grid):
    s = GpuSolver.create((case["nx"], case["ny"], case["nz"]), grid, SolverParams(
        tau0=setup["tau0"], u_in=setup["u"], les=case["les"], operator=case["operator"], walls=case["walls"],
        precision=case.get("precision", "f32"), lateral=case["lateral"]))
    if isinstance(s, Exception):
        raise s
    return s


def _macros(s, shape):
    return _view(s, s.buffers()[0], shape + (4,), "<f4")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        setup = _setup(case, seed)
        s = _solver(case, setup, _grid(case, setup))
        st = {"kind": kind, "solver": s, "steps": case["steps"], "field": None}
        if case["closure"]:
            st["closure"] = c = Closure(1)
            c.params = _params(seed)
            c.attach(s)
        s.step(case["warm"])
        st["macros"] = _macros(s, (case["nz"], case["ny"], case["nx"]))
        if case["field"]:
            st["field"] = np.zeros((s.cells, 4), np.float32)  # the caller's buffer, kept between readouts
        return st
    if kind == "batch":
        members, views = [], []
        for t, setup in _tunnels(case, seed):
            members.append(_solver(dict(t, precision=case["precision"]), setup, _grid(t, setup)))
            views.append(_macros(members[-1], (t["nz"], t["ny"], t["nx"])))
        b = Batch(members)
        b.tune(2)
        b.reset()
        return {"kind": kind, "batch": b, "members": members, "macros": views, "steps": case["steps"]}
    if kind == "train":
        c = Closure(1)
        c.set_dataset(*_samples(case, seed))
        c.params = _params(seed)
        return {"kind": kind, "closure": c, "steps": case["steps"], "batch": case["batch"], "seed": seed % 1000}
    if kind in ("load", "links"):
        return {"kind": kind, "mesh": _mesh(case, seed), "layout": (case["nx"], case["ny"], case["nz"]),
                "floor": case["floor"], "solver": None}
    c, setup, field = _field(case, seed)
    s = _solver(dict(c, les=False, operator="trt", lateral="periodic"), setup, _grid(c, setup))
    s.write_macros(field)
    p = Particles(s, _particles(case, seed), seed % 4096, (2.0, 2.0, case["ny"] - 3.0, case["nz"] - 3.0),
                  (case["ny"] / 8, case["nz"] / 8))
    k = Streaks(s, case["rake"], case["rake"], case["slots"], _rake(case))
    for t in range(FRAMES):
        p.update(H)
        k.advance(H, t, t % 2 == 0)
    return {"kind": kind, "solver": s, "particles": p, "streaks": k, "frame": FRAMES}


def run(st):
    kind = st["kind"]
    if kind == "step":
        s = st["solver"]
        s.step(st["steps"], True)
        s.encode_force()
        f = s.read_force()
        # the drag carries the populations' binary32 accuracy
        out = {"force": np.array([f.fx, f.fy, f.fz], np.float32)}
        out["macros"] = st["macros"] if st["field"] is None else s.macros(out=st["field"])
        return out
    if kind == "batch":
        st["batch"].step(st["steps"], True)
        for s in st["members"]:
            s.encode_force()
        forces = [s.read_force() for s in st["members"]]
        return {"macros": st["macros"], "force": np.array([(f.fx, f.fy, f.fz) for f in forces], np.float32)}
    if kind == "train":
        c = st["closure"]
        first, last = c.train(st["steps"], st["batch"], 1e-3, st["seed"])
        return {"params": c.params, "loss": np.array([first, last], np.float32)}
    if kind == "load":
        if st["solver"] is not None:
            st["solver"].destroy()
        g = voxelize(st["mesh"], None, st["layout"], st["floor"])
        s = st["solver"] = GpuSolver.create(st["layout"], g, SolverParams(tau0=0.56, u_in=0.05, les=True,
                                                                          operator="reg", precision="f16"))
        macros, flags, _ = s.buffers()
        nx, ny, nz = st["layout"]
        return {"flags": _view(s, flags, (nz, ny, nx), "<i4"), "macros": _view(s, macros, (nz, ny, nx, 4), "<f4"),
                "solid": g.solid_cells, "frontal": g.frontal_cells, "watertight": g.watertight}
    if kind == "links":
        g = voxelize(st["mesh"], None, st["layout"], st["floor"], link_fractions=True)
        n = g.cells
        return {"flags": g.geometry[:2 * n].view(np.int32), "fractions": g.geometry[2 * n:].view(np.float32),
                "boundary": g.boundary_cells.view(np.int32), "missed": g.missed_links, "solid": g.solid_cells}
    t = st["frame"]
    st["frame"] = t + 1
    st["particles"].update(H)
    st["streaks"].advance(H, t, t % 2 == 0)
    puffs, _ = st["streaks"].read()
    return {"particles": st["particles"].read(), "puffs": puffs}


def work(case):
    """Each step reads and writes every population of every cell once (about 400 operations a cell); macros and
    read-back fields are written once; a training step reads its minibatch and takes three passes over the
    network's products; a mesh is read once and the geometry written once."""
    kind = case["kind"]
    if kind in ("step", "batch"):
        sizes = [(case["nx"], case["ny"], case["nz"])] if kind == "step" else [
            (t["nx"], t["ny"], t["nz"]) for t, _ in _tunnels(case, 0)]
        cells = sum(a * b * c for a, b, c in sizes)
        per = 400 + (2 * (9 * 32 + 32 * 32 + 32) if case.get("closure") else 0)
        return {"bytes": cells * (2 * 19 * ELEM[case["precision"]] * case["steps"] + 16), "flops": cells * per * case["steps"]}
    if kind == "train":
        n = case["steps"] * case["batch"]
        return {"bytes": n * 40, "flops": n * 6 * (9 * 32 + 32 * 32 + 32)}
    if kind in ("load", "links"):
        cells = case["nx"] * case["ny"] * case["nz"]
        tri = 2 * case["lon"] * (case["lat"] - 1)
        return {"bytes": 36 * tri + cells * (4 + 4 + (16 + 19 * 2 if kind == "load" else 0)), "flops": 200 * tri}
    puffs = case["rake"] ** 2 * case["slots"]
    live = case["rake"] ** 2 * min(case["slots"], FRAMES // 2)
    return {"bytes": 64 * case["particles"] + 20 * puffs + 16 * live, "flops": 150 * case["particles"] + 500 * live}


# ---------------------------------------------------------------- the same in 64 bits, plain torch
class _Flow:
    """The lattice step in binary64 on whole arrays: pull streaming, EQ faces, TRT or regularized collision,
    Smagorinsky, the wall model, halfway or interpolated walls, free-slip faces, the closure's network."""

    def __init__(self, case, setup, params=None):
        self.dev = dev = _device()
        self.case, self.u = case, setup["u"]
        nx, ny, nz = self.shape = case["nx"], case["ny"], case["nz"]
        flags, _ = _flags(case, setup, dev)
        f = flags.reshape(-1)
        n = self.n = f.numel()
        self.kind = kind = f & 7
        self.wall = (kind >= SOLID) & (kind <= FLOOR)
        self.eq = torch.nonzero(kind == EQ).reshape(-1)
        self.C = torch.tensor(C19, dtype=torch.float64, device=dev).T.contiguous()
        self.W = torch.tensor(W19, dtype=torch.float64, device=dev)[:, None]
        cx, cy, cz = self.C
        self.Q = torch.stack([cx * cx, cy * cy, cz * cz, cx * cy, cx * cz, cy * cz])
        nu = float(np.float32((float(np.float32(setup["tau0"])) - 0.5) / 3))
        self.nu, self.tau0, self.cs = nu, 3 * nu + 0.5, 18 * math.sqrt(2) * 0.01
        cell = torch.arange(n, device=dev)
        x, y, z = cell % nx, cell // nx % ny, cell // (nx * ny)
        self.src = torch.empty((19, n), dtype=torch.int64, device=dev)
        slip = case["lateral"] == "free-slip"
        for i, (a, b, c) in enumerate(C19):
            sx, sy, sz = (x - a) % nx, y - b, z - c
            ry, rz = (sy < 0) | (sy >= ny), (sz < 0) | (sz >= nz)
            if slip:
                k = torch.full_like(cell, i)
                my, mz, mm = (C19.index((a, -b if p else b, -c if q else c)) for p, q in ((1, 0), (0, 1), (1, 1)))
                k = torch.where(ry & rz, mm, torch.where(ry, my, torch.where(rz, mz, k)))
                s = sx + nx * (torch.where(ry, y, sy) + ny * torch.where(rz, z, sz))
            else:
                k, s = i, sx + nx * (sy % ny + ny * (sz % nz))
            at = k * n + s
            if i:
                at = torch.where((f >> (3 + i)) & 1 == 1, OPP[i] * n + cell, at)
            self.src[i] = at
        # the wall links, cell by cell
        self.wc, self.bits, q = _fractions(case, setup, flags)
        self.q = torch.full(self.bits.shape, 0.5, dtype=torch.float64, device=dev)
        self.q[self.bits] = q.double()
        d = torch.tensor([a + nx * (b + ny * c) for a, b, c in C19[1:]], device=dev)
        wx, wy, wz = (v[self.wc][:, None] for v in (x, y, z))
        step = torch.tensor(C19[1:], device=dev)
        pull = (wx - step[:, 0]) % nx + nx * ((wy - step[:, 1]) % ny + ny * ((wz - step[:, 2]) % nz))
        ahead = (wx + step[:, 0]) % nx + nx * ((wy + step[:, 1]) % ny + ny * ((wz + step[:, 2]) % nz))
        self.body = self.bits & (kind[pull] == SOLID)
        self.ahead, self.ahead_fluid = ahead, kind[ahead] == FLUID
        self.opp = torch.tensor(OPP[1:], device=dev)
        del d
        rows = torch.arange(ny * nz, device=dev) * nx
        self.out_cell, self.up_cell = rows + nx - 1, rows + nx - 2
        self.params = params
        if params is not None:
            dist = torch.where(self.wall, 0.0, 255.0).double().reshape(nz, ny, nx)
            for _ in range(8):
                best = dist.clone()
                best[:, :, 1:] = torch.minimum(best[:, :, 1:], dist[:, :, :-1] + 1)
                best[:, :, :-1] = torch.minimum(best[:, :, :-1], dist[:, :, 1:] + 1)
                for ax in (0, 1):
                    for sh in (1, -1):
                        best = torch.minimum(best, torch.roll(dist, sh, ax) + 1)
                dist = best
            self.dist = torch.clamp(dist.reshape(-1), max=8.0)
            self.plain = (f == FLUID)
        u = torch.zeros((3, n), dtype=torch.float64, device=dev)
        u[0] = torch.where(self.wall, 0.0, self.u)
        self.P = self.geq(torch.zeros(n, dtype=torch.float64, device=dev), u)
        self.P[:, self.wall] = 0.0
        self.force = [self.momentum(), self.momentum()]
        self.macros = torch.cat([torch.ones((1, n), dtype=torch.float64, device=dev), u])

    def geq(self, rd, u):
        cu = self.C.T @ u
        return self.W * (rd + (1 + rd) * (3 * cu + 4.5 * cu * cu - 1.5 * (u * u).sum(0)))

    def link_values(self):
        """f* reflected and the wall value of every link of the present state."""
        P, w = self.P, self.wc[:, None]
        refl = P[self.opp[None, :], w]
        if self.case["walls"] != "bouzidi":
            return refl, refl
        q = self.q
        low = torch.where(self.ahead_fluid, 2 * q * refl + (1 - 2 * q) * P[self.opp[None, :], self.ahead], refl)
        i = torch.arange(1, 19, device=self.dev)
        high = (refl + (2 * q - 1) * P[i[None, :], w]) / (2 * q)
        return refl, torch.where(q == 0.5, refl, torch.where(q < 0.5, low, high))

    def momentum(self):
        refl, val = self.link_values()
        t = torch.where(self.body, refl + val, 0.0).sum(0)
        return -(self.C[:, 1:] @ t)

    def stress(self, v):
        return self.Q @ v

    def tau(self, pi, rho):
        if not self.case["les"]:
            return torch.full_like(rho, self.tau0)
        q = (pi[:3] ** 2).sum(0) + 2 * (pi[3:] ** 2).sum(0)
        return 0.5 * (self.tau0 + torch.sqrt(self.tau0 ** 2 + self.cs * torch.sqrt(q) / rho))

    def project(self, pi):
        w = torch.tensor([1, 1, 1, 2, 2, 2], dtype=torch.float64, device=self.dev)[:, None]
        return self.Q.T @ (w * pi) - (pi[0] + pi[1] + pi[2]) / 3

    def network(self, tau, pi, rho, u):
        s = -1.5 / (rho * tau) * pi
        ss = (s[:3] ** 2).sum(0) + 2 * (s[3:] ** 2).sum(0)
        off = 2 * (s[3:] ** 2).sum(0)
        a, b, c, d, e, f = s
        t3 = a ** 3 + b ** 3 + c ** 3 + 3 * ((a + b) * d * d + (a + c) * e * e + (b + c) * f * f) + 6 * d * e * f
        x = torch.stack([100 * torch.sqrt(2 * ss), t3 / (ss * torch.sqrt(ss) + 1e-30), off / (ss + 1e-30),
                         torch.sqrt((u * u).sum(0)) / self.u, u[0] / self.u, 0.1 * (rho - 1) / self.u ** 2,
                         self.dist / 8, 10 * (tau - self.tau0) / 3 / self.nu, torch.full_like(rho, 200 * self.nu)])
        w1, b1, w2, b2, w3, b3 = _unpack(torch.tensor(self.params, device=self.dev).double())
        h = torch.tanh(w2 @ torch.tanh(w1 @ x + b1[:, None]) + b2[:, None])
        c = w3 @ h + b3
        return torch.where(self.plain, self.tau0 + (tau - self.tau0) * torch.clamp(1 + c, min=0.0), tau)

    def collide(self, g, e, pi, tau):
        om = 1 / tau
        if self.case["operator"] == "reg":
            return e + (1 - om) * 4.5 * self.W * self.project(pi)
        om_m = 1 / (0.1875 / (tau - 0.5) + 0.5)
        j = torch.tensor(OPP, device=self.dev)
        even, odd = (g + g[j] - e - e[j]) * (0.5 * om), (g - g[j] - e + e[j]) * (0.5 * om_m)
        return g - even - odd

    def wall_model(self, e, rho, u, plain):
        """The LES wall cells' post-collision state (columns: the wall-link cells)."""
        b = torch.zeros((19, len(self.wc)), dtype=torch.float64, device=self.dev)
        b[1:] = self.bits.T.double()
        wb = self.W * b
        normal = self.C @ wb
        ln = torch.sqrt((normal ** 2).sum(0))
        un = torch.where(ln > 1e-3, normal / torch.clamp(ln, min=1e-30), 0.0)
        slip = u - (u * un).sum(0) * un
        speed = torch.sqrt((slip ** 2).sum(0))
        t = slip / torch.clamp(speed, min=1e-30)
        visc = torch.sqrt(self.nu * speed / 0.5)
        power = (speed * (self.nu / 0.5) ** (1 / 7) / 8.3) ** (1 / (1 + 1 / 7))
        ut = torch.where(0.5 * visc / self.nu <= 11.81, visc, power)
        shear = 6 * wb.sum(0) * rho * ut * ut
        j = torch.tensor(OPP, device=self.dev)
        bj = b[j]  # flagged by the opposite direction
        along = (self.C.T @ t) * bj
        flux = (2 * along * (e + self.W)).sum(0)
        sj = 9 * self.W * along
        third = torch.tensor([1, 1, 1, 0, 0, 0], dtype=torch.float64, device=self.dev)[:, None] / 3
        B = (self.Q @ sj) - third * sj.sum(0)
        norm = (B[:3] ** 2).sum(0) + 2 * (B[3:] ** 2).sum(0)
        post = e + 4.5 * (shear - flux) / torch.clamp(norm, min=1e-30) * self.W * self.project(B)
        keep = (speed < 1e-7) | (norm < 0.05) | ((post + self.W) < 0).any(0)
        return torch.where(keep, plain, post)

    def step(self):
        P = self.P
        g = P.reshape(-1)[self.src]
        if self.case["walls"] == "bouzidi":
            _, val = self.link_values()
            rows, cols = torch.nonzero(self.bits, as_tuple=True)
            g[cols + 1, self.wc[rows]] = val[self.bits]
        up = P[:, self.up_cell]
        mass = 1 + up.sum(0)
        outlet = torch.where(self.wall[self.up_cell], 0.0, (self.C @ up) / mass)
        rd = g.sum(0)
        u = (self.C @ g) / (1 + rd)
        rd[self.eq] = 0.0
        u[:, self.eq] = 0.0
        u[0, self.eq] = self.u
        o = self.kind[self.out_cell] == EQ
        u[:, self.out_cell[o]] = outlet[:, o]
        rho = 1 + rd
        e = self.geq(rd, u)
        pi = self.stress(g - e) if self.case["les"] or self.case["operator"] == "reg" else None
        tau = self.tau(pi, rho)
        if self.params is not None:
            tau = self.network(tau, pi, rho, u)
        post = self.collide(g, e, pi, tau)
        if self.case["les"]:
            post[:, self.wc] = self.wall_model(e[:, self.wc], rho[self.wc], u[:, self.wc], post[:, self.wc])
        post[:, self.eq] = e[:, self.eq]
        post[:, self.wall] = 0.0
        self.P = post
        self.force = [self.force[1], self.momentum()]
        rho[self.wall] = 1.0
        u[:, self.wall] = 0.0
        self.macros = torch.cat([rho[None], u])

    def outputs(self, shaped=True):
        f = (0.5 * (self.force[0] + self.force[1])).cpu().numpy()
        m = self.macros.T.contiguous()
        nx, ny, nz = self.shape
        return f, m.reshape(nz, ny, nx, 4) if shaped else m.cpu().numpy()


def _unpack(w):
    return w[:288].reshape(32, 9), w[288:320], w[320:1344].reshape(32, 32), w[1344:1376], w[1376:1408], w[1408]


def _mix64(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _exact_train(case, seed):
    dev = _device()

    def b16(t):
        return t.float().bfloat16().double()

    X, Y = (torch.tensor(a, device=dev) for a in _samples(case, seed))
    w = torch.tensor(_params(seed), device=dev).double()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    losses = []
    for t in range(case["steps"]):
        with np.errstate(over="ignore"):
            at = _mix64(np.uint64(seed % 1000) + (np.uint64(t) << np.uint64(32)) + np.arange(case["batch"], dtype=np.uint64))
        at = torch.tensor((at % np.uint64(case["samples"])).astype(np.int64), device=dev)
        x, y = b16(X[at]), Y[at].double()
        w1, b1, w2, b2, w3, b3 = _unpack(w)
        r1, r2, r3 = b16(w1), b16(w2), b16(w3)
        h1 = b16(torch.tanh(x @ r1.T + b1))
        h2 = b16(torch.tanh(h1 @ r2.T + b2))
        err = h2 @ r3 + b3 - y
        losses.append(float((err * err).mean()))
        d3 = 2 * err / case["batch"]
        d2 = d3[:, None] * r3 * (1 - h2 * h2)
        d1 = (d2 @ r2) * (1 - h1 * h1)
        g = torch.cat([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), d3 @ h2, d3.sum()[None]])
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** (t + 1))) / (torch.sqrt(v / (1 - 0.999 ** (t + 1))) + 1e-8)
    return {"params": w.cpu().numpy(), "loss": np.array([losses[0], losses[-1]])}


def _exact_tracers(case, seed):
    dev = _device()
    c, setup, field = _field(case, seed)
    fluid = (_flags(c, setup, dev)[0].reshape(-1) & 7) == FLUID
    nx, ny, nz = size = (c["nx"], c["ny"], c["nz"])
    top = torch.tensor(size, device=dev)
    M = torch.tensor(field, device=dev).double().reshape(-1, 4)[:, 1:]

    def vel(p):
        q = torch.minimum(torch.clamp(p, min=0.0), (top - 1).double())
        lo = torch.floor(q).long()
        hi = torch.minimum(lo + 1, top - 1)
        w = q - lo
        out = 0.0
        for k in range(8):
            b = [(hi if k >> a & 1 else lo)[:, a] for a in range(3)]
            f = 1.0
            for a in range(3):
                f = f * (w[:, a] if k >> a & 1 else 1 - w[:, a])
            out = out + f[:, None] * M[b[0] + nx * (b[1] + ny * b[2])]
        return out

    def cell_fluid(p):
        k = torch.minimum(torch.clamp(torch.floor(p + 0.5), min=0).long(), top - 1)
        return fluid[k[:, 0] + nx * (k[:, 1] + ny * k[:, 2])]

    def h32(x):
        x = (x ^ (x >> 16)) * 0x7FEB352D & 0xFFFFFFFF
        x = (x ^ (x >> 15)) * 0x846CA68B & 0xFFFFFFFF
        return x ^ (x >> 16)

    rec = torch.tensor(_particles(case, seed), device=dev).double()
    ident = torch.arange(len(rec), device=dev)
    lo = torch.tensor([2.0, 2.0], device=dev).double()
    hi = torch.tensor([ny - 3.0, nz - 3.0], device=dev).double()
    ry = rz = case["rake"]
    rake = _rake(case)
    th = torch.arange(ry * rz, device=dev)
    ty, tz = (th % ry).double() / (max(ry, 2) - 1), (th // ry).double() / (max(rz, 2) - 1)
    nozzle = torch.stack([torch.full_like(ty, rake[0]), rake[1] + (rake[2] - rake[1]) * ty,
                          rake[3] + (rake[4] - rake[3]) * tz, torch.ones_like(ty)], 1)
    puffs = torch.zeros((ry * rz, case["slots"], 4), dtype=torch.float64, device=dev)

    def open3(p):
        return (p >= 0).all(1) & (p <= (top - 1)).all(1) & cell_fluid(p)

    for t in range(FRAMES + 1):
        pos, age, gen = rec[:, :3], rec[:, 3] + 1, rec[:, 7]
        d = vel(pos) * H
        q = pos + d / torch.clamp(torch.sqrt((d * d).sum(1, keepdim=True)), min=1.0)
        inside = (q >= 0).all(1) & (q < (top - 1)).all(1) & cell_fluid(q)
        again = (q[:, 0] >= nx - 2) | ~inside | (age > 4000)
        h = h32((ident + seed % 4096 + (gen + 1).long() * 0x9E3779B9) & 0xFFFFFFFF)
        r = torch.stack([(h >> 8).double(), (h32(h) >> 8).double()], 1) / 16777216.0
        at = lo * (1 - r) + hi * r
        born = torch.cat([torch.full_like(at[:, :1], 2.0), at], 1)
        ok = (born < (top - 1)).all(1) & cell_fluid(born)
        born[~ok, 1:] = torch.tensor([ny / 8, nz / 8], device=dev).double()
        new = torch.where(again[:, None], born, q)
        rec = torch.cat([new, torch.where(again, 0.0, age)[:, None], torch.where(again[:, None], born, pos),
                         torch.where(again, gen + 1, gen)[:, None]], 1)
        # streaklines
        slot = t % case["slots"] if t % 2 == 0 else -1
        flat = puffs.reshape(-1, 4)
        live = flat[:, 3] != 0
        if slot >= 0:
            released = torch.zeros((ry * rz, case["slots"]), dtype=torch.bool, device=dev)
            released[:, slot] = True
            live &= ~released.reshape(-1)
        s = flat[live]
        p, dens = s[:, :3].clone(), s[:, 3].clone()
        count = torch.clamp(torch.ceil(2 * H * torch.sqrt((vel(p) ** 2).sum(1))), 1, 16)
        for k in range(int(count.max()) if len(s) else 0):
            on = (k < count) & (p[:, 0] >= 0)
            hh = (H / count)[:, None]
            d = hh * vel(p + 0.5 * hh * vel(p))
            nxt = p + d / torch.clamp(torch.sqrt((d * d).sum(1, keepdim=True)), min=1.0)
            hit = ~open3(nxt)
            left, went = hit.clone(), nxt.clone()
            for keep in ((1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
                cand = torch.where(torch.tensor(keep, device=dev).bool(), nxt, p)
                take = left & open3(cand)
                went[take] = cand[take]
                left &= ~take
            went[left] = -1.0
            dens = torch.where(on & hit, dens * 0.85 ** (1 / count), dens)
            p = torch.where(on[:, None], went, p)
        alive = (p[:, 0] >= 0) & (p[:, 0] < nx - 2) & (dens > 0.02)
        flat = flat.clone()
        flat[live] = torch.cat([p, torch.where(alive, dens, 0.0)[:, None]], 1)
        puffs = flat.reshape(ry * rz, case["slots"], 4)
        if slot >= 0:
            puffs[:, slot] = nozzle
    return {"particles": rec, "puffs": puffs.reshape(-1, 4)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        flow = _Flow(case, _setup(case, seed), _params(seed) if case["closure"] else None)
        for _ in range(case["warm"] + case["steps"]):
            flow.step()
        f, m = flow.outputs(not case["field"])
        return {"force": f, "macros": m}
    if kind == "batch":
        macros, force = [], []
        for t, setup in _tunnels(case, seed):
            flow = _Flow(t, setup)
            for _ in range(case["steps"]):
                flow.step()
            f, m = flow.outputs()
            macros.append(m)
            force.append(f)
        return {"macros": macros, "force": np.array(force)}
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "tracers":
        return _exact_tracers(case, seed)
    return None  # whole numbers, and fractions of a triangle mesh
