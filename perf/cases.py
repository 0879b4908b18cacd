"""What a user of the water simulation has it do, as cases that can be timed and compared.

A case is one frame of a program that owns its particles: it hands them to a context (`upload`),
steps it (`step`, with the emitter before each step where the scene has one), and takes the new
state, into device arrays for a renderer (`export_positions`, `splat`) or into host arrays
(`download`). The grid build for callers with their own memory (`sph_grid_build_noalloc`) is a call
of its own. Fields of a case:

  kind      frame | grid
  n         particles (frame with scenes > 1: of all scenes together, about)
  scenes    independent scenes of the batch
  state     rest (the dam break's lattice, at rest), fallen (the collapsed column some hundred
            steps later: packed towards the floor, moving) or fountain (a plume over a disc emitter)
  form      plain | mixed | f64
  cells     0: a context as it is created; 2: cells of h/2 set by the caller, with the force
            variant that the autotuner picks for large collapsed columns
  steps     steps between the upload and the result
  out       device | host (positions, velocities, densities, pressures) | image (device, and a splat)
  emit      particles the disc emitter adds before each step
  obstacles axis-aligned box obstacles in the scene
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "gmu-water-simulation_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

H = float(np.float32(0.0457))  # smoothing length; the lattice spacing is half of it
SPACING = H / 2
GRAVITY = (0.0, -9.81, 0.0)
FORCES_LARGE = 10              # force variant of large collapsed columns on cells of h/2
IMAGE = (640, 360)             # splat of a preview window


def _frame(name, n, state, form="plain", cells=0, steps=1, out="device", scenes=1, emit=0, obstacles=0):
    c = {"kind": "frame", "n": n, "scenes": scenes, "state": state, "form": form, "cells": cells, "steps": steps,
         "out": out, "emit": emit, "obstacles": obstacles}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference's default scene (0.4 m box), one step, everything back on the host as its
        # front end wants it: the smallest call, bound by launches and round trips
        _frame("default_scene_1620", 1620, "rest", out="host"),
        # the 20^3 dam break kept on the device for a stretch of steps: replayed graphs of a small scene
        _frame("dam_8000_40_steps", 8000, "rest", steps=40),
        # an interactive scene: a few steps a frame, then a preview image and the vertex buffer
        _frame("preview_61000", 61_000, "fallen", steps=3, out="image"),
        # the fountain: a plume over a disc emitter that adds particles before every step, mixed form
        _frame("fountain_90000_mixed", 90_000, "fountain", form="mixed", steps=3, emit=2000),
        # the 100^3 dam break at its start, in a context as it is created
        _frame("dam_1m_start", 1_000_000, "rest", steps=2),
        # the same size collapsed, on the settings that the tuner picks for it
        _frame("dam_1m_fallen_half_cells", 1_000_000, "fallen", cells=2, steps=2),
        # mixed precision on the same
        _frame("dam_1m_fallen_mixed", 1_000_000, "fallen", form="mixed", cells=2, steps=2),
        # a batch of independent scenes of uneven sizes
        _frame("batch_48_scenes", 700_000, "fallen", steps=2, scenes=48),
        # a large scene with box obstacles
        _frame("dam_4m_obstacles", 4_000_000, "fallen", cells=2, steps=1, obstacles=8),
        # the FP64 run that the other forms are checked against, read back in double
        _frame("check_f64_50000", 50_000, "fallen", form="f64", steps=1, out="host"),
        # the grid build for a caller's own memory: ordinary and near its limits
        {"name": "grid_build_30011", "kind": "grid", "n": 30_011},
        {"name": "grid_build_1000003", "kind": "grid", "n": 1_000_003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["rest", "fallen", "fallen", "half", "half", "mixed", "fountain", "batch", "f64", "grid"])
    if what == "rest":
        n = _log_int(rng, 1000, 1_500_000)
        return _frame(None, n, "rest", steps=rng.randint(1, 40) if n < 50_000 else rng.randint(1, 3),
                      out=rng.choice(["device", "host"]) if n < 50_000 else "device")
    if what == "fallen":
        n = _log_int(rng, 2000, 1_500_000)
        return _frame(None, n, "fallen", steps=rng.randint(1, 3), out=rng.choice(["device", "image"]),
                      obstacles=rng.choice([0, 0, 3]))
    if what == "half":
        return _frame(None, _log_int(rng, 200_000, 2_500_000), "fallen", cells=2, steps=rng.randint(1, 2),
                      obstacles=rng.choice([0, 8]))
    if what == "mixed":
        return _frame(None, _log_int(rng, 5000, 2_000_000), "fallen", form="mixed", cells=rng.choice([0, 2]),
                      steps=rng.randint(1, 2))
    if what == "fountain":
        return _frame(None, _log_int(rng, 10_000, 400_000), "fountain", form=rng.choice(["mixed", "plain"]),
                      steps=rng.randint(1, 4), emit=rng.randint(500, 2500))
    if what == "batch":
        s = rng.randint(3, 96)
        return _frame(None, _log_int(rng, 4000, 24_000) * s, "fallen", steps=rng.randint(1, 3), scenes=s)
    if what == "f64":
        return _frame(None, _log_int(rng, 2000, 120_000), rng.choice(["rest", "fallen"]), form="f64",
                      steps=rng.randint(1, 2), out="host")
    return {"kind": "grid", "n": _log_int(rng, 2000, 1_040_000)}


# ---------------------------------------------------------------------------- scenes
def _sizes(case):
    """Particles of each scene: uneven by up to a factor of about 8, the same for every seed."""
    s = case.get("scenes", 1)
    if s == 1:
        return [case["n"]]
    w = np.exp(np.random.RandomState(17 + s).uniform(0.0, 2.0, s))
    return [max(64, int(v)) for v in case["n"] * w / w.sum()]


def _dims(n, state):
    """Lattice of at least n sites: the dam break's cube, or the wide and low collapsed column."""
    if state == "rest":
        a = max(2, math.ceil(n ** (1 / 3) - 1e-9))
        return a, a, max(1, math.ceil(n / (a * a)))
    a = max(2, math.ceil(n ** (1 / 3) - 1e-9))
    nx, ny = 2 * a, max(2, a // 2)
    return nx, ny, max(1, math.ceil(n / (nx * ny)))


def _box(n, state):
    if state == "fountain":
        return 2.0, 2.0, 2.0
    nx, ny, nz = _dims(n, state)
    if n == 1620 and state == "rest":
        return 0.4, 0.4, 0.4
    if state == "rest":  # the column fills about the left half of its box, which is twice as high
        return 2.19 * nx * SPACING, 2.19 * ny * SPACING, 1.09 * nz * SPACING
    return 1.06 * nx * SPACING, 3.0 * ny * SPACING, 1.03 * nz * SPACING + 0.01


def _scene(n, state, gen):
    """(positions, velocities or None) of n particles, float32 on the device."""
    dev = gen.device
    rand = lambda *s: torch.rand(*s, generator=gen, device=dev, dtype=torch.float32)    # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=gen, device=dev, dtype=torch.float32)  # noqa: E731
    box = torch.tensor(_box(n, state), device=dev)
    if state == "fountain":
        # a tenth still rises and falls over the disc, the rest has spread over the floor
        c = torch.tensor((0.0, -1.0, 0.0), device=dev)
        t = 1.05 * rand(n, 1)
        ang, rad = 2 * math.pi * rand(n), 0.05 * rand(n).sqrt()
        disc = torch.stack((rad * ang.cos(), torch.zeros_like(rad), rad * ang.sin()), 1)
        v0 = torch.tensor((0.0, 5.0, 0.0), device=dev) + 0.2 * randn(n, 3)
        g = torch.tensor(GRAVITY, device=dev)
        pos, vel = c + disc + v0 * t + 0.5 * g * t * t, v0 + g * t
        pool = torch.arange(n, device=dev) >= n // 10
        r = 0.85 * rand(n).sqrt() * min(1.0, (n / 100_000) ** 0.5)
        floor = torch.stack((r * ang.cos(), -0.99 + 0.09 * rand(n) * (1.1 - r), r * ang.sin()), 1)
        pos = torch.where(pool[:, None], floor, pos)
        pos[:, 1].clamp_(min=-0.995)
        vel = torch.where(pool[:, None], 0.6 * randn(n, 3), vel)
        return pos.contiguous(), vel.contiguous()
    nx, ny, nz = _dims(n, state)
    k = torch.arange(n, device=dev)
    ijk = torch.stack((k % nx, (k // nx) % ny, k // (nx * ny)), 1).to(torch.float32)
    if state == "rest":  # 1% jitter, at the min corner
        pos = -box / 2 + SPACING * (ijk + 0.5 + 0.01 * (2 * rand(n, 3) - 1))
        return pos.contiguous(), None
    # collapsed: heights packed towards the floor (1.75 times the lattice's density on average, more
    # at the floor), strong disorder, a sloshing motion with noise
    u = (ijk + 0.5 + 0.35 * (2 * rand(n, 3) - 1)) * SPACING
    height = ny * SPACING / 1.75
    u[:, 1] = height * (u[:, 1].clamp(min=0.0) / (ny * SPACING)) ** 1.3 + 0.004
    pos = -box / 2 + u + torch.tensor((0.01, 0.0, 0.005), device=dev)
    q = pos / box
    vel = 0.8 * randn(n, 3)
    vel[:, 0] += 1.5 * torch.sin(5.0 * q[:, 0]) + 0.5
    vel[:, 1] += -0.8 * torch.cos(4.0 * q[:, 0])
    vel[:, 2] += 0.7 * torch.sin(6.0 * q[:, 2])
    return pos.contiguous(), vel.contiguous()


def _obstacles(case):
    """Box obstacles in the downstream half of the scene, the same for every seed."""
    if not case.get("obstacles"):
        return None
    b = np.array(_box(case["n"], case["state"]))
    r = np.random.RandomState(23)
    out = []
    for _ in range(case["obstacles"]):
        size = r.uniform(0.05, 0.2, 3) * min(1.0, b.min())
        lo = np.array((0.0, -b[1] / 2, -b[2] / 2)) + r.uniform(0, 1, 3) * (b * (0.5, 0.15, 1.0) - size).clip(min=0)
        out.append(np.concatenate((lo, lo + size)))
    return np.array(out, np.float32)


def _grid_box(n):
    """A box of about eight cells per ten particles within the build's limit of 2^20 cells."""
    a = max(2, int((0.8 * n) ** (1 / 3)))
    return tuple(float(np.float32(v * H * 0.999)) for v in (a + 1, a, a))


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 1000)
    if case["kind"] == "grid":
        box = torch.tensor(_grid_box(case["n"]), device="cuda")
        # a cloud that is denser in its middle, some of it outside the box (clamped into its cells)
        u = torch.rand(case["n"], 3, generator=gen, device="cuda")
        v = torch.rand(case["n"], 3, generator=gen, device="cuda")
        return ((0.5 * (u + v) - 0.5) * 1.02 * box).contiguous(), None
    parts = [_scene(n, case["state"], gen) for n in _sizes(case)]
    pos = torch.cat([p for p, _ in parts])
    vel = None if parts[0][1] is None else torch.cat([v for _, v in parts])
    return pos, vel


def _pinned(t):
    if t is None:
        return None
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


# ---------------------------------------------------------------------------- the calls
EMITTER = ((0.0, -0.98, 0.0), 0.05, 5.0, 0.2)  # centre, radius, speed, sigma


def prepare(case, seed):
    import sphcuda

    if case["kind"] == "grid":
        pos, _ = _inputs(case, seed)
        box = _grid_box(case["n"])
        cells = int(np.prod([int(np.ceil(np.float32(b) / np.float32(0.0457))) for b in box]))
        i32 = dict(dtype=torch.int32, device="cuda")
        return {"case": case, "lib": sphcuda.load(), "xyz": pos, "box": (ctypes.c_float * 3)(*box),
                "cell": torch.empty(case["n"], **i32), "start": torch.empty(cells + 1, **i32),
                "order": torch.empty(case["n"], **i32)}
    pos, vel = _inputs(case, seed)
    sizes = _sizes(case)
    form = {"plain": sphcuda.SPH_PLAIN_F32, "mixed": sphcuda.SPH_MIXED, "f64": sphcuda.SPH_F64}[case["form"]]
    obs = _obstacles(case)
    total = pos.shape[0] + case["emit"] * case["steps"]
    ctx = sphcuda.SphContext([_box(n, case["state"]) for n in sizes], sizes if len(sizes) > 1 else [total],
                             precision=form, gravity=GRAVITY, obstacles=None if obs is None else [obs])
    if case["cells"]:
        ctx.set_cell_multiple(case["cells"])
        if case["form"] == "plain":
            ctx.set_variant(0, FORCES_LARGE)
    s = {"case": case, "ctx": ctx, "sizes": np.array(sizes, np.uint32), "n": total, "xyz": _pinned(pos),
         "vel": _pinned(vel)}
    if case["out"] == "host":
        s["xyz_np"], s["vel_np"] = s["xyz"].numpy(), None if vel is None else s["vel"].numpy()
    else:
        s["dev_xyz"] = torch.empty(total, 3, device="cuda")
        s["dev_vel"] = torch.empty(total, 3, device="cuda")
    if case["out"] == "image":
        s["count"] = torch.empty(IMAGE[1], IMAGE[0], dtype=torch.int32, device="cuda")
        s["depth"] = torch.empty(IMAGE[1], IMAGE[0], device="cuda")
    return s


def run(s):
    case = s["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "grid":
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        rc = s["lib"].sph_grid_build_noalloc(ptr(s["xyz"]), case["n"], s["box"], 0.0457, ptr(s["cell"]), ptr(s["start"]),
                                             ptr(s["order"]), ctypes.c_void_p(stream or None))
        if rc:
            raise RuntimeError(f"grid build: status {rc}")
        return {"cell": s["cell"], "start": s["start"], "order": s["order"]}
    ctx = s["ctx"]
    if case["out"] == "host":
        ctx.upload(s["xyz_np"], s["vel_np"], s["sizes"])
    else:
        ctx.upload_raw(s["xyz"].data_ptr(), None if s["vel"] is None else s["vel"].data_ptr(), s["sizes"])
    if case["emit"]:
        for k in range(case["steps"]):
            ctx.emit_fountain(0, 7, k, case["emit"], *EMITTER)
            ctx.step(1)
    else:
        ctx.step(case["steps"])
    if case["out"] == "host":
        return ctx.download()
    ctx.export_positions(s["dev_xyz"].data_ptr(), s["dev_vel"].data_ptr(), stream)
    out = {"pos": s["dev_xyz"], "vel": s["dev_vel"]}
    if case["out"] == "image":
        ctx.splat_raw(0, 2, IMAGE[0], IMAGE[1], s["count"].data_ptr(), s["depth"].data_ptr(), stream)
        out.update(count=s["count"], depth=s["depth"])
    return out


def work(case):
    n = case["n"] + case.get("emit", 0) * case.get("steps", 0)
    if case["kind"] == "grid":
        cells = float(np.prod([np.ceil(b / H) for b in _grid_box(n)]))
        return {"bytes": 12 * n + 8 * n + 4 * cells, "flops": 0}
    # accepted neighbours of a particle: the sphere's 4.19 h^3 at the state's density
    near = {"rest": 33, "fallen": 65, "fountain": 60}[case["state"]]
    real = 8 if case["form"] == "f64" else 4
    moved = (12 if case["state"] == "rest" else 24) * n + 6 * real * n
    moved += 2 * real * n if case["out"] == "host" else 0
    moved += 8 * IMAGE[0] * IMAGE[1] if case["out"] == "image" else 0
    # per accepted neighbour 9 operations of the density sum and 33 of the two force terms
    return {"bytes": moved, "flops": case["steps"] * n * near * 42}


# ---------------------------------------------------------------------------- in 64 bits
def exact(case, seed):
    """The same steps of the same method in 64-bit torch, from the cells of size h. None for runs
    so long that rounding decides them, and for the emitter's own particles."""
    if case["kind"] == "grid" or case["steps"] > 4 or case["emit"]:
        return None
    pos, vel = _inputs(case, seed)
    obs = _obstacles(case)
    x = pos.double()
    v = torch.zeros_like(x) if vel is None else vel.double()
    sizes = _sizes(case)
    boxes = torch.tensor([_box(n, case["state"]) for n in sizes], dtype=torch.float32, device=x.device)
    scene = torch.repeat_interleave(torch.arange(len(sizes), device=x.device), torch.tensor(sizes, device=x.device))
    rho = p = None
    for _ in range(case["steps"]):
        x, v, rho, p = _exact_step(x, v, scene, boxes, obs)
    if case["out"] == "host":
        return {"pos": x, "vel": v, "rho": rho, "p": p}
    out = {"pos": x, "vel": v}
    if case["out"] == "image":
        out.update(count=None, depth=None)
    return out


def _exact_step(x, v, scene, boxes, obs):
    f32 = lambda a: float(np.float32(a))  # noqa: E731
    h, mass, stiff, rho0, mu, dt = H, f32(0.02), 3.0, f32(998.29), 3.5, f32(0.01)
    poly6, spiky, visc = 315 / (64 * math.pi * h ** 9), -45 / (math.pi * h ** 6), 45 / (math.pi * h ** 6)
    res = torch.ceil(boxes / np.float32(0.0457)).long()
    cells = res.prod(1)
    base = torch.cumsum(cells, 0) - cells
    half = (boxes / 2).double()[scene]
    r, b = res[scene], base[scene]
    c = torch.minimum(torch.floor((x + half) / h).long().clamp(min=0), r - 1)
    cell = b + c[:, 0] + r[:, 0] * (c[:, 1] + r[:, 1] * c[:, 2])
    order = torch.argsort(cell, stable=True)
    start = torch.zeros(int(cells.sum()) + 1, dtype=torch.long, device=x.device)
    start[1:] = torch.cumsum(torch.bincount(cell, minlength=start.numel() - 1), 0)
    xs, vs, r, b, c = x[order], v[order], r[order], b[order], c[order]
    sp = [xs[:, a].contiguous() for a in range(3)]
    sv = [vs[:, a].contiguous() for a in range(3)]
    xl, xh = (c[:, 0] - 1).clamp(min=0), torch.minimum(c[:, 0] + 1, r[:, 0] - 1)

    def rows():
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                y, z = c[:, 1] + dy, c[:, 2] + dz
                ok = (y >= 0) & (y < r[:, 1]) & (z >= 0) & (z < r[:, 2])
                row = b + r[:, 0] * (y + r[:, 1] * z)
                jb = torch.where(ok, start[torch.where(ok, row + xl, 0)], 0)
                je = torch.where(ok, start[torch.where(ok, row + xh + 1, 0)], 0)
                at = torch.arange(jb.numel(), device=x.device)
                k, longest = 0, int((je - jb).max())
                while k < longest:
                    if k % 16 == 0:  # the particles whose row goes on
                        at = at[(jb + k < je)[at]]
                    j = jb[at] + k
                    yield at, torch.minimum(j, je[at] - 1), j < je[at]
                    k += 1

    acc = torch.zeros_like(sp[0])
    for i, j, go in rows():
        t = h * h - sum((sp[a][i] - sp[a][j]) ** 2 for a in range(3))
        acc.index_add_(0, i, torch.where(go & (t > 0), t, 0.0) ** 3)
    rho = mass * poly6 * acc
    p = stiff * (rho - rho0)
    q, inv = p / rho ** 2, 1 / rho
    fp, fv = [torch.zeros_like(acc) for _ in range(3)], [torch.zeros_like(acc) for _ in range(3)]
    for i, j, go in rows():
        d = [sp[a][i] - sp[a][j] for a in range(3)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        go = go & (r2 < h * h) & (i != j)
        near = torch.where(go, r2, 1.0).sqrt()
        w = torch.where(go, (q[i] + q[j]) * spiky * (h - near) ** 2 / near, 0.0)
        l = torch.where(go, visc * (h - near) * inv[j], 0.0)
        for a in range(3):
            fp[a].index_add_(0, i, w * d[a])
            fv[a].index_add_(0, i, l * (sv[a][j] - sv[a][i]))
    half = half[order]
    xn, vn = torch.empty_like(x), torch.empty_like(v)
    acc3 = []
    for a in range(3):
        f = (-mass * rho * fp[a] + mu * mass * fv[a] + f32(GRAVITY[a]) * rho) / rho
        for n_inv, wall in ((1.0, -half[:, a]), (-1.0, half[:, a])):
            d = (wall - sp[a]) * n_inv + 0.01
            f = f + torch.where(d > 0, 10000.0 * n_inv * d - 0.9 * sv[a], 0.0)
        acc3.append(f)
    for o in () if obs is None else obs.astype(np.float64):
        d = torch.stack([sp[a] - o[a] + 0.01 for a in range(3)] + [o[3 + a] - sp[a] + 0.01 for a in range(3)], 1)
        inside = (d > 0).all(1)
        face = d.argmin(1)
        for k in range(6):
            sgn, hit = -1.0 if k < 3 else 1.0, inside & (face == k)
            acc3[k % 3] = acc3[k % 3] + torch.where(hit, 10000.0 * sgn * d[:, k] - 0.9 * sv[k % 3], 0.0)
    for a in range(3):
        step = sv[a] * dt + acc3[a] * dt * dt
        xn[order, a], vn[order, a] = sp[a] + step, step / dt
    out = [torch.empty_like(rho) for _ in range(2)]
    out[0][order], out[1][order] = rho, p
    return xn, vn, out[0], out[1]
