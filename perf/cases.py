"""Workloads of the uniform-grid engine, as a user's program runs them through the public API.

What each kind of case stands for:

- "project": one pressure projection from a saved state (gravity, then ``project`` under the
  reference's stop rule and its default tolerance, 1e-6 1/s): the product's headline call. Sizes
  run from the interactive 64 x 64 to the benchmark's 2048 x 2048 dam break, with odd and ragged
  grids, obstacles, and all three precisions.
- "step": whole ``step`` calls (transport, gravity, surface tension, projection) in a simulation
  loop: semi-Lagrangian transport in the reference's gas air or in Dirichlet air, and the
  reference's conservative PLIC transport with surface tension as the serving workload has it.
  "whole" reads the complete state back to the host after the steps, as a host that draws or
  stores every frame does; otherwise the velocities are read in place on the device.
- "batch": one tick of many simulations on one GPU: every grid's substep is enqueued, then all
  grids are projected in one batched solve (what the serving loop does on each tick).
- "viscous": the implicit viscosity solve of a variable-viscosity liquid at the step's default
  tolerance, up to the benchmark's 4096 x 4096.

Every pass starts from the same saved state (``copyStateFrom``), so passes can be repeated.
Initial states are seeded synthetic data made on the GPU; velocities are rounded to FP32, so the
single-precision engine and the 64-bit evaluation below start from identical values.
"""
from __future__ import annotations

import math
import random

import torch

from fluidsim_b200 import FluidGrid, FluidGridState, ProjectionBatch

LIQUID, GAS, GRAVITY = 1000.0, 1.0, -9.8
TOLERANCE, MAX_ITERATIONS = 1e-6, 200


def listed():
    return [
        # The smallest interactive scene: launch count and latency decide.
        dict(name="project_64x64", kind="project", w=64, h=64, precision="fp32", obstacles=0, fill=0.5),
        # The reference's arithmetic (FP64) on an odd grid with obstacles.
        dict(name="project_131x97_fp64", kind="project", w=131, h=97, precision="fp64", obstacles=3, fill=0.6),
        # An ordinary grid.
        dict(name="project_512x512", kind="project", w=512, h=512, precision="fp32", obstacles=0, fill=0.5),
        # The reference's own largest published projection size, in mixed precision.
        dict(name="project_1920x1080_mixed", kind="project", w=1920, h=1080, precision="mixed", obstacles=0, fill=0.45),
        # The benchmark's projection.
        dict(name="project_2048x2048", kind="project", w=2048, h=2048, precision="fp32", obstacles=0, fill=0.5),
        # One tick of a serving class: uneven small and middle grids together.
        dict(name="batch_16_uneven", kind="batch", count=16, lo=64, hi=400, precision="fp32", obstacles=4),
        # A small simulation whose host draws every frame: two steps, then the whole state.
        dict(name="step_300x200_whole", kind="step", w=300, h=200, precision="fp32", transport="semi_lagrangian",
             air="gas", tension=False, obstacles=3, steps=2, whole=True),
        # The benchmark's stepping scene: 1024 x 1024 with obstacles.
        dict(name="step_1024x1024", kind="step", w=1024, h=1024, precision="fp32", transport="semi_lagrangian",
             air="gas", tension=False, obstacles=16, steps=1, whole=False),
        # Free-surface air on a ragged grid.
        dict(name="step_641x483_dirichlet", kind="step", w=641, h=483, precision="fp32", transport="semi_lagrangian",
             air="dirichlet", tension=False, obstacles=6, steps=2, whole=False),
        # The reference's own transport with surface tension, in the reference's precision.
        dict(name="step_256x256_plic_fp64", kind="step", w=256, h=256, precision="fp64", transport="plic",
             air="gas", tension=True, obstacles=0, steps=1, whole=True),
        # Viscous flow, small and the benchmark's size.
        dict(name="viscous_321x239", kind="viscous", w=321, h=239, precision="fp32"),
        dict(name="viscous_4096x4096", kind="viscous", w=4096, h=4096, precision="fp32"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, aspect):
    w = _spread(rng, lo, hi)
    h = int(round(w * math.exp(rng.uniform(-math.log(aspect), math.log(aspect)))))
    return w, min(max(h, lo), hi)


def draw(rng):
    kind = rng.choice(["project"] * 4 + ["step"] * 3 + ["plic", "batch", "viscous"])
    if kind == "project":
        w, h = _sides(rng, 48, 2048, 4.0)
        return dict(kind="project", w=w, h=h, precision=rng.choice(["fp32", "fp32", "fp64", "mixed"]),
                    obstacles=rng.randint(0, 8), fill=round(rng.uniform(0.3, 0.7), 3))
    if kind == "step":
        w, h = _sides(rng, 64, 1100, 2.0)
        return dict(kind="step", w=w, h=h, precision=rng.choice(["fp32", "fp32", "fp64", "mixed"]),
                    transport="semi_lagrangian", air=rng.choice(["gas", "dirichlet"]), tension=False,
                    obstacles=rng.randint(0, 16), steps=rng.randint(1, 3), whole=rng.random() < 0.4)
    if kind == "plic":
        w, h = _sides(rng, 64, 400, 2.0)
        return dict(kind="step", w=w, h=h, precision=rng.choice(["fp32", "fp64"]), transport="plic", air="gas",
                    tension=rng.random() < 0.7, obstacles=0, steps=1, whole=rng.random() < 0.5)
    if kind == "batch":
        lo = _spread(rng, 64, 128)
        return dict(kind="batch", count=rng.randint(3, 24), lo=lo, hi=_spread(rng, 2 * lo, 512),
                    precision=rng.choice(["fp32", "mixed"]), obstacles=rng.randint(0, 6))
    w, h = _sides(rng, 64, 2048, 2.0)
    return dict(kind="viscous", w=w, h=h, precision=rng.choice(["fp32", "fp32", "fp64"]))


# ---------------------------------------------------------------------------------------------
# Scenes (torch, on the GPU; FP64)
# ---------------------------------------------------------------------------------------------

def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt * 7919 + 17) % (1 << 62))
    return g


def _f32(a):
    return a.to(torch.float32).to(torch.float64)


def _close_walls(u, v):
    u[:, 0] = 0.0
    u[:, -1] = 0.0
    v[0, :] = 0.0
    v[-1, :] = 0.0


def _random_faces(w, h, seed):
    g = _generator(seed, 1)
    u = _f32(torch.rand((h, w + 1), generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0)
    v = _f32(torch.rand((h + 1, w), generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0)
    _close_walls(u, v)
    return u, v


def _smooth_faces(w, h, dx, seed, amplitude):
    """Velocities of a random smooth stream function (a few low modes), zero through the walls."""
    rng = random.Random(int(seed) * 31 + 5)
    y = torch.arange(h + 1, device="cuda", dtype=torch.float64)[:, None] / h
    x = torch.arange(w + 1, device="cuda", dtype=torch.float64)[None, :] / w
    psi = torch.zeros((h + 1, w + 1), device="cuda", dtype=torch.float64)
    for _ in range(6):
        kx, ky = rng.randint(1, 4), rng.randint(1, 4)
        psi += rng.uniform(-1.0, 1.0) / (kx + ky) * torch.sin(math.pi * kx * x) * torch.sin(math.pi * ky * y)
    u = (psi[1:, :] - psi[:-1, :]) / dx
    v = -(psi[:, 1:] - psi[:, :-1]) / dx
    scale = amplitude / max(float(u.abs().max()), float(v.abs().max()), 1e-30)
    u, v = _f32(u * scale), _f32(v * scale)
    _close_walls(u, v)
    return u, v


def _circles(w, h, count, seed):
    """Solid circles on a jittered lattice: none touches another or a wall, so no fluid cell is
    cut off from the rest."""
    if count == 0:
        return None
    rng = random.Random(int(seed) * 131 + 7)
    side = min(w, h)
    columns = max(1, int(math.ceil(math.sqrt(count * w / h))))
    rows = int(math.ceil(count / columns))
    pitch = min(w / columns, h / rows)
    places = [(i, j) for j in range(rows) for i in range(columns)]
    rng.shuffle(places)
    y = torch.arange(h, device="cuda", dtype=torch.float64)[:, None] + 0.5
    x = torch.arange(w, device="cuda", dtype=torch.float64)[None, :] + 0.5
    solid = torch.zeros((h, w), device="cuda", dtype=torch.bool)
    for i, j in places[:count]:
        r = min(rng.uniform(0.008, 0.04) * side, 0.5 * pitch - 4.0)
        slack = 0.5 * pitch - 4.0 - r
        if r < 1.0:
            continue
        cx = (i + 0.5) * w / columns + rng.uniform(-slack, slack)
        cy = (j + 0.5) * h / rows + rng.uniform(-slack, slack)
        solid |= (x - cx) ** 2 + (y - cy) ** 2 <= r * r
    return solid


def _pool(w, h, fill, seed):
    """Liquid up to `fill` of the height, the surface row partly filled, and a block above it."""
    rng = random.Random(int(seed) * 17 + 3)
    f = torch.zeros((h, w), device="cuda", dtype=torch.float64)
    level = fill * h
    full = int(math.floor(level))
    f[:full] = 1.0
    if full < h:
        f[full] = level - full
    bw, bh = max(1, w // 5), max(1, min(h - full - 1, 3 * h // 10))
    x0 = rng.randint(0, max(0, w - bw))
    if full + 1 < h:
        f[full: full + bh, x0: x0 + bw] = 1.0
    return f


def _noise(w, h, g, octaves=6, base=4):
    total = torch.zeros((1, 1, h, w), device="cuda", dtype=torch.float64)
    for k in range(octaves):
        n = base << k
        lattice = torch.rand((1, 1, n, n), generator=g, device="cuda", dtype=torch.float64)
        total += torch.nn.functional.interpolate(lattice, (h, w), mode="bilinear", align_corners=True) * 0.5 ** k
    return total[0, 0]


def _ranks(a):
    """Values mapped to (0, 1] by rank."""
    order = torch.argsort(a)
    ranks = torch.empty_like(a)
    ranks[order] = torch.arange(1, a.numel() + 1, device=a.device, dtype=a.dtype)
    return ranks / a.numel()


VISCOSITY = (1e-3, 10.0)


def _scene(case, seed):
    """The initial state: fraction, u, v, masses (FP64 tensors), and the physical parameters."""
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "viscous":
        dx, lo, hi = 1.0 / w, *VISCOSITY
        g = _generator(seed, 2)
        blob = _noise(w, h, g)
        order = blob.reshape(-1).sort().values
        f = (blob >= order[int(0.4 * order.numel())]).to(torch.float64)
        target = torch.full_like(f, lo)
        wet = f > 0
        target[wet] = lo * (hi / lo) ** _ranks(_noise(w, h, g)[wet])
        share = (target - lo) / (hi - lo)
        u, v = _random_faces(w, h, seed)
        area = dx * dx
        liquid = [LIQUID * f * (1.0 - share) * area, LIQUID * f * share * area]
        return dict(w=w, h=h, dx=dx, dt=1.0 / 120.0, f=f, u=u, v=v, liquid=liquid, gas=[GAS * (1.0 - f) * area],
                    solid=None, mu=target)
    tension = bool(case.get("tension"))
    dx = 1.0 / 128.0 if tension or kind == "batch" else 1.0 / w
    solid = _circles(w, h, case["obstacles"], seed)
    f = _pool(w, h, case.get("fill", 0.5), seed)
    if solid is not None:
        f[solid] = 0.0
    if kind == "project":
        u, v = _random_faces(w, h, seed)
        dt = 1.0 / 60.0
    else:
        # Up to a few cells per step in the open; past obstacles less than one, since this flow was
        # not made to go around them and would drag their contents (gas) through the liquid.
        u, v = _smooth_faces(w, h, dx, seed, 0.5 if tension else 0.1 if case["obstacles"] else 1.0)
        dt = 1.0 / 120.0
    area = dx * dx
    return dict(w=w, h=h, dx=dx, dt=dt, f=f, u=u, v=v, liquid=[LIQUID * f * area], gas=[GAS * (1.0 - f) * area],
                solid=solid, mu=None)


def _members(case, seed):
    """The grids of a batch: each a "step" case of its own, with its seed."""
    rng = random.Random(int(seed) * 7 + 1)
    # The sizes belong to the case and not to the seed: a plan is made for its grids.
    sizes = random.Random(case["count"] * 1009 + case["lo"] * 31 + case["hi"])
    members = []
    for _ in range(case["count"]):
        w, h = _sides(sizes, case["lo"], case["hi"], 2.0)
        members.append((dict(kind="batch", w=w, h=h, precision=case["precision"],
                             obstacles=sizes.randint(0, case["obstacles"]), fill=round(sizes.uniform(0.3, 0.7), 3)),
                        rng.randrange(1 << 30)))
    return members


# ---------------------------------------------------------------------------------------------
# The passes
# ---------------------------------------------------------------------------------------------

def _host(t):
    return None if t is None else t.cpu().numpy()


def _configure(grid, case, s):
    grid.configureMaterials([LIQUID] * len(s["liquid"]), [GAS], list(VISCOSITY) if s["mu"] is not None else None,
                            [VISCOSITY[0]] if s["mu"] is not None else None)
    grid.setGravityY(GRAVITY)
    grid.setAirModel(case.get("air", "gas"))
    grid.setTransport(case.get("transport", "semi_lagrangian"))
    if case.get("tension"):
        grid.setSurfaceTension(0.07)
    if s["solid"] is not None:
        grid.setObstacles(_host(s["solid"].to(torch.uint8)))


def _grids(case, seed):
    """(the saved state, the grid that works on it)."""
    s = _scene(case, seed)
    saved = FluidGrid(s["w"], s["h"], s["dx"], case["precision"])
    work = FluidGrid(s["w"], s["h"], s["dx"], case["precision"])
    for grid in (saved, work):
        _configure(grid, case, s)
    saved.upload(FluidGridState(_host(s["f"]), _host(s["u"]), _host(s["v"]), None, [_host(m) for m in s["liquid"]],
                                [_host(m) for m in s["gas"]]))
    work.copyStateFrom(saved)
    return saved, work, s["dt"]


def prepare(case, seed):
    if case["kind"] == "batch":
        grids = [_grids(c, k) for c, k in _members(case, seed)]
        return dict(case=case, grids=grids, batch=ProjectionBatch([work for _, work, _ in grids]))
    saved, work, dt = _grids(case, seed)
    return dict(case=case, saved=saved, work=work, dt=dt)


class _Field:
    """A grid's device array as torch sees it; keeps the grid alive."""

    def __init__(self, grid, pointer, shape):
        self.grid = grid
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8" if grid.precision == "fp64" else "<f4",
                                             data=(pointer, False), version=3)


def _velocities(grid):
    u, v = grid.velocityPointers()
    w, h = grid.getWidth(), grid.getHeight()
    return dict(u=torch.as_tensor(_Field(grid, u, (h, w + 1)), device="cuda"),
                v=torch.as_tensor(_Field(grid, v, (h + 1, w)), device="cuda"))


def _state(grid):
    s = grid.download()
    return dict(fraction=s.liquid_fraction, u=s.u, v=s.v, pressure=s.pressure, liquid=s.liquid_mass, gas=s.gas_mass)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        dt = state["grids"][0][2]
        for saved, work, _ in state["grids"]:
            work.copyStateFrom(saved)
        for _, work, dt in state["grids"]:
            work.advanceSubstep(dt)
        state["batch"].project(dt, MAX_ITERATIONS, TOLERANCE)
        return [_velocities(work) for _, work, _ in state["grids"]]
    work, dt = state["work"], state["dt"]
    work.copyStateFrom(state["saved"])
    if kind == "project":
        work.applyGravity(dt)
        work.project(dt, MAX_ITERATIONS, TOLERANCE)
        return _velocities(work)
    if kind == "step":
        for _ in range(case["steps"]):
            work.step(dt, MAX_ITERATIONS, TOLERANCE)
        return _state(work) if case["whole"] else _velocities(work)
    work.applyViscosity(dt)
    return _velocities(work)


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without, and how far correct implementations differ
# ---------------------------------------------------------------------------------------------

def work(case):
    if case["kind"] == "batch":
        parts = [work(dict(c, steps=1, whole=False, kind="step", transport="semi_lagrangian"))
                 for c, _ in _members(case, 0)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    n = case["w"] * case["h"]
    e = 8 if case["precision"] == "fp64" else 4
    velocity = 2 * e
    if case["kind"] == "project":
        # Velocities in and out; two masses and the two pressures of the warm start in; pressures out.
        return dict(bytes=n * (2 * velocity + 16 + 16 + 16), flops=n * 100.0)
    if case["kind"] == "step":
        per = 2 * velocity + 2 * 8 + 2 * 16 + 32  # velocities, fraction and masses in and out, pressures
        out = (8 * 6 if case["whole"] else 0)
        return dict(bytes=n * (per * case["steps"] + out), flops=n * 300.0 * case["steps"])
    # Velocities in and out, three masses in.
    return dict(bytes=n * (2 * velocity + 24), flops=n * 400.0)


def tolerance(case):
    if case["kind"] == "viscous":
        # CG stopped at 1e-4: a change of rounding moves the iterate it stops at. FP32 against FP64
        # of the same recurrences: 1e-4 (2-norm) and 6e-3 (largest) at most.
        return dict(rel=4e-4, max=0.03) if case["precision"] == "fp32" else dict(rel=1e-5, max=1e-3)
    # Solves of the same system to the same rule by another preconditioner: up to 1e-7 (FP64) and
    # 5e-7 (FP32 and mixed; the batches' slow flows) in the 2-norm, 8e-7 and 1.3e-5 at the worst face.
    if case["precision"] == "fp64":
        return dict(rel=4e-7, max=4e-6)
    return dict(rel=2e-6, max=5e-5)


# ---------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------

def _weights(density, solid):
    """Face weights 2 / (a + b) between open cells, zero elsewhere: right (h, w - 1), down (h - 1, w)."""
    right = 2.0 / (density[:, :-1] + density[:, 1:])
    down = 2.0 / (density[:-1] + density[1:])
    if solid is not None:
        right = torch.where(solid[:, :-1] | solid[:, 1:], 0.0, right)
        down = torch.where(solid[:-1] | solid[1:], 0.0, down)
    return right, down


def _solve_pressure(right, down, b, unknown, singular):
    """A p = b over the unknown cells by Jacobi-preconditioned CG; A the weighted 5-point Laplacian."""
    mask = unknown.to(torch.float64)
    diag = torch.zeros_like(b)
    diag[:, :-1] += right
    diag[:, 1:] += right
    diag[:-1] += down
    diag[1:] += down
    inv = torch.where(unknown & (diag > 0), 1.0 / diag.clamp_min(1e-300), 0.0)
    mask = torch.where(inv > 0, mask, 0.0)
    count = mask.sum()

    def apply(p):
        q = torch.zeros_like(p)
        f = right * (p[:, :-1] - p[:, 1:])
        q[:, :-1] += f
        q[:, 1:] -= f
        f = down * (p[:-1] - p[1:])
        q[:-1] += f
        q[1:] -= f
        return q * mask

    def centred(r):
        return r - mask * (r.sum() / count) if singular else r

    r = centred(b * mask)
    p = torch.zeros_like(b)
    z = inv * r
    d = z.clone()
    rz = (r * z).sum()
    start = float(rz)
    if start == 0.0:
        return p
    for i in range(40000):
        q = apply(d)
        alpha = rz / (d * q).sum()
        p += alpha * d
        r -= alpha * q
        if i % 50 == 49:
            r = centred(b * mask - apply(p))
        z = inv * r
        new = (r * z).sum()
        if i % 50 == 49 and float(new) <= 1e-23 * start:
            break
        d = z + (new / rz) * d
        rz = new
    return p


def _project64(u, v, density, solid, air, dx, dt):
    """The projected velocities (air: cells held at p = 0, or None) and the pressure."""
    h, w = density.shape
    u, v = u.clone(), v.clone()
    _close_walls(u, v)
    if solid is not None:
        u[:, 1:-1][solid[:, :-1] | solid[:, 1:]] = 0.0
        v[1:-1][solid[:-1] | solid[1:]] = 0.0
    right, down = _weights(density, solid)
    unknown = torch.ones((h, w), dtype=torch.bool, device=u.device)
    if solid is not None:
        unknown &= ~solid
    if air is not None:
        unknown &= ~air
    b = -((u[:, 1:] - u[:, :-1]) + (v[1:] - v[:-1])) * (dx / dt)
    p = _solve_pressure(right, down, b, unknown, air is None)
    u[:, 1:-1] -= (p[:, 1:] - p[:, :-1]) / dx * dt * right
    v[1:-1] -= (p[1:] - p[:-1]) / dx * dt * down
    open_cells = unknown if air is None else None
    if open_cells is not None:
        p = torch.where(open_cells, p - p[open_cells].mean(), 0.0)
    return u, v, p


def _sample(a, x, y):
    h, w = a.shape
    x, y = x.clamp(0.0, w - 1.0), y.clamp(0.0, h - 1.0)
    x0, y0 = x.to(torch.int64), y.to(torch.int64)
    x1, y1 = (x0 + 1).clamp(max=w - 1), (y0 + 1).clamp(max=h - 1)
    tx, ty = x - x0, y - y0
    top = a[y0, x0] * (1 - tx) + a[y0, x1] * tx
    bottom = a[y1, x0] * (1 - tx) + a[y1, x1] * tx
    return top * (1 - ty) + bottom * ty


def _advect64(fields, u, v, scale):
    """Midpoint back-tracing of cell fields and face velocities through (u, v); scale = dt / dx."""
    h, w = fields[0].shape

    def positions(nx, ny, ox, oy):
        y = torch.arange(ny, device=u.device, dtype=torch.float64)[:, None] + oy
        x = torch.arange(nx, device=u.device, dtype=torch.float64)[None, :] + ox
        x, y = torch.broadcast_tensors(x, y)
        vx, vy = _sample(u, x, y - 0.5), _sample(v, x - 0.5, y)
        mx, my = x - 0.5 * scale * vx, y - 0.5 * scale * vy
        vx, vy = _sample(u, mx, my - 0.5), _sample(v, mx - 0.5, my)
        return x - scale * vx, y - scale * vy

    bx, by = positions(w, h, 0.5, 0.5)
    moved = [_sample(f, bx - 0.5, by - 0.5) for f in fields]
    bx, by = positions(w + 1, h, 0.0, 0.5)
    nu = _sample(u, bx, by - 0.5)
    bx, by = positions(w, h + 1, 0.5, 0.0)
    nv = _sample(v, bx - 0.5, by)
    _close_walls(nu, nv)
    return moved, nu, nv


def _extend(value, known, layers=4):
    """Unknown faces beside known ones take their mean, layer by layer; the rest are zero."""
    value, known = value.clone(), known.clone()
    for _ in range(layers):
        total, count = torch.zeros_like(value), torch.zeros_like(value)
        have = torch.where(known, value, 0.0)
        k = known.to(torch.float64)
        for a, b in (((slice(1, None), slice(None)), (slice(None, -1), slice(None))),
                     ((slice(None), slice(1, None)), (slice(None), slice(None, -1)))):
            total[a] += have[b]
            count[a] += k[b]
            total[b] += have[a]
            count[b] += k[a]
        new = ~known & (count > 0)
        value = torch.where(new, total / count.clamp_min(1.0), value)
        known = known | new
    return torch.where(known, value, 0.0)


def _extend_air(u, v, f, solid):
    h, w = f.shape
    near = f > 0.5
    if solid is not None:
        near = near | solid
    ku = torch.ones((h, w + 1), dtype=torch.bool, device=u.device)
    kv = torch.ones((h + 1, w), dtype=torch.bool, device=u.device)
    ku[:, 1:-1] = near[:, :-1] | near[:, 1:]
    kv[1:-1] = near[:-1] | near[1:]
    return _extend(u, ku), _extend(v, kv)


def _step64(case, s, steps):
    u, v, f = s["u"], s["v"], s["f"]
    masses = s["liquid"] + s["gas"]
    p = None
    for _ in range(steps):
        if case.get("air") == "dirichlet":
            u, v = _extend_air(u, v, f, s["solid"])
        moved, u, v = _advect64([f] + masses, u, v, s["dt"] / s["dx"])
        f, masses = moved[0], moved[1:]
        v = v.clone()
        v[1:-1] += GRAVITY * s["dt"]
        air = None
        if case.get("air") == "dirichlet":
            air = ~(f > 0.5)
            if s["solid"] is not None:
                air &= ~s["solid"]
        u, v, p = _project64(u, v, sum(masses) / (s["dx"] * s["dx"]), s["solid"], air, s["dx"], s["dt"])
    return f, u, v, p, masses


def _viscous64(s):
    """m (x - x0) = -dt K x by Jacobi-preconditioned CG; K the Hessian of the strain energy."""
    w, h, dx, dt = s["w"], s["h"], s["dx"], s["dt"]
    rho, mu = sum(s["liquid"] + s["gas"]) / (dx * dx), s["mu"]
    area = dx * dx
    mass_u = 0.5 * area * (rho[:, 1:] + rho[:, :-1])
    mass_v = 0.5 * area * (rho[1:] + rho[:-1])
    corner = 0.25 * (mu[1:, 1:] + mu[1:, :-1] + mu[:-1, 1:] + mu[:-1, :-1])

    def apply(a, b):
        # a: interior u faces (h, w - 1); b: interior v faces (h - 1, w). Walls hold zero.
        fu = torch.nn.functional.pad(a, (1, 1))
        fv = torch.nn.functional.pad(b, (0, 0, 1, 1))
        nx = 2.0 * mu * (fu[:, 1:] - fu[:, :-1])
        ny = 2.0 * mu * (fv[1:] - fv[:-1])
        t = corner * ((a[1:] - a[:-1]) + (b[:, 1:] - b[:, :-1]))
        ru = mass_u * a + dt * (nx[:, :-1] - nx[:, 1:])
        ru[1:] += dt * t
        ru[:-1] -= dt * t
        rv = mass_v * b + dt * (ny[:-1] - ny[1:])
        rv[:, 1:] += dt * t
        rv[:, :-1] -= dt * t
        return ru, rv

    def dot(p, q):
        return (p[0] * q[0]).sum() + (p[1] * q[1]).sum()

    du = mass_u + dt * 2.0 * (mu[:, 1:] + mu[:, :-1])
    du[1:] += dt * corner
    du[:-1] += dt * corner
    dv = mass_v + dt * 2.0 * (mu[1:] + mu[:-1])
    dv[:, 1:] += dt * corner
    dv[:, :-1] += dt * corner
    x = [s["u"][:, 1:-1].clone(), s["v"][1:-1].clone()]
    b = (mass_u * x[0], mass_v * x[1])
    ax = apply(*x)
    r = [b[0] - ax[0], b[1] - ax[1]]
    z = [r[0] / du, r[1] / dv]
    d = [z[0].clone(), z[1].clone()]
    rz = dot(r, z)
    start = float(rz)
    for i in range(20000):
        q = apply(*d)
        alpha = rz / dot(d, q)
        for k in (0, 1):
            x[k] += alpha * d[k]
            r[k] -= alpha * q[k]
        z = [r[0] / du, r[1] / dv]
        new = dot(r, z)
        if i % 50 == 49 and float(new) <= 1e-24 * start:
            break
        for k in (0, 1):
            d[k] = z[k] + (new / rz) * d[k]
        rz = new
    u, v = torch.zeros_like(s["u"]), torch.zeros_like(s["v"])
    u[:, 1:-1], v[1:-1] = x[0], x[1]
    return dict(u=u, v=v)


def exact(case, seed):
    if case.get("transport") == "plic":
        return None  # geometric transport: its bits are pinned by the tests, it has no closed 64-bit form here
    if case["kind"] == "batch":
        out = []
        for c, k in _members(case, seed):
            _, u, v, _, _ = _step64(c, _scene(c, k), 1)
            out.append(dict(u=u, v=v))
        return out
    if case["kind"] == "viscous":
        if case["w"] * case["h"] > 700 * 700:
            return None  # minutes
        return _viscous64(_scene(case, seed))
    s = _scene(case, seed)
    if case["kind"] == "project":
        v = s["v"].clone()
        v[1:-1] += GRAVITY * s["dt"]
        u, v, _ = _project64(s["u"], v, sum(s["liquid"] + s["gas"]) / (s["dx"] * s["dx"]), s["solid"], None, s["dx"],
                             s["dt"])
        return dict(u=u, v=v)
    f, u, v, p, masses = _step64(case, s, case["steps"])
    if not case["whole"]:
        return dict(u=u, v=v)
    n = len(s["liquid"])
    return dict(fraction=f, u=u, v=v, pressure=p, liquid=masses[:n], gas=masses[n:])
