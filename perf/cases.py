"""The work that users of the fluid framework have it do, as measurable cases.

`listed()` names the cases, `draw(rng)` gives more of the same ranges,
`prepare(case, seed)` makes what a program holds before a call, `run(state)`
is one pass through the public entry points, `work(case)` the bytes and
operations a pass cannot do without, and `exact(case, seed)` the outputs in
64 bits from plain torch.

Kinds of work:

* step: a program that keeps its particles in device tensors loads them into
  its world, advances some steps in one call, and reads the fields back into
  its tensors (what the resident slab decomposition does every step).
* frame: a host engine exchanges positions and velocities as numpy arrays
  around every step.
* batch: many independent scenes of uneven size in one world.
* pile: fluid that has collapsed onto the floor, hundreds of particles per
  cell (where the long dam-break runs spend most of their time).
* adjoint: recorded forward steps and the reverse sweep, one iteration of a
  differentiable-physics optimisation.
* couple: a frame with a heat grid and point masses in the fluid.

The f64 form's outputs are returned as they are.  The compensated form sums
its pair terms in f32, so the fields made of them are returned as f32 (the
type its consumers take); its positions, which stay f64, are returned as f64.
"""
import math

import numpy as np
import torch

import physics_b200 as pb

H = 0.2  # SphParams::defaults()
SPACING = 0.1
FIELDS = (("pos", pb.FIELD_POS), ("vel", pb.FIELD_VEL), ("acc", pb.FIELD_ACC), ("rho", pb.FIELD_RHO),
          ("p", pb.FIELD_P))


def listed():
    return [
        # The README's quick start: the smallest scene, launches and latency count.
        {"name": "quickstart_f64", "kind": "step", "form": "f64", "nx": 7, "ny": 7, "nz": 7, "spacing": 0.3,
         "dt": 0.01, "steps": 10, "materials": 1},
        # An interactive engine: a small odd-sized block, host arrays in and out every frame.
        {"name": "frame_f64_4k", "kind": "frame", "form": "f64", "nx": 15, "ny": 19, "nz": 15, "spacing": 0.1,
         "dt": 0.005, "steps": 1, "materials": 1},
        # The differentiation form's size, plain stepping.
        {"name": "dam_f64_65k", "kind": "step", "form": "f64", "nx": 32, "ny": 64, "nz": 32, "spacing": 0.1,
         "dt": 0.005, "steps": 4, "materials": 1},
        # Three power-law materials (the shear sum is live) at a ragged size.
        {"name": "materials_f64_112k", "kind": "step", "form": "f64", "nx": 37, "ny": 53, "nz": 57, "spacing": 0.1,
         "dt": 0.005, "steps": 2, "materials": 3},
        # The plain configuration at scale.
        {"name": "dam_f64_1m", "kind": "step", "form": "f64", "nx": 80, "ny": 160, "nz": 80, "spacing": 0.1,
         "dt": 0.005, "steps": 2, "materials": 1},
        # The compensated form on a small odd-sized scene.
        {"name": "dam_comp_8k", "kind": "step", "form": "comp", "nx": 19, "ny": 23, "nz": 19, "spacing": 0.1,
         "dt": 0.005, "steps": 5, "materials": 1},
        # Middle size, ragged, with power-law materials.
        {"name": "materials_comp_380k", "kind": "step", "form": "comp", "nx": 61, "ny": 127, "nz": 49,
         "spacing": 0.105, "dt": 0.005, "steps": 3, "materials": 3},
        # The benchmark's configuration: the largest case.
        {"name": "dam_comp_4m", "kind": "step", "form": "comp", "nx": 128, "ny": 256, "nz": 128, "spacing": 0.1,
         "dt": 0.0025, "steps": 3, "materials": 1},
        # Independent scenes in one world.
        {"name": "batch_comp_24", "kind": "batch", "form": "comp", "scenes": 24, "least": 2000, "most": 60000,
         "dt": 0.005, "steps": 5, "materials": 1},
        # The collapsed regime: a sheet of 160 particles per cell.
        {"name": "pile_comp_100k", "kind": "pile", "form": "comp", "n": 100003, "per_cell": 160.0, "dt": 0.0025,
         "steps": 2, "materials": 1},
        # One optimisation iteration at the differentiation form's size.
        {"name": "adjoint_f64_65k", "kind": "adjoint", "form": "f64", "nx": 32, "ny": 64, "nz": 32, "spacing": 0.1,
         "dt": 0.005, "steps": 10, "every": 5, "materials": 1},
        # A coupled frame: heat grid and point masses around one step.
        {"name": "coupled_f64_32k", "kind": "couple", "form": "f64", "nx": 27, "ny": 45, "nz": 27, "spacing": 0.1,
         "dt": 0.0025, "steps": 1, "materials": 1, "points": 400},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, n):
    a = [rng.uniform(0.6, 1.7) for _ in range(3)]
    s = (n / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
    return [max(2, int(round(s * v))) for v in a]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "frame", "batch", "pile", "adjoint", "couple"])
    form = rng.choice(["f64", "comp"])
    spacing = round(rng.uniform(0.09, 0.13), 4)
    mats = rng.choice([1, 1, 3])
    if kind == "step":
        d = _dims(rng, _log(rng, 350, 9.0e5 if form == "f64" else 3.2e6))
        return {"kind": kind, "form": form, "nx": d[0], "ny": d[1], "nz": d[2], "spacing": spacing,
                "dt": rng.choice([0.0025, 0.005]), "steps": rng.randint(1, 3), "materials": mats}
    if kind == "frame":
        d = _dims(rng, _log(rng, 350, 60000))
        return {"kind": kind, "form": form, "nx": d[0], "ny": d[1], "nz": d[2], "spacing": spacing, "dt": 0.005,
                "steps": 1, "materials": mats}
    if kind == "batch":
        return {"kind": kind, "form": "comp", "scenes": rng.randint(2, 40), "least": 1500,
                "most": int(_log(rng, 4000, 60000)), "dt": 0.005, "steps": rng.randint(1, 5), "materials": 1}
    if kind == "pile":
        return {"kind": kind, "form": "comp", "n": int(_log(rng, 5000, 120000)),
                "per_cell": round(rng.uniform(40.0, 200.0), 1), "dt": 0.0025, "steps": rng.randint(1, 2),
                "materials": rng.choice([1, 3])}
    if kind == "adjoint":
        d = _dims(rng, _log(rng, 800, 65000))
        return {"kind": kind, "form": "f64", "nx": d[0], "ny": d[1], "nz": d[2], "spacing": spacing, "dt": 0.005,
                "steps": rng.randint(3, 10), "every": rng.randint(2, 6), "materials": mats}
    d = _dims(rng, _log(rng, 2000, 60000))
    return {"kind": "couple", "form": "f64", "nx": d[0], "ny": d[1], "nz": d[2], "spacing": spacing, "dt": 0.0025,
            "steps": 1, "materials": mats, "points": rng.randint(20, 600)}


# ---- inputs -----------------------------------------------------------------


def _lattice_mass(s):
    w = 0.0
    c = 315.0 / (64.0 * math.pi * H ** 9)
    m = int(math.ceil(H / s)) + 1
    for i in range(-m, m + 1):
        for j in range(-m, m + 1):
            for k in range(-m, m + 1):
                r = s * math.sqrt(i * i + j * j + k * k)
                if r < H:
                    w += c * (H * H - r * r) ** 3
    return 1000.0 / w


def _block(g, nx, ny, nz, s):
    """A jittered lattice block in the low corner, moving in a smooth field."""
    i = torch.arange(nx * ny * nz, device="cuda")
    base = torch.stack([i // (ny * nz), (i // nz) % ny, i % nz], dim=1).double().add_(0.5).mul_(s)
    pos = base + (2.0 * torch.rand(base.shape, generator=g, device="cuda", dtype=torch.float64) - 1.0) * (0.05 * s)
    ph = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * 6.28
    vel = 0.3 * torch.sin(1.7 * pos[:, [1, 2, 0]] + ph)
    vel += 0.02 * torch.randn(pos.shape, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel


def _batch_shapes(case):
    """Lattice counts and box extents of a batch's scenes: the shapes are the case's."""
    r = np.random.default_rng(case["scenes"] * 7919 + case["most"])
    out = []
    for _ in range(case["scenes"]):
        n = math.exp(r.uniform(math.log(case["least"]), math.log(case["most"])))
        a = r.uniform(0.5, 2.0, 3)
        fill = r.uniform(0.2, 0.5)
        box = (n * SPACING ** 3 / fill / float(np.prod(a))) ** (1.0 / 3.0) * a
        c = np.maximum(2, np.round(box * fill ** (1.0 / 3.0) / SPACING)).astype(int)
        out.append(([int(v) for v in c], [float(v) for v in box]))
    return out


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    d = {}
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        parts = [_block(g, *c, SPACING) for c, _ in shapes]
        pos, vel = torch.cat([p for p, _ in parts]), torch.cat([v for _, v in parts])
        d["counts"] = [p.shape[0] for p, _ in parts]
        d["lo"], d["hi"] = [(0.0, 0.0, 0.0)] * len(shapes), [tuple(b) for _, b in shapes]
        mass = _lattice_mass(SPACING)
    elif kind == "pile":
        n = case["n"]
        edge = math.sqrt(n / case["per_cell"]) * H
        u = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
        pos = torch.stack([u[:, 0] * edge, 0.08 * u[:, 1] ** 2, u[:, 2] * edge], dim=1)
        vel = 0.05 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
        mass = _lattice_mass(SPACING)
        d["box"] = ((0.0,) * 3, (edge, 2.0, edge))
    else:
        s = case["spacing"]
        pos, vel = _block(g, case["nx"], case["ny"], case["nz"], s)
        mass = _lattice_mass(s)
        top = 2.0 * s * max(case["nx"], case["ny"], case["nz"])
        d["box"] = ((0.0,) * 3, (top,) * 3)
    n = pos.shape[0]
    d["n"], d["pos"], d["vel"] = n, pos.contiguous(), vel.contiguous()
    d["mass"] = torch.full((n,), mass, device="cuda", dtype=torch.float64)
    d["mat"] = torch.randint(0, case["materials"], (n,), generator=g, device="cuda", dtype=torch.int32)
    if kind == "adjoint":
        d["gpos"] = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        d["gvel"] = 0.1 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    if kind == "couple":
        m, ext = case["points"], torch.tensor([case["nx"], case["ny"], case["nz"]], device="cuda") * case["spacing"]
        grid = [max(2, int(float(e) / H) + 2) for e in ext]
        d["ppos"] = (torch.rand((m, 3), generator=g, device="cuda", dtype=torch.float64) * ext).cpu().numpy()
        d["pvel"] = 0.2 * torch.randn((m, 3), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        d["pmass"] = (0.01 + 0.02 * torch.rand(m, generator=g, device="cuda", dtype=torch.float64)).cpu().numpy()
        d["temp"] = torch.rand(grid[::-1], generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    return d


def _params(case, d):
    p = pb.SphParams.defaults()
    if "box" in d:
        p.bounds_min, p.bounds_max = d["box"]
    if case["materials"] == 3:
        p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 0.7, 1.3]
    return p


def prepare(case, seed):
    d = _inputs(case, seed)
    w = pb.FluidWorld(_params(case, d), case["form"])
    s = {"case": case, "w": w, "in": d}
    w.set_particles_device(d["pos"], d["mass"], d["vel"], d["mat"])
    if case["kind"] in ("frame", "couple"):
        # The host engine's own arrays, page-locked once.
        for k in ("pos", "vel"):
            s[k] = torch.empty((d["n"], 3), dtype=torch.float64, pin_memory=True).copy_(d[k]).numpy()
            s["out_" + k] = torch.empty((d["n"], 3), dtype=torch.float64, pin_memory=True).numpy()
    if case["kind"] in ("step", "batch", "pile"):
        s["out"] = {k: torch.empty((d["n"], 3) if k in ("pos", "vel", "acc") else (d["n"],), device="cuda",
                                   dtype=torch.float64) for k, _ in FIELDS}
    return s


# ---- one pass -----------------------------------------------------------------


def run(state):
    case, w, d = state["case"], state["w"], state["in"]
    kind = case["kind"]
    if kind in ("step", "pile", "batch"):
        if kind == "batch":
            w.clear_scenes()
        w.set_particles_device(d["pos"], d["mass"], d["vel"], d["mat"])
        if kind == "batch":
            w.set_scenes(d["counts"], d["lo"], d["hi"])
        w.step(case["dt"], case["steps"])
        for k, fld in FIELDS:
            w.get_device(fld, state["out"][k])
        return _typed(case, state["out"])
    if kind == "frame":
        w.set(pb.FIELD_POS, state["pos"])
        w.set(pb.FIELD_VEL, state["vel"])
        w.step(case["dt"], case["steps"])
        w.get(pb.FIELD_POS, state["out_pos"].reshape(-1))
        w.get(pb.FIELD_VEL, state["out_vel"].reshape(-1))
        return _typed(case, {"pos": state["out_pos"], "vel": state["out_vel"]})
    if kind == "adjoint":
        w.set_particles_device(d["pos"], d["mass"], d["vel"], d["mat"])
        w.tape_begin(case["every"])
        w.step(case["dt"], case["steps"])
        g = w.step_backward(d["gpos"], d["gvel"])
        w.tape_clear()
        return g
    dt = case["dt"]
    w.set(pb.FIELD_POS, state["pos"])
    w.set(pb.FIELD_VEL, state["vel"])
    src = w.couple_heat(d["temp"], np.zeros_like(d["temp"]), (0.0, 0.0, 0.0), H, dt, 0.5, 2e-4, 0.1)
    force = w.couple_points(d["ppos"], d["pvel"], d["pmass"], dt, 1.0, 1000.0)
    w.step(dt, case["steps"])
    w.get(pb.FIELD_POS, state["out_pos"].reshape(-1))
    w.get(pb.FIELD_VEL, state["out_vel"].reshape(-1))
    return {"pos": state["out_pos"], "vel": state["out_vel"], "src": src, "force": force}


def _typed(case, out):
    if case["form"] == "f64":
        return out
    f32 = (lambda t: t.float()) if torch.is_tensor(out["pos"]) else (lambda a: a.astype(np.float32))
    return {k: v if k == "pos" else f32(v) for k, v in out.items()}


# ---- what a pass cannot do without --------------------------------------------


def _count(case):
    if case["kind"] == "batch":
        return sum(c[0] * c[1] * c[2] for c, _ in _batch_shapes(case))
    return case["n"] if case["kind"] == "pile" else case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Bytes: the particles read once and the fields written once.  Operations: per step and
    in-range pair the density (12) and force (60) terms; a reverse step about three times that."""
    n = _count(case)
    if case["kind"] == "pile":
        pairs = case["per_cell"] * 2.6
    else:
        s = case.get("spacing", SPACING)
        pairs = 4.0 / 3.0 * math.pi * (H / s) ** 3 if s < H else 1.0
    flops = 72.0 * pairs * n * case["steps"]
    size = n * (56 + 4 + 88)
    if case["kind"] == "frame":
        size = n * 96
    if case["kind"] == "adjoint":
        flops, size = 5.0 * flops, n * (60 + 48 + 48)
    if case["kind"] == "couple":
        size = n * 96 + case["points"] * 80
        flops += case["points"] * 219 * 14.0 + n * 60.0
    return {"bytes": float(size), "flops": float(flops)}


# ---- the same in 64 bits --------------------------------------------------------


def _edges(pos, scene, most=1 << 26):
    """(i, j) of all pairs i != j with |x_i - x_j| < H, in chunks of queries."""
    key = torch.floor(pos * (1.0 / H)).long()
    key = key - key.min(0).values + 1
    dims = key.max(0).values + 2
    if scene is not None:
        key[:, 0] += scene * dims[0]
    lin = (key[:, 0] * dims[1] + key[:, 1]) * dims[2] + key[:, 2]
    sl, order = torch.sort(lin)
    per = [(a * int(dims[1]) + b) * int(dims[2]) for a in (-1, 0, 1) for b in (-1, 0, 1)]
    n, at, out = pos.shape[0], 0, []
    width = max(1, min(n, 1 << 21))
    while at < n:
        q = order[at:at + width]
        lo = torch.stack([torch.searchsorted(sl, lin[q] + o - 1) for o in per])
        hi = torch.stack([torch.searchsorted(sl, lin[q] + o + 1, right=True) for o in per])
        cnt = hi - lo
        if int(cnt.sum()) > most and width > 1:
            width = max(1, width // 2)
            continue
        flat = cnt.reshape(-1)
        own = torch.repeat_interleave(torch.arange(flat.numel(), device=pos.device), flat)
        rank = torch.arange(own.numel(), device=pos.device) - (torch.cumsum(flat, 0) - flat)[own]
        j = order[lo.reshape(-1)[own] + rank]
        i = q[own % q.numel()]
        keep = (i != j) & ((pos[i] - pos[j]).norm(dim=1) < H)
        out.append((i[keep], j[keep]))
        at += q.numel()
    return out


def _exact_step(p, x, v, m, mat, dt, lo, hi, scene=None, body=0.0):
    c6, cs, cl = 315.0 / (64.0 * math.pi * H ** 9), -45.0 / (math.pi * H ** 6), 45.0 / (math.pi * H ** 6)
    with torch.no_grad():
        chunks = _edges(x.detach(), scene)
    zero = torch.zeros_like(m)
    rho = m * (c6 * H ** 6)
    for i, j in chunks:
        r2 = ((x[j] - x[i]) ** 2).sum(1)
        rho = rho.index_add(0, i, m[j] * (c6 * (H * H - r2) ** 3))
    pr = p.stiffness * torch.clamp(rho - p.rest_density, min=0.0)
    pr2, mr = pr / (rho * rho), m / rho
    fp, fv, xs, sh = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x), zero
    for i, j in chunks:
        d, dv = x[j] - x[i], v[j] - v[i]
        r = (d * d).sum(1).sqrt()
        mm = m[i] * m[j]
        fp = fp.index_add(0, i, d * (mm * (pr2[i] + pr2[j]) * cs * (H - r) ** 2 / r)[:, None])
        fv = fv.index_add(0, i, dv * (mm / rho[j] * cl * (H - r))[:, None])
        xs = xs.index_add(0, i, dv * (mr[j] * c6 * (H * H - r * r) ** 3)[:, None])
        if len(p.visc_k) > 1:
            sh = sh.index_add(0, i, dv.norm(dim=1) / (r + 1e-4) * mr[j])
    k = p.visc_k if torch.is_tensor(p.visc_k) else torch.tensor(p.visc_k, device=x.device, dtype=torch.float64)
    e = torch.tensor(p.visc_n, device=x.device, dtype=torch.float64)[mat.long()] - 1.0
    mu = k[mat.long()] * torch.clamp(sh, min=p.shear_min) ** e
    acc = (fp + fv * mu[:, None]) / rho[:, None]
    v1 = v + (acc + torch.tensor(p.gravity, device=x.device, dtype=torch.float64) + body) * dt + xs * p.xsph_eps
    x1 = x + v1 * dt
    wall = (x1 < lo) | (x1 > hi)
    return torch.minimum(torch.maximum(x1, lo), hi), torch.where(wall, -v1 * p.boundary_damp, v1), acc, rho, pr


def exact(case, seed):
    d = _inputs(case, seed)
    p = _params(case, d)
    x, v, m, mat, dt = d["pos"], d["vel"], d["mass"], d["mat"], case["dt"]
    t = (lambda a: torch.tensor(a, device="cuda", dtype=torch.float64))
    scene = None
    if case["kind"] == "batch":
        scene = torch.repeat_interleave(torch.arange(len(d["counts"]), device="cuda"), t(d["counts"]).long())
        lo, hi = t(d["lo"])[scene], t(d["hi"])[scene]
    else:
        lo, hi = t(d["box"][0]).expand_as(x), t(d["box"][1]).expand_as(x)
    if case["kind"] == "adjoint":
        x0, v0 = x.clone().requires_grad_(), v.clone().requires_grad_()
        p.stiffness, p.visc_k = t(p.stiffness).requires_grad_(), t(p.visc_k).requires_grad_()
        x, v = x0, v0
        for _ in range(case["steps"]):
            x, v = _exact_step(p, x, v, m, mat, dt, lo, hi)[:2]
        loss = (x * t(d["gpos"])).sum() + (v * t(d["gvel"])).sum()
        gx, gv, gs, gk = torch.autograd.grad(loss, (x0, v0, p.stiffness, p.visc_k))
        return {"pos": gx, "vel": gv, "stiffness": float(gs), "visc_k0": float(gk[0])}
    if case["kind"] == "couple":
        return _exact_couple(case, d, p, x, v, m, mat, dt, lo, hi)
    with torch.no_grad():
        for _ in range(case["steps"]):
            x, v, acc, rho, pr = _exact_step(p, x, v, m, mat, dt, lo, hi, scene)
    if case["kind"] == "frame":
        return {"pos": x, "vel": v}
    return {"pos": x, "vel": v, "acc": acc, "rho": rho, "p": pr}


def _exact_couple(case, d, p, x, v, m, mat, dt, lo, hi):
    g = torch.tensor(p.gravity, device="cuda", dtype=torch.float64)
    u = torch.from_numpy(d["temp"]).cuda()
    dims = torch.tensor(u.shape[::-1], device="cuda")
    q = x / H
    c = torch.floor(q).long()
    f = q - c
    inside = ((x >= 0.0) & (x <= H * (dims - 1))).all(1)
    c0 = torch.minimum(c.clamp(min=0), dims - 1)
    temp = torch.zeros_like(m)
    for a in range(8):
        o = torch.tensor([a & 1, (a >> 1) & 1, a >> 2], device="cuda")
        k = torch.minimum(c0 + o, dims - 1)
        temp += torch.where(o == 1, f, 1.0 - f).prod(1) * u[k[:, 2], k[:, 1], k[:, 0]]
    body = -g * 2e-4 * (torch.where(inside, temp, 0.5) - 0.5)[:, None]
    src = torch.zeros_like(u).reshape(-1)
    flat = (c0[:, 2] * dims[1] + c0[:, 1]) * dims[0] + c0[:, 0]
    src.index_add_(0, flat[inside], (0.1 * v.norm(dim=1) * dt)[inside])
    key = torch.floor(x * (1.0 / H)).long()
    v, force = v.clone(), []
    for pos, vel, mass in zip(*(torch.from_numpy(d[k]).cuda() for k in ("ppos", "pvel", "pmass"))):
        near = ((key - torch.floor(pos * (1.0 / H)).long()).abs() <= 1).all(1).nonzero()[:, 0]
        mj = m[near]
        vf = (v[near] * mj[:, None]).sum(0) / mj.sum() if near.numel() else torch.zeros_like(g)
        fo = -g * (p.rest_density * mass / 1000.0) + (vf - vel) * mass
        force.append(fo)
        if near.numel():
            v[near] -= fo * dt * (mj / mj.sum())[:, None]
    x, v = _exact_step(p, x, v, m, mat, dt, lo, hi, body=body)[:2]
    return {"pos": x, "vel": v, "src": src.reshape(u.shape), "force": torch.stack(force)}
