"""Workloads that the framework's performance is measured on.

Each case is one call pattern of a user's program through the public entry points (`Scene`, `SceneBatch`,
`DiffRollout` / `rollout`, `ckmpm_simulate_noalloc`), with seeded synthetic particles of the shapes and materials of
`ckmpm_b200.scenes`:

* frame:    restore a saved state, advance `steps` substeps, read the result back (what a rollout from a saved
            state, a parameter sweep or a frame of an animation does); `out` is "state" (x, v, F, aux, ids) or
            "positions" (the per-frame position export into pinned memory);
* adaptive: the same with the CFL-controlled frame loop that `MPMEngine.Simulate` runs;
* batch:    many independent scenes in one handle;
* noalloc:  the one-call, allocation-free simulation on device arrays;
* job:      a whole short job: scene creation, upload, setup, substeps, position export, destruction;
* diff:     forward and adjoint of a differentiable rollout.

`exact` restates all of them in plain torch in 64 bits.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from ckmpm_b200 import MPMConfig, MPMMaterial, MPMModel, Scene, _capi
from ckmpm_b200.batch import SceneBatch
from ckmpm_b200.diff import DiffRollout, rollout

#: E, nu and density of the elastic and granular materials, as ckmpm_b200.scenes gives them.
ELASTIC = {"fixed_corotated": (5e4, 0.3, 1000.0), "drucker_prager": (3.5e5, 0.3, 1600.0), "von_mises": (2e4, 0.3, 1000.0),
           "nacc": (2e4, 0.4, 1000.0), "linear": (5e4, 0.3, 1000.0)}
FLUID = (1e4, 7.15, 0.1, 1000.0)  # bulk, gamma, viscosity, density
PPC = 8


def listed():
    return [
        # The smallest call: 2k particles, a handful of substeps. Launch latency and the read-back count.
        {"name": "cube_2k", "kind": "frame", "material": "fixed_corotated", "shape": "box", "n": 2000, "blocks": 16,
         "boundary": "sticky_blocks", "layout": "lattice", "dt": 1e-4, "steps": 8, "out": "state"},
        # The jelly cube of the benchmark (16.8k particles), one frame of 100 substeps.
        {"name": "jelly_cube", "kind": "frame", "material": "fixed_corotated", "shape": "box", "n": 16795, "blocks": 16,
         "boundary": "sticky_blocks", "layout": "lattice", "dt": 1e-4, "steps": 100, "out": "state"},
        # The parity tests' sand column on the slip floor, with plastic flow from the first substeps.
        {"name": "sand_small", "kind": "frame", "material": "drucker_prager", "shape": "cylinder", "n": 16471, "blocks": 16,
         "boundary": "slip_floor", "layout": "lattice", "dt": 1e-4, "steps": 50, "out": "state"},
        # The benchmark's headline scene: the 1.69M-particle sand column, positions exported after the frame.
        {"name": "sand_column", "kind": "frame", "material": "drucker_prager", "shape": "cylinder", "n": 1686824, "blocks": 64,
         "boundary": "slip_floor", "layout": "lattice", "dt": 5e-5, "steps": 50, "out": "positions"},
        # The mixed dam break (fluid block and 64 elastic spheres) at 17M particles: the largest scene.
        {"name": "dam_break", "kind": "frame", "material": "fluid", "shape": "box", "n": 16000000, "blocks": 64, "spheres": 64,
         "sphere_n": 15300, "boundary": "sticky_blocks", "layout": "lattice", "dt": 4e-5, "steps": 8, "out": "positions"},
        # Cam-clay between slip walls given as a boundary field, unordered particles, an odd domain.
        {"name": "clay_field", "kind": "frame", "material": "nacc", "shape": "sphere", "n": 60013, "blocks": 19,
         "boundary": "field", "layout": "random", "dt": 8e-5, "steps": 24, "out": "state"},
        # One short frame of the engine's CFL-controlled loop, von Mises with driven rigid particles.
        {"name": "adaptive_metal", "kind": "adaptive", "material": "von_mises", "shape": "box", "n": 8626, "blocks": 16,
         "boundary": "sticky_blocks", "layout": "lattice", "dt": 1e-4, "frame_time": 0.0033, "cfl": 0.5, "rigid": 2048,
         "out": "state"},
        # 256 independent scenes of 2k to 200k particles and mixed materials (the batched benchmark).
        {"name": "batch_256", "kind": "batch", "scenes": 256, "n_min": 2000, "n_max": 200000, "mix": 1, "blocks": 16,
         "dt": 1e-4, "steps": 32},
        # The allocation-free call that plugins use, device arrays in and out.
        {"name": "noalloc_fluid", "kind": "noalloc", "material": "fluid", "shape": "box", "n": 24389, "blocks": 16,
         "boundary": "sticky_blocks", "layout": "lattice", "dt": 1e-4, "steps": 64},
        # A whole short job on a fresh scene: what the first frame of a program costs.
        {"name": "job_sand", "kind": "job", "material": "drucker_prager", "shape": "cylinder", "n": 210853, "blocks": 32,
         "boundary": "slip_floor", "layout": "lattice", "dt": 1e-4, "steps": 20},
        # The differentiable cube of the benchmark: forward and adjoint of 200 substeps, every substep kept.
        {"name": "diff_cube", "kind": "diff", "n": 50626, "blocks": 16, "layout": "lattice", "dt": 1e-4, "steps": 200, "every": 1},
        # A small differentiable rollout that recomputes from checkpoints (memory-limited training).
        {"name": "diff_recompute", "kind": "diff", "n": 7001, "blocks": 11, "layout": "random", "dt": 1e-4, "steps": 60, "every": 10},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _blocks_for(n, room):
    """Blocks per axis of a cubic domain that holds n particles at 8 per cell with the two-block walls."""
    side = (n / PPC) ** (1 / 3)
    return max(9, math.ceil((side * room + 20) / 4))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "adaptive", "batch", "noalloc", "job", "diff", "diff"])
    shape = rng.choice(["box", "sphere", "cylinder"])
    layout = rng.choice(["lattice", "lattice", "random"])
    if kind == "diff":
        n = int(_log(rng, 1500, 60000))
        return {"kind": "diff", "n": n, "blocks": rng.randint(max(7, _blocks_for(n, 1.0)), 20), "layout": layout, "dt": 1e-4,
                "steps": rng.randint(8, 120), "every": rng.choice([1, 1, 1, 4, 7])}
    if kind == "batch":
        scenes = int(_log(rng, 5, 256))
        n_max = int(_log(rng, 3000, 100000))
        return {"kind": "batch", "scenes": scenes, "n_min": max(300, int(n_max / rng.uniform(1.5, 60))), "n_max": n_max,
                "mix": rng.randrange(1 << 20), "blocks": rng.randint(max(13, _blocks_for(n_max, 1.6)), 18),
                "dt": 1e-4, "steps": rng.randint(4, 32)}
    top = {"frame": 4e6, "adaptive": 3e5, "noalloc": 50000, "job": 1e6}[kind]
    n = int(_log(rng, 1200, top))
    blocks = _blocks_for(n, {"box": 1.15, "sphere": 1.4, "cylinder": 2.25}[shape]) + rng.randint(0, 6)
    if kind == "noalloc":
        blocks = min(blocks, 16)
    material = rng.choice(["fixed_corotated", "fixed_corotated", "drucker_prager", "drucker_prager", "fluid", "fluid", "von_mises",
                           "nacc"] + ([] if kind == "noalloc" else ["linear"]))
    boundary = rng.choice(["sticky_blocks", "slip_floor"] + (["field"] if kind in ("frame", "adaptive") and n < 300000 else []))
    case = {"kind": kind, "material": material, "shape": shape, "n": n, "blocks": blocks, "boundary": boundary, "layout": layout,
            "dt": round(0.0064 / (4 * blocks), 8)}
    if kind == "adaptive":
        steps = rng.randint(6, 60)
        case.update(frame_time=round(case["dt"] * (steps - 0.5), 9), cfl=rng.choice([0.3, 0.5]),
                    rigid=n // 4 if material == "von_mises" and rng.random() < 0.5 else 0)
    else:
        case["steps"] = rng.randint(5, max(6, min(120, int(8e7 / n))))
    if material == "nacc":  # Cam-clay's hardening amplifies rounding: longer runs of it cannot be compared
        case["layout"] = "random"
        if kind != "adaptive":
            case["steps"] = min(case["steps"], 24)
    if kind in ("frame", "adaptive"):
        case["out"] = "state" if n < 200000 else "positions"
    return case


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _points(case, n, shape, center, gen, spacing):
    """n particles on the lattice sites nearest to `center` in the shape's own distance, jittered within their site
    ("lattice"), or uniform over the same sites in no order ("random"). Cell units."""
    dev = gen.device
    aspect = {"box": (1.0, 1.0, 1.0), "sphere": (1.0, 1.0, 1.0), "cylinder": (0.55, 1.5, 0.55), "slab": (0.6, 0.9, 1.55)}[shape]
    vol = {"sphere": 4 * math.pi / 3, "cylinder": 2 * math.pi}.get(shape, 8.0)
    r = (n / vol / (aspect[0] * aspect[1] * aspect[2])) ** (1 / 3)  # half extent along an axis of aspect 1, in sites
    half = [int(math.ceil(r * a * 1.06)) + 2 for a in aspect]
    axes = [torch.arange(-h, h, device=dev, dtype=torch.float32) for h in half]
    d = [((a + 0.5).abs() / s) for a, s in zip(axes, aspect)]
    dx, dy, dz = d[0][:, None, None], d[1][None, :, None], d[2][None, None, :]
    if shape == "sphere":
        metric = dx * dx + dy * dy + dz * dz
    elif shape == "cylinder":
        metric = torch.maximum(torch.sqrt(dx * dx + dz * dz), dy)
    else:
        metric = torch.maximum(torch.maximum(dx, dy), dz)
    metric = metric.reshape(-1)
    pick = torch.sort(metric, stable=True).indices[:n].sort().values
    ny, nz = 2 * half[1], 2 * half[2]
    site = torch.stack([pick // (ny * nz) - half[0], (pick // nz) % ny - half[1], pick % nz - half[2]], 1).to(torch.float32)
    if case["layout"] == "random":
        site = site[torch.randint(0, n, (n,), generator=gen, device=dev)]
    u = torch.rand((n, 3), generator=gen, device=dev)
    return (site + u) * spacing + torch.tensor(center, device=dev)


def _velocities(x, c, gen, swirl):
    """A smooth velocity field, v0 + G d + d (d . e) / R with d = x - c: the body moves and shears, one side of it is
    squeezed and the other pulled apart from the first substep, so every branch of a material's law is met."""
    dev = x.device
    v0 = torch.rand(3, generator=gen, device=dev) * 2 - 1
    G = (torch.rand((3, 3), generator=gen, device=dev) * 2 - 1) * swirl
    e = torch.randn(3, generator=gen, device=dev)
    d = x - c
    R = d.norm(dim=1).max()
    return (v0 + d @ G.T + d * (d @ (e / e.norm()))[:, None] * (swirl / R)).contiguous()


def _lame(E, nu):
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _material(kind, E=None, nu=None):
    """(MPMMaterial, density)"""
    if kind == "fluid":
        bulk, gamma, visc, rho = FLUID
        return MPMMaterial.fluid(bulk if E is None else E / gamma, gamma, visc), rho
    e, p, rho = ELASTIC[kind]
    lam, mu = _lame(e if E is None else E, p if nu is None else nu)
    if kind == "von_mises":
        return MPMMaterial.von_mises(mu, lam, 100.0), rho
    if kind == "nacc":
        return MPMMaterial.nacc(mu, lam, -0.01, 0.5, 0.8, 2.36, True), rho
    return getattr(MPMMaterial, kind)(lam, mu), rho


def _config(case):
    b = case["blocks"]
    cfg = MPMConfig(dx=1.0 / (4 * b), domain_blocks=(b, b, b), dt=case["dt"], boundary=case.get("boundary", "sticky_blocks"),
                    floor_cells=8.0, track_ids=True)
    if case.get("rigid"):
        cfg.exist_rigid_particle = True
        cfg.rigid_particle_count = case["rigid"]
        cfg.rigid_particle_velocity = (1.0, -0.5, 0.25)
    if cfg.boundary == "field":
        cfg.boundary_field = _field(4 * b)
    return cfg


def _field(m):
    """Slip walls two cells inside the two-block margin and a fixed box of cells in one corner."""
    rule = np.zeros((m, m, m), np.uint8)
    param = np.zeros((m, m, m, 3), np.float32)
    for axis in range(3):
        for lo in (True, False):
            at = [slice(None)] * 3
            at[axis] = slice(0, 9) if lo else slice(m - 9, m)
            rule[tuple(at)] = _capi.CELL_SLIP
            n = np.zeros(3, np.float32)
            n[axis] = 1.0 if lo else -1.0
            param[tuple(at)] = n
    rule[:12, :12, :12] = _capi.CELL_FIXED
    return rule.reshape(-1), param.reshape(-1, 3)


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _models(case, seed):
    """[{kind, x, v, mass, vol, material}] on the device, float32, and the scene's dx."""
    gen = _gen(seed)
    m = 4 * case["blocks"]
    dx = 1.0 / m
    spacing = round(PPC ** (1 / 3)) ** -1
    out = []

    def body(kind, shape, n, center, swirl):
        x = (_points(case, n, shape, center, gen, spacing) * dx).contiguous()
        c = torch.tensor([t * dx for t in center], device=x.device)
        mat, rho = _material(kind)
        vol = dx ** 3 / PPC
        out.append({"kind": kind, "x": x, "v": _velocities(x, c, gen, swirl), "mass": rho * vol, "vol": vol, "material": mat})

    if case.get("spheres"):
        cells = case["n"] / PPC
        half = [0.6, 0.9, 1.55]
        r = (cells / 8 / (half[0] * half[1] * half[2])) ** (1 / 3)
        body(case["material"], "slab", case["n"], [10 + r * half[0], 10 + r * half[1], m / 2], 0.5)
        x0 = 10 + 2 * r * half[0] + 14
        k = round(case["spheres"] ** (1 / 3))
        step = [(m - 12 - x0) / k, (m - 24) / k, (m - 24) / k]
        jit = torch.rand((k * k * k, 3), generator=gen, device=gen.device).cpu()
        xs, vs = [], []
        for i in range(k * k * k):
            cell = [i // (k * k), (i // k) % k, i % k]
            lo = [x0, 12, 12]
            c = [lo[a] + (cell[a] + 0.5 + 0.1 * (float(jit[i, a]) - 0.5)) * step[a] for a in range(3)]
            p = _points(case, case["sphere_n"], "sphere", c, gen, spacing) * dx
            xs.append(p)
            vs.append((torch.rand((1, 3), generator=gen, device=p.device) * 4 - 2).expand(len(p), 3))
        mat, rho = _material("fixed_corotated")
        vol = dx ** 3 / PPC
        out.append({"kind": "fixed_corotated", "x": torch.cat(xs).contiguous(), "v": torch.cat(vs).contiguous(), "mass": rho * vol,
                    "vol": vol, "material": mat})
    else:
        c = [m / 2 + float(t) for t in (torch.rand(3, generator=gen, device=gen.device) - 0.5).cpu()]
        if case.get("boundary") == "slip_floor":  # standing on the floor
            aspect = {"cylinder": 1.5}.get(case["shape"], 1.0)
            vol = {"sphere": 4 * math.pi / 3, "cylinder": 2 * math.pi * 0.55 * 0.55 * 1.5}.get(case["shape"], 8.0)
            c[1] = 8.6 + aspect * (case["n"] / PPC / vol) ** (1 / 3)
        body(case["material"], case["shape"], case["n"], c, 5.0)
    return out, dx


def _batch_models(case, seed):
    """One model a scene; sizes, shapes and materials come from the case, jitter and motion from the seed."""
    pick = random.Random(case["mix"])
    gen = _gen(seed)
    m = 4 * case["blocks"]
    dx = 1.0 / m
    spacing = round(PPC ** (1 / 3)) ** -1
    vol = dx ** 3 / PPC
    out = []
    for _ in range(case["scenes"]):
        n = int(_log(pick, case["n_min"], case["n_max"]))
        kind = pick.choice(["fixed_corotated", "fluid", "drucker_prager"])
        shape = pick.choice(["box", "sphere"])
        mat, rho = _material(kind, _log(pick, 1e4, 3e5), pick.uniform(0.2, 0.4))
        room = max(0.0, m - 24 - 2.1 * (n / PPC) ** (1 / 3) / (1.0 if shape == "sphere" else 2.0))
        c = [m / 2 + pick.uniform(-0.5, 0.5) * room * 0.8 for _ in range(3)]
        x = (_points({"layout": "lattice"}, n, shape, c, gen, spacing) * dx).contiguous()
        cc = torch.tensor([t * dx for t in c], device=x.device)
        out.append({"kind": kind, "x": x, "v": _velocities(x, cc, gen, 5.0), "mass": rho * vol, "vol": vol, "material": mat})
    return out, dx


def _host(t, pinned=False):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned and torch.cuda.is_available())
    h.copy_(t)
    return h.numpy()


def _diff_inputs(case, seed):
    gen = _gen(seed)
    m = 4 * case["blocks"]
    dx = 1.0 / m
    c = [m / 2 + float(t) for t in (torch.rand(3, generator=gen, device=gen.device) - 0.5).cpu()]
    x = (_points(case, case["n"], "box", c, gen, 0.5) * dx).contiguous()
    cc = torch.tensor([t * dx for t in c], device=x.device)
    v = _velocities(x, cc, gen, 5.0)
    n, dev = case["n"], x.device
    logE = (math.log(5e4) + 0.2 * torch.randn(n, generator=gen, device=dev)).contiguous()
    gx = torch.randn((n, 3), generator=gen, device=dev) / n
    gF = 0.01 * torch.randn((n, 3, 3), generator=gen, device=dev) / n
    vol = dx ** 3 / PPC
    return {"x0": x, "v0": v, "logE": logE, "gx": gx, "gF": gF, "mass": 1000.0 * vol, "vol": vol, "dx": dx}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "diff":
        d = _diff_inputs(case, seed)
        sim = DiffRollout(_config(case), case["n"], d["mass"], d["vol"], nu=0.3, nsteps=case["steps"], dt=case["dt"],
                          checkpoint_every=case["every"])
        for k in ("x0", "v0", "logE"):
            d[k].requires_grad_(True)
        return {"case": case, "sim": sim, **d}
    if kind == "batch":
        bodies, _ = _batch_models(case, seed)
        models = [MPMModel(b["mass"], b["vol"], _host(b["x"]), _host(b["v"]), b["material"]) for b in bodies]
        scene = SceneBatch(_config(case), models, _host(torch.cat([b["x"] for b in bodies]), True),
                           _host(torch.cat([b["v"] for b in bodies]), True))
        sizes = [sum(len(b["x"]) for b in bodies)]
        scene.setup()
        return _saved(case, scene, sizes)
    bodies, _ = _models(case, seed)
    cfg = _config(case)
    if kind == "noalloc":
        b = bodies[0]
        n = case["n"]
        dev = b["x"].device
        out = [torch.empty(s, device=dev) for s in ((n, 3), (n, 3), (n, 3, 3), (n,))]
        return {"case": case, "desc": cfg.to_c(), "mat": b["material"].to_c(), "body": b, "out": out, "lib": _capi.lib()}
    models = [MPMModel(b["mass"], b["vol"], _host(b["x"], True), _host(b["v"], True), b["material"]) for b in bodies]
    if kind == "job":
        return {"case": case, "cfg": cfg, "models": models,
                "x": [_host(torch.zeros_like(b["x"]), True) for b in bodies]}
    scene = Scene(cfg)
    for m in models:
        scene.add_model(m)
    scene.setup()
    return _saved(case, scene, [len(b["x"]) for b in bodies])


def _saved(case, scene, sizes):
    """The handle with its state saved, and pinned buffers where positions are exported."""
    saved = torch.empty(scene.checkpoint_bytes(), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    scene.checkpoint_save(saved.data_ptr())
    scene.status_check()
    st = {"case": case, "scene": scene, "saved": saved}
    if case.get("out", "positions") == "positions":
        st["x"] = [torch.empty((n, 3), pin_memory=True).numpy() for n in sizes]
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "diff":
        xT, FT = rollout(state["sim"], state["x0"], state["v0"], state["logE"])
        gx0, gv0, gE = torch.autograd.grad((xT, FT), (state["x0"], state["v0"], state["logE"]), (state["gx"], state["gF"]))
        return {"xT": xT.detach(), "FT": FT.detach(), "gx0": gx0, "gv0": gv0, "glogE": gE}
    if kind == "noalloc":
        b, out = state["body"], state["out"]
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        live, msg = C.c_uint32(), C.c_char_p()
        code = state["lib"].ckmpm_simulate_noalloc(
            C.byref(state["desc"]), C.byref(state["mat"]), case["n"], p(b["x"]), p(b["v"]), case["n"], b["mass"], b["vol"],
            case["steps"], case["dt"], C.c_void_p(torch.cuda.current_stream().cuda_stream), p(out[0]), p(out[1]), p(out[2]),
            p(out[3]), C.byref(live), C.byref(msg))
        if code:
            raise RuntimeError("ckmpm_simulate_noalloc: %s" % msg.value)
        return {"x": out[0], "v": out[1], "F": out[2], "aux": out[3], "live": live.value}
    if kind == "job":
        scene = Scene(state["cfg"])
        for m in state["models"]:
            scene.add_model(m)
        scene.setup()
        scene.step_async(case["steps"], case["dt"])
        for i, x in enumerate(state["x"]):
            scene.export_positions_async(i, x)
        scene.status_check()
        scene.export_wait()
        scene.close()
        return {"x": state["x"]}
    scene = state["scene"]
    scene.checkpoint_restore(state["saved"].data_ptr())
    if kind == "adaptive":
        scene.step_adaptive(1 << 20, case["dt"], case["cfl"], case["frame_time"])
    elif "x" in state:
        scene.step_async(case["steps"], case["dt"])
    else:
        scene.step(case["steps"], case["dt"])
    if "x" in state:
        for i, x in enumerate(state["x"]):
            scene.export_positions_async(i, x)
        if kind != "adaptive":
            scene.status_check()
        scene.export_wait()
        return {"x": state["x"]}
    s = scene.state(0)
    return {"x": s.x, "v": s.v, "F": s.F, "aux": s.aux, "id": s.id}


# ---------------------------------------------------------------- work and tolerance

STATE = {"fixed_corotated": 48, "drucker_prager": 52, "von_mises": 52, "nacc": 52, "linear": 84, "fluid": 16}
#: Operations of one particle and substep: both grids' G2P and P2G over 16 nodes, F, the stress with its SVD.
OPS = {"fixed_corotated": 1500, "drucker_prager": 1700, "von_mises": 1900, "nacc": 1900, "linear": 900, "fluid": 800}


def work(case):
    """Every substep reads and writes each particle's state once; the result is read out once."""
    if case["kind"] == "diff":
        n, k = case["n"], case["steps"]
        return {"bytes": n * k * (2 * 48 + 3 * 48), "flops": n * k * (1500 + 4500)}
    if case["kind"] == "batch":
        pick = random.Random(case["mix"])
        rows = []
        for _ in range(case["scenes"]):
            n = int(_log(pick, case["n_min"], case["n_max"]))
            kind = pick.choice(["fixed_corotated", "fluid", "drucker_prager"])
            pick.choice(["box", "sphere"])
            _log(pick, 1e4, 3e5)
            for _ in range(4):
                pick.uniform(0, 1)
            rows.append((kind, n))
    else:
        rows = [(case["material"], case["n"])]
        if case.get("spheres"):
            rows.append(("fixed_corotated", case["spheres"] * case["sphere_n"]))
    k = case.get("steps") or math.ceil(case["frame_time"] / case["dt"])
    out = 12 if case.get("out", "positions") == "positions" and case["kind"] != "noalloc" else 68
    return {"bytes": sum(n * (2 * STATE[m] * k + out) for m, n in rows), "flops": sum(n * OPS[m] * k for m, n in rows)}


def tolerance(case):
    """About four times the distance between the engine and the 64-bit restatement, measured over the ranges of draw()
    (float32 state throughout): positions 0.6-7e-7, diff gradients 6e-5, log Jp of sand 8e-4 (its sign decides the
    branch) and of Cam-clay 9e-3 (its hardening amplifies rounding), elastic and fluid velocities 2e-6."""
    if case["kind"] == "diff":
        return {"rel": 3e-4, "max": 0.02}
    if case["kind"] in ("batch", "job") or case.get("out") == "positions":
        return {"rel": 4e-6, "max": 5e-5}
    if case["material"] == "nacc":
        return {"rel": 3e-2, "max": 0.99}
    if case["material"] == "drucker_prager":
        return {"rel": 3e-3, "max": 0.05}
    if case["material"] == "von_mises":
        return {"rel": 1e-4, "max": 1e-3}
    return {"rel": 1e-5, "max": 1e-4}


# ---------------------------------------------------------------- the same in 64 bits


def _f32(v):
    return float(np.float32(v))


def _mm(a, b):
    """Products of [n, 3, 3] matrices."""
    return (a[:, :, :, None] * b[:, None, :, :]).sum(2)


def _det(F):
    return (F[:, 0, 0] * (F[:, 1, 1] * F[:, 2, 2] - F[:, 1, 2] * F[:, 2, 1])
            - F[:, 0, 1] * (F[:, 1, 0] * F[:, 2, 2] - F[:, 1, 2] * F[:, 2, 0])
            + F[:, 0, 2] * (F[:, 1, 0] * F[:, 2, 1] - F[:, 1, 1] * F[:, 2, 0]))


def _cof(F):
    """Cofactor matrix: F^-T times det F."""
    r0, r1, r2 = F[:, 0], F[:, 1], F[:, 2]
    return torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0), torch.linalg.cross(r0, r1)], 1)


def _inv(F):
    return _cof(F).transpose(1, 2) / _det(F)[:, None, None]


def _eig(M):
    """Eigenvalues [n, 3] and eigenvectors [n, 3, 3] (columns) of symmetric matrices: cyclic Jacobi to convergence."""
    m = [[M[:, i, j].clone() for j in range(3)] for i in range(3)]
    one, zero = torch.ones_like(m[0][0]), torch.zeros_like(m[0][0])
    V = [[one.clone() if i == j else zero.clone() for j in range(3)] for i in range(3)]
    for _ in range(7):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            a = m[p][q]
            d, e = m[q][q] - m[p][p], 2 * a
            den = d + torch.copysign(torch.sqrt(d * d + e * e), d)
            t = torch.where(den.abs() > 1e-300, e / torch.where(den.abs() > 1e-300, den, one), zero)
            c = torch.rsqrt(1 + t * t)
            s = t * c
            m[p][p], m[q][q] = m[p][p] - t * a, m[q][q] + t * a
            rp, rq = m[r][p], m[r][q]
            m[r][p] = m[p][r] = c * rp - s * rq
            m[r][q] = m[q][r] = s * rp + c * rq
            m[p][q] = m[q][p] = zero
            for k in range(3):
                vp, vq = V[k][p], V[k][q]
                V[k][p], V[k][q] = c * vp - s * vq, s * vp + c * vq
    return torch.stack([m[0][0], m[1][1], m[2][2]], 1), torch.stack([torch.stack(r, 1) for r in V], 1)


def _svd(F):
    """U, S, V with F = U diag(S) V^T, S > 0 (every F here keeps a positive determinant)."""
    lam, V = _eig(_mm(F.transpose(1, 2), F))
    S = torch.sqrt(lam)
    return _mm(F, V) / S[:, None, :], S, V


def _udu(U, d, W):
    return _mm(U * d[:, None, :], W.transpose(1, 2))


def _stress(g, F, aux, Q, C3, dt):
    """(F, aux, Q, tau) of group g after the trial update, in 64 bits."""
    kind, eye = g["kind"], torch.eye(3, dtype=C3.dtype, device=C3.device)
    p = g["p"]
    if kind == "fluid":
        bulk, gamma, visc = p[0], p[1], p[2]
        tr = C3[:, 0, 0] + C3[:, 1, 1] + C3[:, 2, 2]
        J = aux + tr * dt * aux
        pr = bulk * (J ** (-gamma) - 1)
        return F, J, Q, J[:, None, None] * ((C3 + C3.transpose(1, 2)) * _col(visc) - _col(pr) * eye)
    F = _mm(eye + dt * C3, F)
    if kind == "linear":
        t = 50.0 * (C3 + C3.transpose(1, 2) - eye) * dt
        q = (Q + t) * _det(F)[:, None, None]
        q[:, 1:] = 0
        return F, aux, q, q
    U, S, V = _svd(F)
    if kind == "fixed_corotated":
        lam, mu = p[0], p[1]
        J = S.prod(1)
        return F, aux, Q, _udu(U, 2 * _one(mu) * S * (S - 1) + _one(lam * J * (J - 1)), U)
    if kind == "drucker_prager":
        lam, mu = p[0], p[1]
        ys = math.sqrt(2.0 / 3.0) * 2.0 * 0.5 / (3.0 - 0.5)
        eps = torch.log(S.clamp(min=1e-4))
        etr = eps.sum(1) + aux
        eh = eps - etr[:, None] / 3
        ehn = torch.sqrt((eh * eh).sum(1))
        dg = ehn + (3 * lam + 2 * mu) / (2 * mu) * etr * ys
        H = torch.where((dg <= 0)[:, None], eps, eps - (dg / ehn.clamp(min=1e-300))[:, None] * eh)
        tension = etr >= 0
        H = torch.where(tension[:, None], torch.zeros_like(H), H)
        aux = torch.where(tension, etr, torch.zeros_like(aux))
        return _udu(U, torch.exp(H), V), aux, Q, _udu(U, 2 * _one(mu) * H + _one(lam * H.sum(1)), U)
    if kind == "von_mises":
        mu, lam, yld = p[0], p[1], p[2]
        eps = torch.log(S)
        eh = eps - eps.sum(1, keepdim=True) / 3
        ehn = torch.sqrt((eh * eh).sum(1))
        yf = ehn - yld / (2 * mu)
        flow = yf > 0
        H = torch.where(flow[:, None], eps - (yf / ehn.clamp(min=1e-300))[:, None] * eh, eps)
        F = torch.where(flow[:, None, None], _udu(U, torch.exp(H), V), F)
        return F, aux, Q, _udu(U, 2 * _one(mu) * H + _one(lam * H.sum(1)), U)
    # Cam-clay (F is kept up to a rotation on the right: only F F^T matters)
    mu, lam, beta, xi, msq, hard = p[0], p[1], p[3], p[4], p[5] ** 2, p[6] != 0
    K = 2 * mu / 3 + lam
    p0 = K * (1e-5 + torch.sinh(xi * (-aux).clamp(min=0)))
    pmin = -beta * p0
    je = S.prod(1)
    bh = S * S
    btr3 = bh.sum(1) / 3
    devf = mu * je ** (-2.0 / 3)
    sh = devf[:, None] * (bh - btr3[:, None])
    ptr = -K * 0.5 * (je - 1 / je) * je
    ysh = 1.5 * (1 + 2 * beta)
    yph = msq * (ptr - pmin) * (ptr - p0)
    sn2 = (sh * sh).sum(1)
    y = ysh * sn2 + yph
    clamp = (ptr > p0) | (ptr < pmin)
    pp = torch.where(ptr > p0, p0, pmin)
    jn = torch.sqrt(-2 * pp / K + 1)
    S1 = (jn ** (1.0 / 3))[:, None].expand_as(S)
    a1 = aux + (torch.log(je / jn) if hard else 0)
    surf = ~clamp & (y >= 1e-4)
    coef = je ** (2.0 / 3) / mu * torch.sqrt((-yph / ysh).clamp(min=0)) / torch.sqrt(sn2.clamp(min=1e-300))
    S2 = torch.sqrt((sh * coef[:, None] + btr3[:, None]).clamp(min=1e-300))
    pc = (1 - beta) * p0 / 2
    d0, d1 = pc - ptr, -torch.sqrt(1.5 * sn2)
    dn = torch.sqrt(d0 * d0 + d1 * d1).clamp(min=1e-300)
    d0, d1 = d0 / dn, d1 / dn
    A = msq * d0 * d0 + (1 + 2 * beta) * d1 * d1
    B = msq * d0 * (2 * pc - p0 - pmin)
    Cc = msq * (pc - pmin) * (pc - p0)
    root = torch.sqrt((B * B - 4 * A * Cc).clamp(min=0))
    safe = torch.where(A.abs() > 1e-300, A, torch.ones_like(A))
    p1, p2 = pc + (-B + root) / (2 * safe) * d0, pc + (-B - root) / (2 * safe) * d0
    pf = torch.where((ptr - pc) * (p1 - pc) > 0, p1, p2)
    jn2 = torch.sqrt((-2 * pf / K + 1).abs())
    moves = surf & hard & (p0 > 1e-4) & (ptr < p0 - 1e-4) & (ptr > 1e-4 + pmin) & (jn2 > 1e-4)
    a2 = aux + torch.where(moves, 9 * torch.log(je / jn2.clamp(min=1e-300)), torch.zeros_like(aux))
    Sn = torch.where(clamp[:, None], S1, torch.where(surf[:, None], S2, S))
    F = torch.where((clamp | surf)[:, None, None], _udu(U, Sn, V), F)
    aux = torch.where(clamp, a1, torch.where(surf, a2, aux))
    b = _mm(F, F.transpose(1, 2))
    J = Sn.prod(1)
    tr3 = (b[:, 0, 0] + b[:, 1, 1] + b[:, 2, 2]) / 3
    return F, aux, Q, devf[:, None, None] * (b - tr3[:, None, None] * eye) + (K * 0.5 * (J * J - 1))[:, None, None] * eye


def _one(v):
    """A scalar or per-particle value against [n, 3]."""
    return v[:, None] if torch.is_tensor(v) else v


def _col(v):
    """A scalar or per-particle value against [n, 3, 3]."""
    return v[:, None, None] if torch.is_tensor(v) else v


class _Grid:
    """Both staggered grids of `scenes` stacked domains, the CK weights and the transfers, in 64 bits."""

    def __init__(self, cells, scenes, dx, cfg, device):
        self.m, self.scenes, self.dx, self.cfg, self.dev = cells, scenes, dx, cfg, device
        self.inv = _f32(1.0 / dx)
        self.nodes = 2 * scenes * cells ** 3
        k = torch.arange(cells, device=device)
        b = k // 4
        nb = cells // 4
        edge = (b < 2) | (b + 2 >= nb)
        ex, ey, ez = edge[:, None, None], edge[None, :, None], edge[None, None, :]
        top = (b + 2 >= nb)[None, :, None]
        self.floor = None
        if cfg.boundary == "sticky_blocks":
            self.out = ex | ey | ez
        elif cfg.boundary == "slip_floor":
            self.out = (ex | ez | top).expand(cells, cells, cells)
            self.floor = ((k.to(torch.float64) < cfg.floor_cells)[None, :, None] & ~self.out)
        else:
            self.out = None
            rule, param = cfg.boundary_field
            self.rule = torch.as_tensor(rule, device=device).long().reshape(cells, cells, cells)
            self.param = torch.as_tensor(param, device=device).double().reshape(cells, cells, cells, 3)

    def stencil(self, x):
        """Per grid: base cell [n, 3] and offset [n, 3]."""
        xs = x * self.inv
        got = []
        for g in (-1.0, 1.0):
            base = torch.trunc(xs.detach() - 0.25 * g)
            got.append((base.long(), xs - base - 0.25 * g))
        return got

    def nodes_of(self, x, w):
        """Yields (flat node index, weight, offset from the particle in world units) of the 16 nodes; and D."""
        D = torch.zeros(len(x), 3, 3, dtype=torch.float64, device=self.dev)
        rows = []
        for g, (base, o) in enumerate(self.stencil(x)):
            w0 = 1 - o + torch.sin(2 * math.pi * o) / (2 * math.pi)
            ws = (w0, 1 - w0)
            for n in range(8):
                d = ((n >> 2) & 1, (n >> 1) & 1, n & 1)
                wt = ws[d[0]][:, 0] * ws[d[1]][:, 1] * ws[d[2]][:, 2]
                c = base + torch.tensor(d, device=self.dev)
                flat = (((w * 2 + g) * self.m + c[:, 0]) * self.m + c[:, 1]) * self.m + c[:, 2]
                r = (torch.tensor(d, dtype=torch.float64, device=self.dev) - o) * self.dx
                D = D + wt[:, None, None] * r[:, :, None] * r[:, None, :]
                rows.append((flat, wt, r))
        return rows, D

    def velocity(self, grid, dt):
        """Node velocities after the grid update of [nodes, 4] masses and momenta."""
        m = grid[:, 0]
        live = m > self.cfg.mass_clamp
        v = grid[:, 1:] / torch.where(live, m, torch.ones_like(m))[:, None]
        v = v + torch.tensor([0.0, self.cfg.gravity * dt, 0.0], dtype=torch.float64, device=self.dev)
        v = torch.where(live[:, None], v, torch.zeros_like(v))
        shape = (2 * self.scenes, self.m, self.m, self.m, 3)
        v = v.reshape(shape)
        if self.out is not None:
            v = torch.where(self.out[None, ..., None], torch.zeros_like(v), v)
            if self.floor is not None:
                y = torch.where(self.floor[None], v[..., 1].clamp(min=0), v[..., 1])
                v = torch.stack([v[..., 0], y, v[..., 2]], -1)
        else:
            n = self.param[None]
            dot = (v * n).sum(-1, keepdim=True)
            r = self.rule[None, ..., None]
            v = torch.where(r == 1, torch.zeros_like(v), v)
            v = torch.where((r == 2) | ((r == 4) & (dot < 0)), v - dot * n, v)
            v = torch.where((r == 3) & live.reshape(shape[:-1])[..., None], n.expand_as(v), v)
        return v.reshape(-1, 3)

    def gather(self, vel, x, w):
        """v, C = B D^-1 and D of the G2P at x."""
        rows, D = self.nodes_of(x, w)
        v = torch.zeros_like(x)
        B = torch.zeros_like(D)
        for flat, wt, r in rows:
            wv = vel.index_select(0, flat) * wt[:, None]
            v = v + wv
            B = B + wv[:, :, None] * r[:, None, :]
        return 0.5 * v, _mm(B, _inv(D)), D

    def scatter(self, grid, x, w, mass, v, tau, C3, D, ndt, vol):
        """Adds the P2G of particles at x to grid [nodes, 4]; D is the G2P's. Returns the grid."""
        rows, Dn = self.nodes_of(x, w)
        A = None
        if tau is not None:
            A = C3 - _col(ndt * vol / mass) * _mm(_inv(0.5 * (D + Dn)), tau)
        for flat, wt, r in rows:
            u = v if A is None else v + (A * r[:, None, :]).sum(2)
            grid = grid.index_add(0, flat, torch.cat([torch.ones_like(wt)[:, None], u], 1) * (mass * wt)[:, None])
        return grid


def _params(mat):
    return [_f32(v) for v in mat.params()]


def _simulate(case, groups, cfg, dx, scenes):
    """Runs groups of particles (dicts of kind, p, x, v, w, mass, vol) in 64 bits; leaves x, F, aux, vel in them."""
    dev = groups[0]["x"].device
    G = _Grid(4 * case["blocks"], scenes, dx, cfg, dev)
    chunk = 1 << 21
    dt0 = _f32(case["dt"])

    def parts(n):
        return [slice(i, min(n, i + chunk)) for i in range(0, n, chunk)]

    def at(v, s):
        return v[s] if torch.is_tensor(v) and v.dim() else v

    grid = torch.zeros(G.nodes, 4, dtype=torch.float64, device=dev)
    for g in groups:
        n = len(g["x"])
        g["F"] = torch.eye(3, dtype=torch.float64, device=dev).expand(n, 3, 3).contiguous() if g["kind"] != "fluid" else None
        g["Q"] = torch.zeros(n, 3, 3, dtype=torch.float64, device=dev) if g["kind"] == "linear" else None
        start = {"fluid": lambda: g["p"][3], "nacc": lambda: g["p"][2], "von_mises": lambda: 1.0}.get(g["kind"], lambda: 0.0)()
        g["aux"] = torch.zeros(n, dtype=torch.float64, device=dev) + start
        g["rigid"] = None
        if case.get("rigid") and g["kind"] == "von_mises":
            g["aux"][:case["rigid"]] = 0.0
            g["rigid"] = (g["aux"] == 0)
        for s in parts(n):
            grid = G.scatter(grid, g["x"][s], g["w"][s], at(g["mass"], s), g["v"][s], None, None, None, 0.0, None)
    rigid_v = torch.tensor([_f32(c) for c in cfg.rigid_particle_velocity], dtype=torch.float64, device=dev) if case.get("rigid") else None
    cur, time = 0.0, 0.0
    end = case.get("frame_time")
    lightest = min(float(g["mass"].min()) if torch.is_tensor(g["mass"]) else g["mass"] for g in groups)
    done = 0
    while (done < case["steps"]) if end is None else (end - time > 0):
        vel = G.velocity(grid, cur)
        nxt = dt0
        if end is not None:
            heavy = grid[:, 0] > max(cfg.mass_clamp, lightest * 2.0 ** -16)
            vmax = math.sqrt(float((vel * vel).sum(1)[heavy].max()))
            nxt = min(dt0, end - time)
            if vmax > 0:
                nxt = min(nxt, dx * _f32(case["cfl"]) / vmax)
        nxt32 = _f32(nxt)
        grid = torch.zeros_like(grid)
        for g in groups:
            for s in parts(len(g["x"])):
                x, w = g["x"][s], g["w"][s]
                v, C3, D = G.gather(vel, x, w)
                adv = v
                if g["rigid"] is not None:
                    r = g["rigid"][s]
                    C3 = torch.where(r[:, None, None], torch.zeros_like(C3), C3)
                    D = torch.where(r[:, None, None], torch.zeros_like(D), D)
                    v = torch.where(r[:, None], torch.zeros_like(v), v)
                    adv = torch.where(r[:, None], rigid_v.expand_as(v), v)
                x = x + _f32(cur) * adv
                part = {**g, "p": [at(q, s) for q in g["p"]]}
                F, aux, Q, tau = _stress(part, None if g["F"] is None else g["F"][s], g["aux"][s],
                                         None if g["Q"] is None else g["Q"][s], C3, _f32(cur))
                g["x"][s], g["aux"][s] = x, aux
                if g["F"] is not None:
                    g["F"][s] = F
                if g["Q"] is not None:
                    g["Q"][s] = Q
                grid = G.scatter(grid, x, w, at(g["mass"], s), v, tau, C3, D, nxt32, at(g["vol"], s))
        cur = nxt
        time += nxt
        done += 1
    vel = G.velocity(grid, _f32(cur))
    for g in groups:
        g["vel"] = torch.cat([G.gather(vel, g["x"][s], g["w"][s])[0] for s in parts(len(g["x"]))])
        if g["rigid"] is not None:
            g["vel"][g["rigid"]] = 0.0


def _polar(F):
    """Rotation of the polar decomposition by Newton's iteration (differentiable: it converges quadratically)."""
    R = F
    for _ in range(7):
        R = 0.5 * (R + _cof(R) / _det(R)[:, None, None])
    return R


def _exact_diff(case, seed):
    from torch.utils.checkpoint import checkpoint

    d = _diff_inputs(case, seed)
    dev = d["x0"].device
    dx = _f32(d["dx"])
    G = _Grid(4 * case["blocks"], 1, dx, _config(case), dev)
    x0, v0, logE = (d[k].double().requires_grad_(True) for k in ("x0", "v0", "logE"))
    E = torch.exp(logE)
    nu = _f32(0.3)
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    mass, vol, dt = _f32(d["mass"]), _f32(d["vol"]), _f32(case["dt"])
    w = torch.zeros(case["n"], dtype=torch.long, device=dev)
    eye = torch.eye(3, dtype=torch.float64, device=dev)

    def substep(grid, x, F, lam, mu, cur):
        vel = G.velocity(grid, cur)
        v, C3, D = G.gather(vel, x, w)
        x = x + cur * v
        F = _mm(eye + cur * C3, F)
        J = _det(F)
        tau = 2 * _col(mu) * _mm(F - _polar(F), F.transpose(1, 2)) + _col(lam * J * (J - 1)) * eye
        return G.scatter(torch.zeros_like(grid), x, w, mass, v, tau, C3, D, dt, vol), x, F

    grid = torch.zeros(G.nodes, 4, dtype=torch.float64, device=dev)
    grid = G.scatter(grid, x0, w, mass, v0, None, None, None, 0.0, None)
    x, F = x0, eye.expand(case["n"], 3, 3).contiguous()
    for s in range(case["steps"]):
        grid, x, F = checkpoint(substep, grid, x, F, lam, mu, 0.0 if s == 0 else dt, use_reentrant=False)
    gx0, gv0, gE = torch.autograd.grad((x, F), (x0, v0, logE), (d["gx"].double(), d["gF"].double()))
    return {"xT": x.detach(), "FT": F.detach(), "gx0": gx0, "gv0": gv0, "glogE": gE}


def exact(case, seed):
    if case["kind"] == "diff":
        if case["n"] * case["steps"] > 1.2e7:
            return None
        return _exact_diff(case, seed)
    cfg = _config(case)
    batch = case["kind"] == "batch"
    bodies, dx = _batch_models(case, seed) if batch else _models(case, seed)
    dx = _f32(dx)
    groups = []
    with torch.no_grad():
        if batch:
            sizes = [len(b["x"]) for b in bodies]
            at = np.concatenate([[0], np.cumsum(sizes)])
            for kind in ("fixed_corotated", "fluid", "drucker_prager"):
                mine = [i for i, b in enumerate(bodies) if b["kind"] == kind]
                if not mine:
                    continue
                dev = bodies[0]["x"].device
                each = torch.tensor([sizes[i] for i in mine], device=dev)
                spread = lambda vals: torch.tensor(vals, dtype=torch.float64, device=dev).repeat_interleave(each)  # noqa: B023,E731
                ps = [_params(bodies[i]["material"]) for i in mine]
                groups.append({"kind": kind, "p": [spread([p[k] for p in ps]) for k in range(4)],
                               "x": torch.cat([bodies[i]["x"] for i in mine]).double(),
                               "v": torch.cat([bodies[i]["v"] for i in mine]).double(),
                               "w": torch.tensor(mine, device=dev).repeat_interleave(each),
                               "mass": spread([_f32(bodies[i]["mass"]) for i in mine]),
                               "vol": spread([_f32(bodies[i]["vol"]) for i in mine]),
                               "to": torch.cat([torch.arange(int(at[i]), int(at[i + 1]), device=dev) for i in mine])})
            _simulate(case, groups, cfg, dx, case["scenes"])
            x = torch.empty(int(at[-1]), 3, dtype=torch.float64, device=groups[0]["x"].device)
            for g in groups:
                x[g["to"]] = g["x"]
            return {"x": [x]}
        for b in bodies:
            n = len(b["x"])
            groups.append({"kind": b["kind"], "p": _params(b["material"]), "x": b["x"].double(), "v": b["v"].double(),
                           "w": torch.zeros(n, dtype=torch.long, device=b["x"].device), "mass": _f32(b["mass"]), "vol": _f32(b["vol"])})
        del bodies
        _simulate(case, groups, cfg, dx, 1)
        if case["kind"] == "job" or case.get("out") == "positions":
            return {"x": [g["x"] for g in groups]}
        g = groups[0]
        n = len(g["x"])
        if g["kind"] == "fluid":
            F = torch.eye(3, dtype=torch.float64, device=g["x"].device).expand(n, 3, 3)
        else:
            F = None if g["kind"] == "nacc" else g["F"]  # Cam-clay keeps F up to a rotation on the right
        got = {"x": g["x"], "v": g["vel"], "F": F, "aux": g["aux"]}
        got["live" if case["kind"] == "noalloc" else "id"] = None
        return got
