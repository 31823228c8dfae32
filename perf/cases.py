"""The work that programs using this framework have it do, as cases that can be timed and compared.

Each case is a dict of plain values; `prepare` makes what a program has in hand before the call,
`run` is one pass through the public entry points, `work` the bytes and operations a pass cannot do
without, `exact` the same outputs in 64-bit arithmetic written here in plain torch.

Kinds of case:
  world      one scene on the device: upload, a number of substeps, download (device arrays)
  batched    many scenes in one world, the same three calls for all of them at once
  pipelined  the host-to-host batch call, scenes in groups whose copies overlap other groups' substeps
  served     requests through the continuous-batching server, submit to results in host buffers
  near       the engine's near-field call on host MpssBuffer arrays (reference mode, full state)
  mid        the engine's mid-field call on host MpssBuffer arrays (velocity only)
  ck         the CK-MPM solver on device records
  tick       the engine tick's passes around the substep on device arrays
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ae-engine_b200"))
import ae_mpm as M  # noqa: E402
import ae_mpm_scenes as S  # noqa: E402

FIELDS = ("pos", "vel", "F", "J", "C", "mass", "mat")
WIDTH = {"pos": 3, "vel": 3, "F": 9, "J": 1, "C": 9, "mass": 1, "mat": 1}


def listed():
    return [
        # the smallest scenes a program steps: a handful of blocks, launches and latency are all there is
        {"name": "world_water_2k", "kind": "world", "scene": "water", "grid": 32, "particles": 2309, "substeps": 50,
         "sort_interval": 1, "deterministic": False},
        # the plain single-scene configuration, with the library's default options
        {"name": "world_jelly_32k", "kind": "world", "scene": "jelly", "grid": 64, "particles": 32768, "substeps": 60,
         "sort_interval": 1, "deterministic": False},
        # two snow bodies in collision, part of the particles yielding, with the options the autotuner picks for it
        {"name": "world_snow_1m", "kind": "world", "scene": "snow", "grid": 128, "particles": 1048576, "substeps": 40,
         "sort_interval": 16, "deterministic": False},
        # the largest single scene: the mixed-material dam break
        {"name": "world_dam_8m", "kind": "world", "scene": "dam", "grid": 256, "particles": 8388608, "substeps": 16,
         "sort_interval": 16, "deterministic": False},
        # lockstep replay: the same scene at an eighth of the size in the bitwise reproducible mode
        {"name": "world_dam_1m_replay", "kind": "world", "scene": "dam", "grid": 128, "particles": 1000003,
         "substeps": 12, "sort_interval": 1, "deterministic": True},
        # the batched configuration: 512 uneven scenes stepped together on the device
        {"name": "batched_512", "kind": "batched", "scenes": 512, "substeps": 32, "sort_interval": 16, "plan": 4},
        # a batch of host-resident scenes advanced and returned in one call
        {"name": "pipelined_96", "kind": "pipelined", "scenes": 96, "substeps": 60, "groups": 8, "plan": 7},
        # a burst of requests through the server
        {"name": "served_40", "kind": "served", "requests": 40, "least": 20, "most": 120, "plan": 11},
        # the engine's near-field tick: a sparse ascending list out of a large buffer
        {"name": "near_10k", "kind": "near", "selected": 10000, "capacity": 1000055},
        # the engine's mid-field tick: half of the buffer, position and velocity only
        {"name": "mid_490k", "kind": "mid", "selected": 490045, "capacity": 1000055},
        # the CK-MPM elastic block
        {"name": "ck_2m", "kind": "ck", "particles": 2097152, "grid": 128, "h": 1.0, "steps": 10},
        # LOD, far field, coarse field and housekeeping of one engine tick
        {"name": "tick_1m", "kind": "tick", "particles": 1048576, "max_near": 10000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("world", "world", "world", "batched", "pipelined", "served", "near", "mid", "ck", "tick"))
    if kind == "world":
        scene = rng.choice(("water", "jelly", "snow", "dam"))
        if scene == "dam":  # the dam's bodies fill a fixed share of the domain: 4 to 8 particles per cell
            grid = rng.choice((96, 128, 160, 192))
            n = int(grid ** 3 * rng.uniform(0.25, 0.5))
        else:
            grid = rng.choice((32, 48, 64, 96, 128))
            n = _log_int(rng, 1500, min(1 << 20, grid ** 3 // 2))
        return {"kind": kind, "scene": scene, "grid": grid, "particles": n, "substeps": rng.randint(12, 60 if n < 300000 else 24),
                "sort_interval": rng.choice((1, 8, 16)), "deterministic": rng.random() < 0.2}
    if kind == "batched":
        return {"kind": kind, "scenes": _log_int(rng, 16, 384), "substeps": rng.randint(16, 40),
                "sort_interval": rng.choice((1, 8, 16)), "plan": rng.randint(20, 1 << 20)}
    if kind == "pipelined":
        return {"kind": kind, "scenes": rng.randint(24, 96), "substeps": rng.randint(20, 80), "groups": rng.randint(2, 8),
                "plan": rng.randint(20, 1 << 20)}
    if kind == "served":
        return {"kind": kind, "requests": rng.randint(8, 40), "least": 20, "most": rng.randint(60, 140),
                "plan": rng.randint(20, 1 << 20)}
    if kind == "near":
        n = _log_int(rng, 1000, 60000)
        return {"kind": kind, "selected": n, "capacity": max(n, _log_int(rng, 100000, 1000055))}
    if kind == "mid":
        n = _log_int(rng, 60000, 490045)
        return {"kind": kind, "selected": n, "capacity": int(n * rng.uniform(1.1, 3.0))}
    if kind == "ck":
        return {"kind": kind, "particles": _log_int(rng, 20000, 2097152), "grid": 128, "h": rng.choice((1.0, 0.999, 0.7)),
                "steps": rng.randint(4, 10)}
    return {"kind": kind, "particles": _log_int(rng, 50000, 1048576), "max_near": _log_int(rng, 2000, 20000)}


# ------------------------------------------------------------------------------------------------
# scenes
# ------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)


def _time_step(grid):
    return 1e-4 if grid <= 64 else 5e-5 if grid <= 128 else 2e-5

# small matrices, one per particle, without a batched-library call each
def _mv(a, d):
    return (a * d[:, None, :]).sum(2)


def _mm(a, b):
    return (a[:, :, :, None] * b[:, None, :, :]).sum(2)


def _cofactor(f):
    """Cofactor matrix, det(F) F^-T."""
    return torch.stack([torch.linalg.cross(f[:, (i + 1) % 3], f[:, (i + 2) % 3], dim=1) for i in range(3)], 1)


def _det(f):
    return (f[:, 0] * torch.linalg.cross(f[:, 1], f[:, 2], dim=1)).sum(1)


MATERIAL = {"jelly": S.jelly, "snow": S.snow, "water": S.water}


def _batch_scene(rng):
    """(grid, particles, material) of one scene of the batched population."""
    return rng.choice((32, 48, 64)), _log_int(rng, 2048, 65536), rng.choice(("jelly", "snow", "water"))


def _scenes(case):
    """The scenes of a case as dicts: grid, dt, materials, substeps and the bodies in it.  A body is
    (lower corner, side, particles, material index, material kind, base velocity, on a lattice)."""
    kind = case["kind"]
    if kind == "world":
        grid, n, scene = case["grid"], case["particles"], case["scene"]
        if scene == "dam":
            base, nw, ne = 4.0 / grid, int(n * 0.60), int(n * 0.25)
            side, sside = 0.198, 0.21
            bodies = [((base,) * 3, (0.5, 0.375, 0.2), nw, 0, "water", (0, 0, 0), False),
                      ((0.6, base, 0.1), (side,) * 3, ne // 2, 1, "jelly", (0, 0, 0), False),
                      ((0.6, base, 0.5), (side,) * 3, ne - ne // 2, 1, "jelly", (0, 0, 0), False),
                      ((0.3, 0.5, 0.3), (sside,) * 3, n - nw - ne, 2, "snow", (0, -1.0, 0), False)]
            mats = [S.water(K=1e4, rho=1000.0), S.jelly(E=1e5, nu=0.3, rho=1000.0), S.snow()]
        elif scene == "snow":  # about 31 particles per cell in two bodies about to touch
            side = min((n / 2 / 31.0) ** (1 / 3) / grid, 0.4)
            lo, gap = 0.5 - side / 2, 0.25 / grid
            bodies = [((0.5 - gap - side, lo, lo), (side,) * 3, n // 2, 0, "snow", (2, 0, 0), True),
                      ((0.5 + gap, lo, lo), (side,) * 3, n - n // 2, 0, "snow", (-2, 0, 0), True)]
            mats = [S.snow()]
        else:
            ppc = 15.6 if scene == "jelly" else 8.0
            side = min((n / ppc) ** (1 / 3) / grid, 1.0 - 10.0 / grid)
            bodies = [((0.5 - side / 2,) * 3, (side,) * 3, n, 0, scene, (0, 0, 0), scene == "jelly")]
            mats = [MATERIAL[scene]()]
        return [{"grid": grid, "dt": _time_step(grid), "mats": mats, "bodies": bodies, "substeps": case["substeps"]}]
    rng, out = random.Random(case["plan"]), []
    for _ in range(case["requests"] if kind == "served" else case["scenes"]):
        grid, n, mat = _batch_scene(rng)
        side = min((n / 8.0) ** (1 / 3) / grid, 1.0 - 10.0 / grid)
        lo = tuple(5.0 / grid + rng.random() * max(1.0 - 10.0 / grid - side, 0.0) for _ in range(3))
        v = tuple(rng.uniform(-1, 1) for _ in range(3))
        steps = rng.randint(case["least"], case["most"]) if kind == "served" else case["substeps"]
        out.append({"grid": grid, "dt": _time_step(grid), "mats": [MATERIAL[mat]()],
                    "bodies": [(lo, (side,) * 3, n, 0, mat, v, False)], "substeps": steps})
    return out


def _count(scene):
    return sum(b[2] for b in scene["bodies"])


def _lattice(gen, lo, side, n):
    """n positions in a box in lattice order, one or more jittered in each of m^3 sub-cells."""
    m = max(1, int(round(n ** (1 / 3))))
    while m > 1 and n % m ** 3:
        m -= 1
    if m ** 3 * 64 < n:  # n has no cube to speak of: the first n of the next larger lattice
        m, k = int(math.ceil(n ** (1 / 3))), 1
    else:
        k = n // m ** 3
    i = torch.arange(n, device="cuda") // k
    cell = torch.stack((i // (m * m), i // m % m, i % m), 1).double()
    return lo + (cell + _rand(gen, n, 3)) * (side / m)


def _particles(case, seed, scenes):
    """All scenes' particles one after another, as device tensors: bodies in motion and under load,
    with the APIC matrix of their velocity field and a deformation that varies over the body."""
    gen = _gen(seed)
    parts = []
    for sc in scenes:
        for lo, side, n, mat, kind, v0, lattice in sc["bodies"]:
            lo_t = torch.tensor(lo, device="cuda", dtype=torch.float64)
            side_t = torch.tensor(side, device="cuda", dtype=torch.float64)
            x = _lattice(gen, lo_t, side_t, n) if lattice else lo_t + _rand(gen, n, 3) * side_t
            parts.append((x, lo_t + side_t / 2, side_t, n, mat, kind, v0, sc["mats"][mat].density))
    counts = torch.tensor([p[3] for p in parts], device="cuda")

    def per_particle(rows):
        return torch.repeat_interleave(rows, counts, 0)

    b = len(parts)
    pos = torch.cat([p[0] for p in parts])
    center, side = torch.stack([p[1] for p in parts]), torch.stack([p[2] for p in parts])
    base = torch.tensor([p[6] for p in parts], device="cuda", dtype=torch.float64)
    grad = (_rand(gen, b, 3, 3) - 0.5) * 12.0  # 1/s
    strain = torch.tensor([{"jelly": 0.006, "snow": 0.012, "water": 0.0}[p[5]] for p in parts], device="cuda",
                          dtype=torch.float64)
    phase = _rand(gen, b, 3, 3) * (2 * math.pi)
    r = pos - per_particle(center)
    k = 2 * math.pi / per_particle(side)
    wave = 0.3  # m/s
    g = per_particle(grad)
    nxt = [1, 2, 0]
    vel = per_particle(base) + _mv(g, r) + wave * torch.sin((k * r)[:, nxt])
    c = g.clone()
    for i, j in enumerate(nxt):
        c[:, i, j] += wave * k[:, j] * torch.cos(k[:, j] * r[:, j])
    f = per_particle(strain)[:, None, None] * torch.sin((k * r)[:, None, :] + per_particle(phase))
    f += torch.eye(3, device="cuda", dtype=torch.float64)
    fluid = per_particle(torch.tensor([p[5] == "water" for p in parts], device="cuda"))
    snow = per_particle(torch.tensor([p[5] == "snow" for p in parts], device="cuda"))
    s = 0.5 + 0.5 * torch.sin(k[:, 1] * r[:, 1])
    j = torch.where(fluid, 1.0 - 1e-3 * s, torch.where(snow, 1.0 - 0.01 * s, _det(f)))
    mass = torch.tensor([p[7] * float(p[2].prod()) / p[3] for p in parts], device="cuda", dtype=torch.float64)
    mat = torch.tensor([p[4] for p in parts], device="cuda", dtype=torch.int16)
    out = {"pos": pos, "vel": vel, "F": f.reshape(-1, 9), "J": j, "C": c.reshape(-1, 9), "mass": per_particle(mass)}
    out = {q: t.float().contiguous() for q, t in out.items()}
    out["mat"] = per_particle(mat).contiguous()
    return out


def _scene_objects(scenes):
    return [M.Scene(n=(s["grid"],) * 3, dx=1.0 / s["grid"], dt=s["dt"], materials=s["mats"], max_particles=_count(s))
            for s in scenes]


def _views(arrays, counts):
    """One library view per scene of arrays that hold the scenes one after another."""
    views, at = (M.ParticlesView * len(counts))(), 0
    for i, n in enumerate(counts):
        views[i] = M.ParticlesView(*(arrays[f].data_ptr() + at * WIDTH[f] * arrays[f].element_size() for f in FIELDS))
        at += n
    return views


def _numpy_particles(arrays, counts):
    """One M.Particles per scene over host arrays that hold the scenes one after another."""
    out, at = [], 0
    for n in counts:
        out.append(M.Particles(*((arrays[f][at:at + n].view(np.uint16) if f == "mat" else arrays[f][at:at + n])
                                 for f in FIELDS)))
        at += n
    return out


# ------------------------------------------------------------------------------------------------
# the engine's buffers
# ------------------------------------------------------------------------------------------------
NEAR = {"grid": 64, "dx": 1.6, "dt": 1.0 / 60.0}  # a window of 102.4 m, the player at its centre
MID = {"grid": 32, "dx": 12.5, "dt": 0.2}         # 400 m
TICK = {"near": 50.0, "mid": 200.0, "coarse_n": 16, "coarse_dx": 50.0, "dt": 1.0, "bounds": 750.0, "min_temp": 10.0,
        "max_temp": 8000.0}
GROUND = (("neo", 1e5, 0.3, 1000.0, 0.0, 0.0, 0.0), ("fluid", 5e4, 0.4, 1000.0, 0.0, 0.0, 0.0),
          ("sand", 2e5, 0.3, 1600.0, 0.0, 35.0, 100.0), ("clay", 2e5, 0.3, 2000.0, 2e3, 0.0, 0.0))
MODELS = [M.NEO_HOOKEAN, M.NEWTONIAN_FLUID, M.DRUCKER_PRAGER, M.VON_MISES]


def _engine_buffer(case, seed):
    """MpssBuffer arrays (device) and the ascending list of the selected particles: a ball or a shell
    around the player in shuffled buffer order, every material of the table among them."""
    gen = _gen(seed)
    near = case["kind"] == "near"
    n, cap = case["selected"], case["capacity"]
    half = (NEAR["grid"] * NEAR["dx"] if near else MID["grid"] * MID["dx"]) / 2
    r0, r1 = (0.0, 50.0) if near else (50.0, 200.0)
    chosen = torch.zeros(cap, dtype=torch.bool, device="cuda")
    chosen[torch.randperm(cap, generator=gen, device="cuda")[:n]] = True
    d = torch.randn(cap, 3, generator=gen, device="cuda", dtype=torch.float64)
    d /= d.norm(dim=1, keepdim=True)
    u = _rand(gen, cap)
    rad = torch.where(chosen, (r0 ** 3 + u * (r1 ** 3 - r0 ** 3)) ** (1 / 3), r1 + u * r1)
    f = torch.eye(3, device="cuda", dtype=torch.float64) + 0.004 * (_rand(gen, cap, 3, 3) - 0.5)
    a = {"pos": half + d * rad[:, None], "vel": 3.0 * torch.randn(cap, 3, generator=gen, device="cuda", dtype=torch.float64),
         "F": f.reshape(-1, 9), "J": _det(f), "C": _rand(gen, cap, 9) - 0.5, "mass": 0.5 + _rand(gen, cap)}
    a = {q: t.float() for q, t in a.items()}
    a["mat"] = torch.randint(0, 4, (cap,), generator=gen, device="cuda", dtype=torch.int16)
    return a, chosen.nonzero()[:, 0]


def _tick_arrays(case, seed):
    gen = _gen(seed)
    n = case["particles"]
    pos = _rand(gen, n, 3) * 1600 - 800
    close = torch.rand(n, generator=gen, device="cuda") < 0.03
    pos = torch.where(close[:, None], pos * 0.05, pos)
    return {"pos": pos.float(), "vel": 3.0 * torch.randn(n, 3, generator=gen, device="cuda"),
            "temp": (250 + 2250 * _rand(gen, n)).float(), "mass": (0.5 + 1.5 * _rand(gen, n)).float(),
            "active": (_rand(gen, n) > 0.05).to(torch.uint8),
            "phase": torch.zeros(n, dtype=torch.uint8, device="cuda"),
            "mat": torch.randint(0, 4, (n,), generator=gen, device="cuda", dtype=torch.int16),
            "coarse": (288.15 + 20 * _rand(gen, TICK["coarse_n"] ** 3)).float()}


def _ck_records(case, seed):
    """Records of an elastic block under load: a jittered lattice at 8 per cell, falling and shearing."""
    gen = _gen(seed)
    n, h = case["particles"], case["h"]
    m = int(math.ceil(n ** (1 / 3)))
    i = torch.arange(n, device="cuda")
    cell = torch.stack((i // (m * m), i // m % m, i % m), 1).double()
    spacing = 0.5 * h
    x = h * torch.tensor([32.0, 40.0, 32.0], device="cuda", dtype=torch.float64) + (cell + 0.25 + 0.5 * _rand(gen, n, 3)) * spacing
    v = 0.5 * torch.sin(x[:, [1, 2, 0]] * (2 * math.pi / (32 * h))) + 0.05 * torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)
    v[:, 1] -= 1.0
    f = torch.eye(3, device="cuda", dtype=torch.float64) + 0.02 * torch.sin(x[:, None, :] * (2 * math.pi / (32 * h)) + _rand(gen, 3, 3) * 6.28)
    b = 0.05 * (_rand(gen, n, 9) - 0.5)
    vol = torch.full((n, 1), spacing ** 3, device="cuda", dtype=torch.float64)
    return torch.cat((x, v, b, f.reshape(-1, 9), vol, 1000.0 * vol), 1).float().contiguous()


def _ck_config(case):
    return M.ck_config(dt=5e-3, grid_n=case["grid"], grid_h=case["h"], bounds_min=(0, 0, 0),
                       bounds_max=(case["grid"] * case["h"],) * 3)


def _split_records(r):
    return {"pos": r[:, 0:3], "vel": r[:, 3:6], "affine": r[:, 6:15], "deformation": r[:, 15:24], "constants": r[:, 24:26]}


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    ctx = M.Context(0)
    st = {"case": case, "ctx": ctx}
    if kind in ("world", "batched", "pipelined", "served"):
        scenes = _scenes(case)
        counts = [_count(s) for s in scenes]
        arrays = _particles(case, seed, scenes)
        objects = _scene_objects(scenes)
        st.update(scenes=scenes, counts=counts)
        if kind in ("world", "batched"):
            opts = M.exec_opts(sort_interval=case["sort_interval"], deterministic=int(case.get("deterministic", False)))
            out = {f: torch.zeros_like(t) for f, t in arrays.items()}
            st.update(world=M.World(ctx, objects, opts), arrays=arrays, out=out, vin=_views(arrays, counts),
                      vout=_views(out, counts), ids=np.arange(len(counts), dtype=np.uint32),
                      sizes=np.asarray(counts, np.uint64))
        else:
            # the pipelined call wants page-locked arrays, the server copies at submit
            host = {f: t.cpu() for f, t in arrays.items()}
            if kind == "pipelined":
                host = {f: t.pin_memory() for f, t in host.items()}
            res = {f: torch.zeros(t.shape, dtype=t.dtype, pin_memory=kind == "pipelined") for f, t in host.items()}
            st.update(host=host, out=res)
            parts = _numpy_particles({f: t.numpy() for f, t in host.items()}, counts)
            outs = _numpy_particles({f: t.numpy() for f, t in res.items()}, counts)
            if kind == "pipelined":
                st.update(batch=M.Batch(ctx, objects, M.exec_opts(sort_interval=16), groups=case["groups"]),
                          parts=M.ViewArray(parts), outs=M.ViewArray(outs))
            else:
                st.update(server=M.Server(ctx, hbm_budget_bytes=16 << 30, substeps_per_tick=20,
                                          exec_options=M.exec_opts(sort_interval=16)),
                          parts=parts, outs=outs, objects=objects)
    elif kind in ("near", "mid"):
        arrays, idx = _engine_buffer(case, seed)
        host = {f: t.cpu().numpy() for f, t in arrays.items()}
        host["mat"] = host["mat"].view(np.uint16)
        win = NEAR if kind == "near" else MID
        n = win["grid"]
        st.update(parts=M.Particles(*(host[f] for f in FIELDS)), idx=idx.cpu().numpy().astype(np.uint64),
                  grid=M.Grid(n, n, n, win["dx"], (0.0, 0.0, 0.0)), dt=win["dt"],
                  config=M.Config(grid_dx=win["dx"], grid_size=(n, n, n), substeps=1, gravity=(0, -9.81, 0), damping=0.995),
                  mats=[M.material(young_modulus=e, poisson_ratio=nu, density=rho, yield_stress=y, friction_angle=phi,
                                   cohesion=coh, hardening=0.0) for _, e, nu, rho, y, phi, coh in GROUND])
    elif kind == "ck":
        init = _ck_records(case, seed)
        st.update(init=init, records=torch.empty_like(init), config=_ck_config(case))
    else:
        init = _tick_arrays(case, seed)
        n = case["particles"]
        origin = np.full(3, -TICK["coarse_n"] * TICK["coarse_dx"] / 2, np.float32)
        st.update(init=init, work={q: t.clone() for q, t in init.items()},
                  lists=[torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(3)],
                  player=np.zeros(3, np.float32), origin=origin, lo=np.full(3, -TICK["bounds"], np.float32),
                  hi=np.full(3, TICK["bounds"], np.float32))
    torch.cuda.synchronize()
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind, lib = case["kind"], ctx.lib
    if kind == "world":
        w = st["world"]
        ctx.check(lib.ae_mpm_world_upload(w.h, 0, st["vin"], st["counts"][0]))
        w.step(case["substeps"])
        ctx.check(lib.ae_mpm_world_download(w.h, 0, st["vout"]))
        return st["out"]
    if kind == "batched":
        w, k = st["world"], len(st["counts"])
        ctx.check(lib.ae_mpm_world_upload_many(w.h, k, st["ids"].ctypes.data, ctypes.addressof(st["vin"]),
                                               st["sizes"].ctypes.data))
        w.step(case["substeps"])
        ctx.check(lib.ae_mpm_world_download_many(w.h, k, st["ids"].ctypes.data, ctypes.addressof(st["vout"])))
        return st["out"]
    if kind == "pipelined":
        st["batch"].run(st["parts"], case["substeps"], out=st["outs"])
        return st["out"]
    if kind == "served":
        srv = st["server"]
        for scene, p, o, s in zip(st["objects"], st["parts"], st["outs"], st["scenes"]):
            srv.submit(scene, p, s["substeps"], o)
        if srv.drain(60.0) != M.OK:
            raise RuntimeError("the server did not drain")
        srv.poll(4 * len(st["parts"]))
        return st["out"]
    if kind == "near":
        p = st["parts"]
        ctx.step_parallel_with_grid(p, st["grid"], st["config"], st["mats"], MODELS, st["dt"], st["idx"])
        return {"pos": p.pos, "vel": p.vel, "F": p.F, "J": p.J, "C": p.C}
    if kind == "mid":
        p = st["parts"]
        ctx.step_velocity_only_parallel(p, st["grid"], st["config"], st["dt"], st["idx"])
        return {"pos": p.pos, "vel": p.vel}
    if kind == "ck":
        st["records"].copy_(st["init"])
        ctx.check(lib.ae_mpm_ck_step(ctx.h, st["records"].data_ptr(), case["particles"], ctypes.byref(st["config"]),
                                     case["steps"]))
        return _split_records(st["records"])
    return _run_tick(st)


def _run_tick(st):
    """One tick: the engine has just written this frame's positions and velocities."""
    case, ctx, d = st["case"], st["ctx"], st["work"]
    lib, h, n = ctx.lib, ctx.h, case["particles"]
    for q in ("pos", "vel", "temp", "phase", "coarse"):
        d[q].copy_(st["init"][q])
    p = {q: t.data_ptr() for q, t in d.items()}
    near, mid, far = (t.data_ptr() for t in st["lists"])
    c = [ctypes.c_uint64(0) for _ in range(3)]
    ctx.check(lib.ae_mpm_lod_classify(h, p["pos"], p["active"], n, st["player"].ctypes.data, TICK["near"], TICK["mid"],
                                      case["max_near"], near, ctypes.byref(c[0]), mid, ctypes.byref(c[1]), far,
                                      ctypes.byref(c[2])))
    ctx.check(lib.ae_mpm_far_field_update(h, p["pos"], p["vel"], p["temp"], n, far, c[2].value, p["coarse"],
                                          TICK["coarse_n"], TICK["coarse_dx"], st["origin"].ctypes.data, TICK["dt"]))
    ctx.check(lib.ae_mpm_coarse_field_update(h, p["pos"], p["mass"], p["temp"], p["active"], n, near, c[0].value,
                                             p["coarse"], TICK["coarse_n"], TICK["coarse_dx"],
                                             st["origin"].ctypes.data, TICK["dt"]))
    changes = ctypes.c_uint32(0)
    ctx.check(lib.ae_mpm_mpss_housekeeping(h, p["pos"], p["vel"], p["temp"], p["phase"], p["mat"], p["active"], n,
                                           st["lo"].ctypes.data, st["hi"].ctypes.data, TICK["min_temp"],
                                           TICK["max_temp"], 7, ctypes.byref(changes)))
    return {"near": st["lists"][0], "mid": st["lists"][1], "far": st["lists"][2], "counts": [x.value for x in c],
            "pos": d["pos"], "vel": d["vel"], "temp": d["temp"], "phase": d["phase"], "coarse": d["coarse"],
            "changes": changes.value}


def work(case):
    """Per particle and substep a pass reads the state (104 B) and writes what changes (100 B); in and
    out once each (106 B).  A quadratic stencil costs about 27 x (7 + 13) fused operations and the
    material update about 200; the host cases count the bytes that cross to the device and back."""
    kind = case["kind"]
    if kind in ("world", "batched", "pipelined", "served"):
        scenes = _scenes(case)
        steps = sum(_count(s) * s["substeps"] for s in scenes)
        return {"bytes": 204.0 * steps + 212.0 * sum(_count(s) for s in scenes), "flops": 1500.0 * steps}
    if kind == "near":
        return {"bytes": (104 + 100 + 8) * case["selected"], "flops": 2500 * case["selected"]}
    if kind == "mid":
        return {"bytes": (28 + 24 + 8) * case["selected"], "flops": 600 * case["selected"]}
    if kind == "ck":
        return {"bytes": 200.0 * case["particles"] * case["steps"], "flops": 700.0 * case["particles"] * case["steps"]}
    n = case["particles"]
    return {"bytes": (13 + 8 + 32 + 61) * n, "flops": 60.0 * n}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("world", "batched", "pipelined", "served"):
        if case.get("scenes", 0) > 600 or case.get("particles", 0) > 9e6:
            return None
        scenes = _scenes(case)
        return _exact_physics(scenes, _particles(case, seed, scenes))
    if kind in ("near", "mid"):
        return _exact_engine(case, seed)
    if kind == "ck":
        return _exact_ck(case, seed)
    return _exact_tick(case, seed)


def _stretch(f):
    """Singular values and right vectors of F by cyclic Jacobi on F^T F (well-conditioned F)."""
    a = _mm(f.transpose(1, 2), f)
    v = torch.eye(3, dtype=f.dtype, device=f.device).expand_as(f).clone()
    for _ in range(6):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = a[:, p, q]
            tau = (a[:, q, q] - a[:, p, p]) / torch.where(apq == 0, torch.ones_like(apq), 2 * apq)
            t = torch.where(tau >= 0, 1.0, -1.0) / (tau.abs() + torch.sqrt(1 + tau * tau))
            t = torch.where(apq == 0, torch.zeros_like(t), t)
            c = (1 / torch.sqrt(1 + t * t))[:, None]
            s = t[:, None] * c
            ap, aq = a[:, :, p].clone(), a[:, :, q].clone()
            a[:, :, p], a[:, :, q] = c * ap - s * aq, s * ap + c * aq
            ap, aq = a[:, p, :].clone(), a[:, q, :].clone()
            a[:, p, :], a[:, q, :] = c * ap - s * aq, s * ap + c * aq
            vp, vq = v[:, :, p].clone(), v[:, :, q].clone()
            v[:, :, p], v[:, :, q] = c * vp - s * vq, s * vp + c * vq
    return torch.sqrt(torch.diagonal(a, dim1=1, dim2=2)), v


def _exact_physics(scenes, arrays):
    """MLS-MPM with sticky walls; scenes side by side in one node array."""
    dev = "cuda"
    counts = torch.tensor([_count(s) for s in scenes], device=dev)
    f32 = np.float32
    nodes = torch.tensor([s["grid"] for s in scenes], device=dev)
    first = torch.cumsum(nodes ** 3, 0) - nodes ** 3
    total = int((nodes ** 3).sum())

    def each(values):
        return torch.repeat_interleave(torch.tensor([float(v) for v in values], device=dev, dtype=torch.float64), counts)

    dx, inv = each(f32(1.0 / s["grid"]) for s in scenes), each(f32(1) / f32(1.0 / s["grid"]) for s in scenes)
    dt = each(f32(s["dt"]) for s in scenes)
    steps = torch.repeat_interleave(torch.tensor([s["substeps"] for s in scenes], device=dev), counts)
    n = torch.repeat_interleave(nodes, counts)
    off = torch.repeat_interleave(first, counts)
    node_dt = torch.repeat_interleave(torch.tensor([float(f32(s["dt"])) for s in scenes], device=dev, dtype=torch.float64), nodes ** 3)
    local = torch.arange(total, device=dev) - torch.repeat_interleave(first, nodes ** 3)
    gn = torch.repeat_interleave(nodes, nodes ** 3)
    wall = torch.zeros(total, dtype=torch.bool, device=dev)
    for c in (local % gn, local // gn % gn, local // (gn * gn)):
        wall |= (c < 3) | (c >= gn - 3)
    del local, gn
    # the materials' derived constants are single precision in the interface's semantics
    table = []
    for s in scenes:
        for m in s["mats"]:
            e, nu = f32(m.young_modulus), f32(m.poisson_ratio)
            table.append((m.model, m.density, e / (f32(2) * (f32(1) + nu)),
                          e * nu / ((f32(1) + nu) * (f32(1) - f32(2) * nu)), m.bulk_modulus, f32(1) - f32(m.theta_c),
                          f32(1) + f32(m.theta_s), m.hardening_xi))
    start = np.cumsum([0] + [len(s["mats"]) for s in scenes])[:-1]
    mat = arrays["mat"].long() + torch.repeat_interleave(torch.tensor(start, device=dev), counts)
    table = torch.tensor([[float(v) for v in row] for row in table], device=dev, dtype=torch.float64)[mat]
    model, rho, mu, la, bulk, lo, hi, xi = (table[:, i].contiguous() for i in range(8))
    lo, hi = lo.float().double(), hi.float().double()
    fluid, snow = model == M.PHYS_FLUID, model == M.PHYS_SNOW
    del table
    x, v = arrays["pos"].double(), arrays["vel"].double()
    f, c = arrays["F"].double().reshape(-1, 3, 3), arrays["C"].double().reshape(-1, 3, 3)
    j, m = arrays["J"].double(), arrays["mass"].double()
    eye = torch.eye(3, device=dev, dtype=torch.float64)
    grav = torch.tensor([0.0, float(f32(-9.8)), 0.0], device=dev, dtype=torch.float64)
    same = int(steps.min()) == int(steps.max())
    for step in range(int(steps.max())):
        on = slice(None) if same else (steps > step).nonzero()[:, 0]
        xo, vo, fo, co, jo, mo = x[on], v[on], f[on], c[on], j[on], m[on]
        dxo, dto, no, offo, invo = dx[on], dt[on], n[on], off[on], inv[on]
        fl, sn = fluid[on], snow[on]
        hard = torch.where(sn, torch.exp(xi[on] * (1 - jo)).clamp(0.1, 5), torch.ones_like(jo))
        tau = (mu[on] * hard)[:, None, None] * (_mm(fo, fo.transpose(1, 2)) - eye)
        tau += (la[on] * hard * torch.log(_det(fo).clamp(0.01, 100)))[:, None, None] * eye
        tau = torch.where(fl[:, None, None], (bulk[on] * (jo - 1))[:, None, None] * eye, tau)
        a = mo[:, None, None] * co - (4 * dto * (mo / rho[on]) * invo * invo)[:, None, None] * tau
        del tau
        xg = xo * invo[:, None]
        base = torch.floor(xg - 0.5)
        fx = xg - base
        base = base.long()
        w = torch.stack((0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2), 2)
        acc = torch.zeros(total, 4, device=dev, dtype=torch.float64)

        def stencil():
            for o in range(27):
                oi, oj, ok = o % 3, o // 3 % 3, o // 9
                idx = offo + ((base[:, 2] + ok) * no + base[:, 1] + oj) * no + base[:, 0] + oi
                d = (torch.tensor([oi, oj, ok], device=dev, dtype=torch.float64) - fx) * dxo[:, None]
                yield idx, w[:, 0, oi] * w[:, 1, oj] * w[:, 2, ok], d

        for idx, ww, d in stencil():
            mom = mo[:, None] * vo + _mv(a, d)
            acc.index_add_(0, idx, ww[:, None] * torch.cat((mo[:, None], mom), 1))
        del a
        mass = acc[:, 0]
        gv = torch.where((mass > 0)[:, None], acc[:, 1:] / mass.clamp_min(1e-300)[:, None] + node_dt[:, None] * grav, 0.0)
        gv[wall] = 0.0
        vn, b = torch.zeros_like(vo), torch.zeros_like(fo)
        for idx, ww, d in stencil():
            g = ww[:, None] * gv[idx]
            vn += g
            b += g[:, :, None] * d[:, None, :]
        cn = (4 * invo * invo)[:, None, None] * b
        del b, acc, gv
        xn = xo + dto[:, None] * vn
        xn = torch.minimum(torch.maximum(xn, dxo[:, None]), ((no - 2) * dxo)[:, None])
        trace = cn[:, 0, 0] + cn[:, 1, 1] + cn[:, 2, 2]
        fn = _mm(eye + dto[:, None, None] * cn, fo)
        fn = torch.where(fl[:, None, None], fo, fn)
        jn = torch.where(fl, (jo * (1 + dto * trace)).clamp_min(0.01), torch.where(sn, jo, _det(fn)))
        at = sn.nonzero()[:, 0]
        if at.numel():
            s, vr = _stretch(fn[at])
            cl = torch.minimum(torch.maximum(s, lo[on][at][:, None]), hi[on][at][:, None])
            fn[at] = _mm(_mm(fn[at], vr * (cl / s)[:, None, :]), vr.transpose(1, 2))
            jn[at] = jn[at] * s.prod(1) / cl.prod(1)
        if same:
            x, v, f, c, j = xn, vn, fn, cn, jn
        else:
            x[on], v[on], f[on], c[on], j[on] = xn, vn, fn, cn, jn
    return {"pos": x, "vel": v, "F": f.reshape(-1, 9), "J": j, "C": c.reshape(-1, 9), "mass": m, "mat": None}


def _spline(x):
    ax = x.abs()
    return torch.where(ax < 0.5, 0.75 - ax * ax, torch.where(ax < 1.5, 0.5 * (1.5 - ax) ** 2, 0.0))


def _spline_slope(x):
    ax = x.abs()
    return torch.where(ax < 0.5, -2 * x, torch.where(ax < 1.5, -(1.5 - ax) * torch.sign(x), 0.0))


def _ground_stress(mat, f, j):
    """Cauchy stress of the table's four models; for F near the identity the reference's polar
    iteration returns R = I, so S = F."""
    out = torch.zeros_like(f)
    eye = torch.eye(3, device=f.device, dtype=f.dtype)
    for k, (name, e, nu, _, y, phi, coh) in enumerate(GROUND):
        at = (mat == k).nonzero()[:, 0]
        fk, jk = f[at], j[at]
        e, nu = np.float32(e), np.float32(nu)
        mu = float(e / (np.float32(2) * (np.float32(1) + nu)))
        la = float(e * nu / ((np.float32(1) + nu) * (np.float32(1) - np.float32(2) * nu)))
        if name == "fluid":
            s = (float(e / (np.float32(3) * (np.float32(1) - np.float32(2) * nu))) * (jk - 1))[:, None, None] * eye
        elif name == "neo":
            s = (mu / jk)[:, None, None] * (_mm(fk, fk.transpose(1, 2)) - eye) + (la * torch.log(jk) / jk)[:, None, None] * eye
        else:
            eps = fk - eye
            tr = torch.diagonal(eps, dim1=1, dim2=2).sum(1)
            dev = 2 * mu * (eps - (tr / 3)[:, None, None] * eye)
            norm = torch.sqrt(0.5 * (dev * dev).sum((1, 2)))
            p = -la * tr
            if name == "sand":
                sp, cp = math.sin(math.radians(phi)), math.cos(math.radians(phi))
                al, kk = 2 * sp / (math.sqrt(3) * (3 - sp)), 6 * coh * cp / (math.sqrt(3) * (3 - sp))
                sc = torch.where(norm + al * p - kk > 0, (kk - al * p).clamp_min(0) / norm.clamp_min(1e-10), 1.0)
            else:
                thr = y / math.sqrt(3)
                sc = torch.where(norm > thr, thr / norm.clamp_min(1e-300), 1.0)
            s = dev * sc[:, None, None] - p[:, None, None] * eye
        out[at] = s
    return out


def _exact_engine(case, seed):
    """One substep of the engine's reference-mode or velocity-only solver over the selected particles."""
    arrays, sel = _engine_buffer(case, seed)
    near = case["kind"] == "near"
    win = NEAR if near else MID
    g, dx = win["grid"], float(np.float32(win["dx"]))
    inv, dt = float(np.float32(1) / np.float32(win["dx"])), float(np.float32(win["dt"]))
    x, v, m = arrays["pos"][sel].double(), arrays["vel"][sel].double(), arrays["mass"][sel].double()
    f, c = arrays["F"][sel].double().reshape(-1, 3, 3), arrays["C"][sel].double().reshape(-1, 3, 3)
    q = x * inv - 0.5
    fl = torch.floor(q)
    fx = q - fl
    base = fl.long().clamp_min(0)
    w = torch.stack([_spline(k - fx) for k in range(3)], 2)
    dw = torch.stack([_spline_slope(k - fx) for k in range(3)], 2) * inv
    if near:
        rho = torch.tensor([row[3] for row in GROUND], device="cuda", dtype=torch.float64)[arrays["mat"][sel].long()]
        sv = dt * (m / rho)[:, None, None] * _ground_stress(arrays["mat"][sel], f, arrays["J"][sel].double())
    grid = torch.zeros(g ** 3, 4, device="cuda", dtype=torch.float64)

    def stencil():
        for o in range(27):
            i, jj, k = o % 3, o // 3 % 3, o // 9
            node = base + torch.tensor([i, jj, k], device="cuda")
            ww = w[:, 0, i] * w[:, 1, jj] * w[:, 2, k]
            ok = (ww >= 1e-10) & (node < g).all(1)
            idx = torch.where(ok, (node[:, 2] * g + node[:, 1]) * g + node[:, 0], 0)
            yield idx, torch.where(ok, ww, 0.0), ok, (node.double() + 0.5) * dx - x, torch.stack((dw[:, 0, i], dw[:, 1, jj], dw[:, 2, k]), 1)

    for idx, ww, ok, d, e in stencil():
        wm = ww * m
        mom = wm[:, None] * (v + _mv(c, d)) if near else wm[:, None] * v
        if near:
            mom = mom + torch.where(ok[:, None], _mv(sv, e), 0.0)
        grid.index_add_(0, idx, torch.cat((wm[:, None], mom), 1))
    mass = grid[:, 0]
    gv = torch.where((mass > 1e-12)[:, None], grid[:, 1:] / mass.clamp_min(1e-300)[:, None], 0.0)
    gv[:, 1] += torch.where(mass > 1e-12, dt * float(np.float32(-9.81)), 0.0)
    floor = torch.arange(g ** 3, device="cuda") // g % g == 0
    gv[floor] = torch.stack((gv[floor, 0] * float(np.float32(0.9)), gv[floor, 1].clamp_min(0), gv[floor, 2] * float(np.float32(0.9))), 1)
    nv, nc, grad = torch.zeros_like(v), torch.zeros_like(f), torch.zeros_like(f)
    for idx, ww, ok, d, e in stencil():
        ww = torch.where(mass[idx] >= 1e-12, ww, 0.0)
        u = ww[:, None] * gv[idx]
        nv += u
        nc += (4 * inv * inv) * u[:, :, None] * d[:, None, :]
        grad -= u[:, :, None] * e[:, None, :]
    nv = nv.clamp(-50, 50)
    nx = x + dt * nv
    hit = nx[:, 1] < 0
    nx[:, 1] = nx[:, 1].clamp_min(0)
    nv[:, 1] = torch.where(hit, nv[:, 1].clamp_min(0) * 0.5, nv[:, 1])
    top = (g - 1) * dx
    for a in (0, 2):
        low, high = nx[:, a] < 0, nx[:, a] > top
        nv[:, a] = torch.where(low, nv[:, a].clamp_min(0) * 0.5, torch.where(high, nv[:, a].clamp_max(0) * 0.5, nv[:, a]))
        nx[:, a] = nx[:, a].clamp(0, top)
    out = {q: arrays[q].double() for q in ("pos", "vel", "F", "J", "C")}
    out["pos"][sel] = nx
    out["vel"][sel] = nv * float(np.float32(0.995))
    if not near:
        return {"pos": out["pos"], "vel": out["vel"]}
    eye = torch.eye(3, device="cuda", dtype=torch.float64)
    nf = _mm(eye + dt * grad, f)
    good = (nf.abs() <= 1e3).all(2).all(1)
    nf = torch.where(good[:, None, None], nf, eye)
    out["F"][sel] = nf.reshape(-1, 9)
    out["J"][sel] = torch.where(good, _det(nf).clamp(0.1, 10), 1.0)
    out["C"][sel] = nc.reshape(-1, 9)
    return out


def _exact_ck(case, seed):
    """CkMpmSolver steps: matrices are stored by columns."""
    r = _ck_records(case, seed).double()
    cfg = _ck_config(case)
    g, h, dt = case["grid"], float(np.float32(case["h"])), float(np.float32(cfg.dt))
    e, nu = float(cfg.youngs_modulus), float(np.float32(cfg.poissons_ratio))
    mu, la = e / (2 * (1 + nu)), e * nu / ((1 + nu) * (1 - 2 * nu))
    x, v = r[:, 0:3].clone(), r[:, 3:6].clone()
    b, f = (r[:, s].reshape(-1, 3, 3).transpose(1, 2).clone() for s in (slice(6, 15), slice(15, 24)))
    vol, m = r[:, 24], r[:, 25]
    rest = float(np.float32(cfg.restitution))
    bounds = [(float(cfg.bounds_min[a]), float(cfg.bounds_max[a])) for a in range(3)]
    eye = torch.eye(3, device="cuda", dtype=torch.float64)
    grav = torch.tensor([float(q) for q in cfg.gravity], device="cuda", dtype=torch.float64)

    def kernel(d):
        rr = d.abs() / h
        a = 1 - rr * rr
        return torch.where(rr < 1, a ** 3 / h, 0.0), torch.where(rr < 1, -6 * d * a * a / h ** 3, 0.0)

    def capped(u, cap):
        ln = u.norm(dim=1, keepdim=True)
        return torch.where(ln > cap, u * (cap / ln.clamp_min(1e-300)), u)

    def stencil():
        base = torch.floor(x / h).long()
        axes = [[kernel((base[:, a].double() + d + 0.5) * h - x[:, a]) for d in range(2)] for a in range(3)]
        for o in range(8):
            di = (o & 1, o >> 1 & 1, o >> 2)
            node = base + torch.tensor(di, device="cuda")
            ok = ((node >= 0) & (node < g)).all(1)
            (wx, gx), (wy, gy), (wz, gz) = (axes[a][di[a]] for a in range(3))
            idx = torch.where(ok, (node[:, 2] * g + node[:, 1]) * g + node[:, 0], 0)
            grad = torch.stack((gx * wy * wz, wx * gy * wz, wx * wy * gz), 1)
            yield idx, torch.where(ok, wx * wy * wz, 0.0), torch.where(ok[:, None], grad, 0.0), (node.double() + 0.5) * h - x

    at = torch.arange(g ** 3, device="cuda")
    place = [(c.double() + 0.5) * h for c in (at % g, at // g % g, at // (g * g))]
    for _ in range(case["steps"]):
        det = _det(f)
        fit = _cofactor(f) / det[:, None, None]
        p = mu * (f - fit) + (la * torch.log(det.clamp_min(1e-10)))[:, None, None] * fit
        grid = torch.zeros(g ** 3, 7, device="cuda", dtype=torch.float64)
        for idx, w, grad, d in stencil():
            wm = (w * m)[:, None]
            force = capped(-vol[:, None] * _mv(p, grad), 1e4)
            grid.index_add_(0, idx, torch.cat((wm, wm * (v + _mv(b, d)), force), 1))
        mass = grid[:, :1]
        ms = mass.clamp_min(1e-300)
        gv = torch.where(mass > 1e-10, capped(grid[:, 1:4] / ms + dt * (grid[:, 4:7] / ms + grav), 50.0), 0.0)
        for a, (lo, hi) in enumerate(bounds):
            back = ((place[a] < lo) & (gv[:, a] < 0)) | ((place[a] > hi) & (gv[:, a] > 0))
            gv[:, a] = torch.where(back, -rest * gv[:, a], gv[:, a])
        v, b = torch.zeros_like(v), torch.zeros_like(b)
        for idx, w, _, d in stencil():
            u = w[:, None] * gv[idx]
            v = v + u
            b = b + (4 / (h * h)) * u[:, :, None] * d[:, None, :]
        v = capped(v, 50.0)
        grad_v = (4 / (h * h)) * b
        norm = grad_v.norm(dim=1).amax(1)
        fn = _mm(eye + dt * grad_v * torch.where(norm > 100, 100 / norm, 1.0)[:, None, None], f)
        fd = _det(fn).abs()
        f = torch.where(((fd > 1e-10) & (fd < 100))[:, None, None], fn, f)
        x = x + dt * v
        for a, (lo, hi) in enumerate(bounds):
            low, high = x[:, a] < lo, x[:, a] > hi
            v[:, a] = torch.where((low & (v[:, a] < 0)) | (high & (v[:, a] > 0)), -rest * v[:, a], v[:, a])
            x[:, a] = x[:, a].clamp(lo, hi)
    cols = [t.transpose(1, 2).reshape(-1, 9) for t in (b, f)]
    return _split_records(torch.cat((x, v, cols[0], cols[1], r[:, 24:26]), 1))


def _exact_tick(case, seed):
    """The tick's floating outputs; the index lists and phases are whole numbers."""
    d = _tick_arrays(case, seed)
    f32 = torch.float32
    # the distances decide in single precision
    sq = d["pos"] * d["pos"]
    d2 = (sq[:, 0] + sq[:, 1]) + sq[:, 2]
    on = d["active"] != 0
    near = (on & (d2 < torch.tensor(TICK["near"] ** 2, dtype=f32))).nonzero()[:, 0]
    far = (on & ~(d2 < torch.tensor(TICK["mid"] ** 2, dtype=f32))).nonzero()[:, 0]
    if near.numel() > case["max_near"]:
        order = torch.argsort(d2[near], stable=True)[:case["max_near"]]
        near = near[torch.sort(order).values]
    n, cdx, dt = TICK["coarse_n"], TICK["coarse_dx"], TICK["dt"]
    origin = -n * cdx / 2
    pos, vel, temp, field = d["pos"].double(), d["vel"].double(), d["temp"].double(), d["coarse"].double()
    vel[far, 1] -= float(np.float32(9.81)) * dt
    pos[far, 1] += vel[far, 1] * dt
    cell = ((pos[far] - origin) / cdx).trunc().long()
    ok = ((cell >= 0) & (cell < n)).all(1)
    at, cell = far[ok], cell[ok]
    temp[at] += (field[cell[:, 0] + n * (cell[:, 1] + n * cell[:, 2])] - temp[at]) * float(np.float32(0.02)) * dt
    cell = ((pos[near] - origin) / cdx).trunc().long()
    idx = cell[:, 0] + n * (cell[:, 1] + n * cell[:, 2])
    m = d["mass"].double()[near]
    tm = torch.zeros_like(field).index_add_(0, idx, temp[near] * m)
    ms = torch.zeros_like(field).index_add_(0, idx, m)
    field = torch.where(ms > 1e-6, field + (tm / ms.clamp_min(1e-300) - field) * min(float(np.float32(0.1)) * dt, 1.0), field)
    cube = field.reshape(n, n, n)
    lap, count = torch.zeros_like(cube), torch.zeros_like(cube)
    for a in range(3):
        for s in (1, -1):
            src, dst = [slice(None)] * 3, [slice(None)] * 3
            src[a], dst[a] = (slice(0, -1), slice(1, None)) if s == 1 else (slice(1, None), slice(0, -1))
            lap[tuple(dst)] += cube[tuple(src)]
            count[tuple(dst)] += 1
    cube = cube + min(10.0 * dt / (cdx * cdx), float(np.float32(0.16))) * (lap / count - cube) * count
    on = on[:, None]
    for side, sign in ((-TICK["bounds"], 1.0), (TICK["bounds"], -1.0)):
        out = on & (sign * (pos - side) < 0)
        vel = torch.where(out & (sign * vel < 0), -0.5 * vel, vel)
        pos = torch.where(out, side, pos)
    temp = torch.where(on[:, 0], temp.clamp(TICK["min_temp"], TICK["max_temp"]), temp)
    return {"near": None, "mid": None, "far": None, "counts": None, "pos": pos, "vel": vel, "temp": temp, "phase": None,
            "coarse": cube.reshape(-1), "changes": None}
