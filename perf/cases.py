"""The calls whose time counts, and the inputs they are timed on.

Every case goes through the C ABI as :mod:`nbody_gb300.native` binds it, as a program that
uses the library calls it: accelerations over the caller's device buffers, a frame of a
simulation (upload, steps, download), one accelerate and its readback, the energy
diagnostics, and picking in the tree. Inputs are seeded draws of the scenes that
``nbody_gb300/scenes.py`` describes, made on the GPU.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nbody_gb300 import native

G = 1.0


def listed():
    return [
        # the smallest call: one accelerate of a scene of a thousand bodies in the reference's
        # interleaved layout under its own cutoff law, from an engine's device buffer; latency
        {"name": "accel_aos_1000", "kind": "accel", "n": 1000, "layout": "aos", "law": "cutoff", "scene": "disk"},
        # an ordinary direct sum over split device buffers, at no round size
        {"name": "accel_soa_20011", "kind": "accel", "n": 20011, "layout": "soa", "law": "softened", "scene": "plummer"},
        # the largest direct sum: 2^20 bodies uniform in a cube
        {"name": "accel_soa_1m", "kind": "accel", "n": 1 << 20, "layout": "soa", "law": "softened", "scene": "cube"},
        # a small system advanced many steps between readbacks: 4096 bodies, 100 steps
        {"name": "steps_4096", "kind": "steps", "n": 4096, "steps": 100, "layout": "soa", "law": "softened",
         "precision": "fp32", "scene": "plummer"},
        # compensated positions and velocities, a few steps of a frame
        {"name": "steps_comp_50021", "kind": "steps", "n": 50021, "steps": 4, "layout": "soa", "law": "softened",
         "precision": "comp", "scene": "plummer"},
        # the FP64 form, which references and error measurements run on
        {"name": "fp64_12289", "kind": "fp64", "n": 12289, "law": "softened", "scene": "plummer"},
        # 512 independent systems of 64 to 8192 bodies, advanced together
        {"name": "batch_512", "kind": "batch", "systems": 512, "lo": 64, "hi": 8192, "steps": 10},
        # Barnes-Hut, two Plummer spheres of 131072 bodies, the reference's walk, opening
        # parameter and fixed box; 20 steps between readbacks
        {"name": "bh_steps_262144", "kind": "bh", "n": 262144, "steps": 20, "layout": "soa", "law": "softened",
         "scene": "pair", "theta": 0.5, "walk": "target", "box": "fixed"},
        # the reference's own Barnes-Hut setting at a million bodies: interleaved bodies, cutoff
        # law, theta 0.5, fixed box, a disk; a frame's accelerations
        {"name": "bh_aos_1000003", "kind": "bh", "n": 1000003, "steps": 0, "layout": "aos", "law": "cutoff",
         "scene": "disk", "theta": 0.5, "walk": "target", "box": "fixed"},
        # the largest tree: disk and halo of 16.8M bodies at the conventional theta 0.5 (2 in the
        # reference's convention), walked by groups
        {"name": "bh_group_16m", "kind": "bh", "n": 1 << 24, "steps": 0, "layout": "soa", "law": "softened",
         "scene": "halo", "theta": 2.0, "walk": "group", "box": "fitted"},
        # energy and momentum of a system, as a run's drift is followed
        {"name": "energy_200003", "kind": "energy", "n": 200003, "scene": "plummer"},
        # a renderer's frame: a tree over the current bodies, and the bodies under many rays
        {"name": "pick_250007", "kind": "pick", "n": 250007, "rays": 20011, "scene": "plummer"},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n))


def draw(rng):
    kind = rng.choice(["accel", "accel", "steps", "fp64", "batch", "bh", "bh", "bh", "energy", "pick"])
    law = rng.choice(["softened", "cutoff"])
    layout = rng.choice(["soa", "aos"])
    if kind == "accel":
        return {"kind": kind, "n": _log_int(rng, 500, 1 << 20), "layout": layout, "law": law,
                "scene": rng.choice(["plummer", "cube", "disk"])}
    if kind == "steps":
        return {"kind": kind, "n": _log_int(rng, 500, 60000), "steps": rng.randint(2, 30), "layout": layout,
                "law": "softened", "precision": rng.choice(["fp32", "comp"]), "scene": rng.choice(["plummer", "cube"])}
    if kind == "fp64":
        return {"kind": kind, "n": _log_int(rng, 2000, 40000), "law": law, "scene": rng.choice(["plummer", "cube"])}
    if kind == "batch":
        lo = rng.choice([16, 64, 256])
        return {"kind": kind, "systems": _log_int(rng, 32, 600), "lo": lo, "hi": rng.choice([1024, 4096, 8192]),
                "steps": rng.randint(2, 20)}
    if kind == "energy":
        return {"kind": kind, "n": _log_int(rng, 5000, 400000), "scene": rng.choice(["plummer", "cube"])}
    if kind == "pick":
        return {"kind": kind, "n": _log_int(rng, 20000, 400000), "rays": _log_int(rng, 500, 100000), "scene": "plummer"}
    n = _log_int(rng, 20000, 1 << 24)
    return {"kind": "bh", "n": n, "steps": rng.choice([0, 0, rng.randint(2, 6)]), "layout": layout, "law": law,
            "scene": rng.choice(["pair", "halo", "disk"]), "theta": rng.choice([0.5, 0.75, 1.33, 2.0]),
            "walk": rng.choice(["target", "group"]), "box": rng.choice(["fixed", "fitted"])}


# --- scenes -----------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _directions(g, n):
    z = 2 * _uniform(g, n) - 1
    phi = 2 * math.pi * _uniform(g, n)
    s = torch.sqrt(torch.clamp(1 - z * z, min=0))
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _plummer(g, n, rmax=10.0):
    """Positions and isotropic velocities of a Plummer sphere of unit mass and radius."""
    top = rmax ** 3 / (1 + rmax * rmax) ** 1.5
    x = _uniform(g, n).clamp(min=1e-6) * top
    r = 1 / torch.sqrt(x ** (-2.0 / 3.0) - 1)
    sigma = torch.sqrt(1 / (6 * torch.sqrt(1 + r * r)))
    vel = torch.randn(n, 3, generator=g, device="cuda") * sigma[:, None]
    return _directions(g, n) * r[:, None], vel


def _scene(scene, n, seed):
    """(n, 12) bodies on the GPU: pos, radius, vel, mass, acc, pad; the edge of a fixed box."""
    g = _generator(seed)
    b = torch.zeros(n, 12, device="cuda")
    size = 64.0
    if scene == "plummer":
        b[:, 0:3], b[:, 4:7] = _plummer(g, n)
        b[:, 7] = 1.0 / n
    elif scene == "pair":
        pos, vel = _plummer(g, n)
        side = torch.where(torch.arange(n, device="cuda") < n // 2, -0.5, 0.5)
        b[:, 0:3] = pos + side[:, None] * torch.tensor([10.0, 2.0, 0.0], device="cuda")
        b[:, 4:7] = vel - side[:, None] * torch.tensor([0.3, 0.0, 0.0], device="cuda")
        b[:, 7] = 2.0 / n
    elif scene == "cube":
        b[:, 0:3] = _uniform(g, n, 3)
        m = torch.exp(0.5 * torch.randn(n, generator=g, device="cuda"))
        b[:, 7] = m / m.sum()
        size = 4.0
    elif scene == "disk":
        # a thin disk around a heavy central body, as the reference's demonstration scenes
        r = 250.0 * torch.sqrt(_uniform(g, n))
        phi = 2 * math.pi * _uniform(g, n)
        b[:, 0], b[:, 1] = r * torch.cos(phi), r * torch.sin(phi)
        b[:, 2] = torch.randn(n, generator=g, device="cuda")
        v = torch.sqrt(1e6 / (r + 1))
        b[:, 4], b[:, 5] = -v * torch.sin(phi), v * torch.cos(phi)
        b[:, 7] = 1.0
        b[0] = 0
        b[0, 7] = 1e6
        size = 10000.0
    else:
        # halo: an exponential disk within a Hernquist halo, 12 : 4.777
        nd = int(round(n * 12 / 16.777))
        r = (-3.0 * torch.log(_uniform(g, nd, 2).clamp(min=1e-7).prod(1))).clamp(max=40.0)
        phi = 2 * math.pi * _uniform(g, nd)
        b[:nd, 0], b[:nd, 1] = r * torch.cos(phi), r * torch.sin(phi)
        b[:nd, 2] = 0.3 * torch.atanh((2 * _uniform(g, nd) - 1).clamp(-0.999999, 0.999999))
        b[:nd, 4], b[:nd, 5] = -0.5 * torch.sin(phi), 0.5 * torch.cos(phi)
        su = torch.sqrt(_uniform(g, n - nd) * (200.0 / 210.0) ** 2)
        b[nd:, 0:3] = _directions(g, n - nd) * (10 * su / (1 - su))[:, None]
        b[nd:, 4:7] = 0.3 * torch.randn(n - nd, 3, generator=g, device="cuda")
        b[:nd, 7] = 1.0 / nd
        b[nd:, 7] = 5.0 / nd
        size = 512.0
    # a body's radius: a hundredth of the mean spacing, which the cutoff law reads
    b[:, 3] = 0.01 * float((b[:, 0:3].amax(0) - b[:, 0:3].amin(0)).max()) / n ** (1.0 / 3.0)
    return b, size


def _eps2(case):
    return {"cube": 1e-6, "halo": 2.5e-5, "disk": 1e-2}.get(case.get("scene"), 1e-4)


def _dt(case):
    return {"disk": 1e-4, "halo": 2.5e-4}.get(case.get("scene"), 1e-3)


def _params(case, size=0.0):
    kind = case["kind"]
    law = native.LAW_CUTOFF if case.get("law") == "cutoff" else native.LAW_SOFTENED
    mode = {"batch": native.MODE_BATCHED, "bh": native.MODE_NLOGN, "pick": native.MODE_NLOGN}.get(kind, native.MODE_N2)
    precision = native.PREC_FP32
    if kind == "fp64":
        precision = native.PREC_FP64
    elif case.get("precision") == "comp":
        precision = native.PREC_COMPENSATED
    return native.params(dt=_dt(case), theta=case.get("theta", 0.5), G=G,
                         eps2=_eps2(case) if law == native.LAW_SOFTENED else 0.0, size=size, mode=mode, law=law,
                         precision=precision, tree_box=1 if case.get("box", "fitted") == "fitted" else 0,
                         walk=native.WALK_GROUP if case.get("walk") == "group" else native.WALK_TARGET)


def _layout(case):
    return native.LAYOUT_AOS if case.get("layout") == "aos" else native.LAYOUT_SOA


def _offsets(case):
    """System sizes, log-uniform in [lo, hi]: part of the case, so that outputs keep their shape."""
    u = np.random.Generator(np.random.Philox(case["systems"])).uniform(math.log(case["lo"]), math.log(case["hi"]), case["systems"])
    return np.concatenate([[0], np.cumsum(np.rint(np.exp(u)).astype(np.int64))])


# --- what a program has in hand ------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "ctx": native.Context(_layout(case))}
    ctx = state["ctx"]
    if kind == "batch":
        off = _offsets(case)
        bodies, size = _scene("plummer", int(off[-1]), seed)
        counts = torch.from_numpy(np.diff(off)).cuda()
        bodies[:, 7] = torch.repeat_interleave(1.0 / counts.float(), counts)
    else:
        bodies, size = _scene(case["scene"], case["n"], seed)
    state["p"] = _params(case, size)
    if kind == "accel":
        if case["layout"] == "aos":
            state["bodies"] = bodies
        else:
            state["pm"] = bodies[:, [0, 1, 2, 7]].contiguous()
            state["vr"] = bodies[:, [4, 5, 6, 3]].contiguous()
            state["acc"] = torch.zeros_like(state["pm"])
        torch.cuda.synchronize()
        return state
    host = bodies.cpu().numpy()
    del bodies
    # state in host memory is one array of Body records, written once and read into
    state["out"] = host.copy()
    if kind in ("steps", "batch") or (kind == "bh" and case["steps"]):
        state["in"] = host
    ctx.upload_bodies(host)
    if kind == "batch":
        ctx.set_systems(off)
    if kind == "pick":
        r = np.random.Generator(np.random.Philox(seed))
        origin = r.normal(0.0, 30.0, (case["rays"], 3)).astype(np.float32)
        at = host[r.integers(0, case["n"], case["rays"]), 0:3]
        state["rays"] = np.concatenate([origin, at - origin], 1).astype(np.float32)
    ctx.synchronize()
    return state


def run(state):
    case, ctx, p = state["case"], state["ctx"], state["p"]
    kind = case["kind"]
    if kind == "accel":
        if case["layout"] == "aos":
            ctx.dev_accel_aos(state["bodies"].data_ptr(), case["n"], p)
            return state["bodies"][:, 8:11]
        ctx.dev_accel_soa(state["pm"].data_ptr(), state["vr"].data_ptr(), state["acc"].data_ptr(), case["n"], p)
        return state["acc"]
    if kind == "energy":
        return ctx.energy(p)
    if kind == "pick":
        ctx.accelerate(p)
        hits, counts = ctx.tree_query(state["rays"], stop=native.QUERY_FIRST_BODY, max_hits=64)
        return {"hits": hits, "counts": counts}
    out = state["out"]
    if case.get("steps"):
        ctx.upload_bodies(state["in"])
        ctx.update_graph(p, case["steps"])
        ctx.download_bodies(into=out)
        return {"pos": out[:, 0:3], "vel": out[:, 4:7], "acc": out[:, 8:11]}
    ctx.accelerate(p)
    ctx.download_bodies(mask=native.READ_ACCELERATIONS, into=out)
    return out[:, 8:11]


# --- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        # the mean of a log-uniform size, and of its square
        span = math.log(case["hi"] / case["lo"])
        mean = (case["hi"] - case["lo"]) / span
        square = (case["hi"] ** 2 - case["lo"] ** 2) / (2 * span)
        return {"bytes": case["systems"] * mean * (48 * 2 + 96 * case["steps"]),
                "flops": 20.0 * case["systems"] * square * case["steps"]}
    n = case["n"]
    steps = max(1, case.get("steps", 1) or 1)
    if kind == "accel":
        return {"bytes": 32.0 * n, "flops": 20.0 * n * n}
    if kind == "steps":
        return {"bytes": n * (96.0 + 96.0 * steps), "flops": 20.0 * n * n * steps}
    if kind == "fp64":
        return {"bytes": 28.0 * n, "flops": 20.0 * n * n}
    if kind == "energy":
        # every pair once: three differences, their squares' sum, a root, a product and a sum
        return {"bytes": 32.0 * n, "flops": 0.5 * n * n * 12}
    if kind == "pick":
        # the tree's nodes (about four 48-byte records a body) written once, 30 nodes read a ray
        return {"bytes": n * (16.0 + 4 * 48) + case["rays"] * (24.0 + 260 + 30 * 48), "flops": 20.0 * n * math.log2(n)}
    # a tree over the bodies (a key and an index sorted, cells of 64 bytes), and per body about
    # 5 theta^2 + 4 interactions a level of the tree
    inter = (5.0 * case["theta"] ** 2 + 4.0) * math.log2(n)
    return {"bytes": steps * n * (16.0 + 24 + 32 + 16 + 16), "flops": steps * 20.0 * n * inter}


# --- the same in 64 bits -------------------------------------------------------------------------

def _accel64(x, m, eps2, r2):
    """Accelerations of all bodies; r2 is None for the softened law, else the cutoff per target."""
    n = x.shape[0]
    out = torch.empty_like(x)
    step = max(1, (1 << 26) // n)
    for i in range(0, n, step):
        d = [x[:, a][None, :] - x[i:i + step, a][:, None] for a in range(3)]
        s = d[0] * d[0]
        s.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        if r2 is None:
            w = torch.rsqrt(s + eps2)
        else:
            w = torch.where(s > r2[i:i + step, None], torch.rsqrt(s), 0.0)
        w = w * w * w * m[None, :]
        for a in range(3):
            out[i:i + step, a] = G * (d[a] * w).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pick", "bh"):
        return None     # whole numbers; sums over an approximation's own cells
    steps = max(1, case.get("steps", 1) or 1)
    eps2 = float(np.float32(_eps2(case)))
    dt = float(np.float32(_dt(case)))
    if kind == "batch":
        off = _offsets(case)
        if float(np.sum(np.diff(off).astype(np.float64) ** 2)) * steps > 5e10:
            return None
        bodies, _ = _scene("plummer", int(off[-1]), seed)
        counts = torch.from_numpy(np.diff(off)).cuda()
        bodies[:, 7] = torch.repeat_interleave(1.0 / counts.float(), counts)
        parts = [bodies[off[s]:off[s + 1]] for s in range(len(off) - 1)]
    else:
        if float(case["n"]) ** 2 * steps > 5e10:
            return None
        bodies, _ = _scene(case["scene"], case["n"], seed)
        parts = [bodies]
    if kind == "energy":
        x, v, m = bodies[:, 0:3].double(), bodies[:, 4:7].double(), bodies[:, 7].double()
        n = x.shape[0]
        step = max(1, (1 << 26) // n)
        pot = torch.zeros((), dtype=torch.float64, device="cuda")
        for i in range(0, n, step):
            s = (x[:, 0][None, :] - x[i:i + step, 0][:, None]) ** 2
            s += (x[:, 1][None, :] - x[i:i + step, 1][:, None]) ** 2
            s += (x[:, 2][None, :] - x[i:i + step, 2][:, None]) ** 2
            w = torch.rsqrt(s + eps2)
            k = torch.arange(w.shape[0], device="cuda")
            w[k, k + i] = 0.0
            pot += ((w * m[None, :]).sum(1) * m[i:i + step]).sum()
        return {"kinetic": 0.5 * float((m * (v * v).sum(1)).sum()), "potential": -0.5 * G * float(pot),
                "momentum": (m[:, None] * v).sum(0).cpu()}
    res = []
    for b in parts:
        x, v, m = b[:, 0:3].double(), b[:, 4:7].double(), b[:, 7].double()
        r2 = b[:, 3].double() ** 2 if case.get("law") == "cutoff" else None
        for k in range(steps):
            a = _accel64(x, m, eps2, r2)
            if kind in ("steps", "batch"):
                v = v + a * dt
                x = x + v * dt
        res.append((x, v, a))
    x, v, a = (torch.cat([r[k] for r in res]) for k in range(3))
    if kind in ("steps", "batch"):
        return {"pos": x.cpu(), "vel": v.cpu(), "acc": a.cpu()}
    if kind == "accel" and case["layout"] == "soa":
        return torch.cat([a, torch.zeros_like(a[:, :1])], 1)
    return a.cpu() if kind == "fp64" else a
