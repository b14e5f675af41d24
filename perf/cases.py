"""The workloads whose speed this framework is judged by, each through its public entry points.

A case is a dict of plain values; ``listed()`` gives the standing ones and
``draw(rng)`` more of the same ranges.  Kinds:

* ``step``      one eager build + walk + update of one system (``Context.step``): a program that
                looks at its bodies after every step;
* ``replay``    several steps of one system in one call (``Context.step`` with nsteps > 1, replayed
                from a CUDA graph): the inner loop of a simulation between two outputs;
* ``forces``    tree and accelerations only (``Context.build`` + ``Context.forces``): a program with
                an integrator of its own;
* ``batched``   many independent systems per launch (``Context.set_systems`` + ``graph_step``);
* ``adjoint``   forward trajectory and its gradients (``Adjoint.forward`` + ``backward``);
* ``host``      the reference's host class, phase by phase, with the copy back to the host
                (``BarnesHut.update``);
* ``energy``    the diagnostics of a run: potential, kinetic energy and momenta.

Bodies are the repository's workloads (star + disk, binary star + disk, Plummer sphere, their radius
laws, masses and constants as in ``nns_gb300.ic``), drawn on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nns_gb300 import ic
from nns_gb300.adjoint import Adjoint
from nns_gb300.barnes_hut import BarnesHut, Context, State

# ---- initial conditions on the GPU ---------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _u(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _disk(g, n, rmin, rmax, zfrac=0.01):
    r = rmin + (rmax - rmin) * _u(g, n)
    phi = 2.0 * math.pi * _u(g, n)
    z = zfrac * r * torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    v = torch.sqrt(1.0 / r)
    return torch.stack([r * phi.cos(), r * phi.sin(), z, v * phi.sin(), -v * phi.cos(), torch.zeros_like(r)])


def _star_disk(g, n):
    b = torch.empty(7, n, device="cuda", dtype=torch.float64)
    b[:6] = _disk(g, n, 0.1, 1.0)
    b[6] = 1e-6
    b[:, 0] = 0.0
    b[6, 0] = 1.0
    return b


def _binary_disk(g, n):
    b = torch.empty(7, n, device="cuda", dtype=torch.float64)
    b[:6] = _disk(g, n, 0.3, 2.0)
    b[6] = 1e-8
    vs = 0.5 * math.sqrt(1.0 / 0.2)
    for k, sgn in ((0, 1.0), (1, -1.0)):
        b[:, k] = torch.tensor([0.1 * sgn, 0.0, 0.0, 0.0, -vs * sgn, 0.0, 0.5], device="cuda", dtype=torch.float64)
    return b


def _sphere(g, n):
    ct = 2.0 * _u(g, n) - 1.0
    st = torch.sqrt(1.0 - ct * ct)
    ph = 2.0 * math.pi * _u(g, n)
    return torch.stack([st * ph.cos(), st * ph.sin(), ct])


def _plummer(g, n):
    b = torch.empty(7, n, device="cuda", dtype=torch.float64)
    u = (_u(g, n) * (1.0 + 1.0 / 400.0) ** -1.5).clamp_min(1e-12)
    r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    b[:3] = r * _sphere(g, n)
    q = torch.zeros_like(r)
    todo = torch.arange(n, device="cuda")
    while todo.numel():  # speeds by rejection on q^2 (1 - q^2)^(7/2)
        c = _u(g, todo.numel())
        ok = 0.1 * _u(g, todo.numel()) < c * c * (1.0 - c * c) ** 3.5
        q[todo[ok]] = c[ok]
        todo = todo[~ok]
    b[3:6] = q * math.sqrt(2.0) * (1.0 + r * r) ** -0.25 * _sphere(g, n)
    b[6] = 1.0 / n
    return b


_MODELS = {"star_disk": _star_disk, "binary_disk": _binary_disk, "plummer": _plummer}
# softening and time step of each model's workload
_EPS = {"star_disk": 0.01, "binary_disk": 0.005, "plummer": 0.01}
_DT = {"star_disk": 1e-3, "binary_disk": 5e-4, "plummer": 1e-3}
_THETA = 0.5


def _offsets(case):
    sizes = ic.batched_sizes(case["systems"], ic.SEED0 + case.get("sizes_seed", 0), case["lo"], case["hi"])
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)


def _bodies(case, seed):
    """(7, n) float32 on the GPU: x, y, z, vx, vy, vz, m."""
    g = _gen(seed)
    if case["kind"] == "batched":  # independent star + disk systems
        off = _offsets(case)
        b = _star_disk(g, int(off[-1]))
        at = torch.as_tensor(off[:-1], device="cuda")
        b[:6, at] = 0.0
        b[6, at] = 1.0
        return b.float()
    return _MODELS[case["model"]](g, case["n"]).float()


def _state(b):
    z = lambda: torch.zeros(b.shape[1], dtype=torch.float32, device="cuda")  # noqa: E731
    r = [b[k].clone() for k in range(7)]
    return State(*r[:6], z(), z(), z(), r[6])


# ---- the cases -----------------------------------------------------------------------------------


def listed():
    return [
        # the smallest simulation in earnest: a thousand bodies, stepped one by one
        {"name": "step_star_1000", "kind": "step", "model": "star_disk", "n": 1000},
        # a small cluster in a program with its own integrator; an odd size
        {"name": "forces_plummer_5003", "kind": "forces", "model": "plummer", "n": 5003},
        # the 16384-body star + disk configuration, ten steps per call
        {"name": "replay_star_16384", "kind": "replay", "model": "star_disk", "n": 16384, "steps": 10},
        # the reference's host class at the reference's disk size: every phase entry point, timed
        # phases, bodies copied back each step
        {"name": "host_star_32768", "kind": "host", "model": "star_disk", "n": 32768},
        # the trajectory-gradient workload, shortened: checkpoints, recompute, reverse pass
        {"name": "adjoint_plummer_65536", "kind": "adjoint", "model": "plummer", "n": 65536, "steps": 8, "every": 4},
        # energy and momenta of a mid-size cluster, as a run's log takes them
        {"name": "energy_plummer_100003", "kind": "energy", "model": "plummer", "n": 100003},
        # an ordinary cluster between two outputs
        {"name": "replay_plummer_131071", "kind": "replay", "model": "plummer", "n": 131071, "steps": 4},
        # a survey of independent small systems, uneven sizes
        {"name": "batched_200", "kind": "batched", "systems": 200, "lo": 10.0, "hi": 16.0},
        # the accurate form: cell quadrupoles
        {"name": "step_quad_700001", "kind": "step", "model": "binary_disk", "n": 700001, "multipole": 1},
        # the Plummer 2^20 configuration
        {"name": "step_plummer_1048576", "kind": "step", "model": "plummer", "n": 1 << 20},
        # Hilbert order with compensated sums, a size that is no power of two
        {"name": "step_comp_hilbert_3000001", "kind": "step", "model": "binary_disk", "n": 3000001,
         "compensated": 1, "key_order": 1},
        # the headline: 2^24 bodies of the binary star + disk
        {"name": "step_binary_16777216", "kind": "step", "model": "binary_disk", "n": 1 << 24},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "replay", "replay", "forces", "batched", "adjoint", "host", "energy"])
    model = rng.choice(["star_disk", "binary_disk", "plummer"])
    if kind == "step":
        c = {"kind": kind, "model": model, "n": _size(rng, 1000, 1 << 23)}
        opt = rng.choice(["", "", "multipole", "compensated", "compensated2", "key_order", "leaf_size"])
        if opt:
            c["n"] = min(c["n"], 4000000 if opt != "multipole" else 2000000)
            c[opt.rstrip("2")] = {"compensated2": 2, "leaf_size": 4}.get(opt, 1)
        return c
    if kind == "replay":
        return {"kind": kind, "model": model, "n": _size(rng, 1000, 1000000), "steps": rng.randint(2, 10)}
    if kind == "forces":
        return {"kind": kind, "model": model, "n": _size(rng, 1000, 4000000)}
    if kind == "batched":
        lo = rng.uniform(8.0, 11.0)
        return {"kind": kind, "systems": rng.randint(8, 400), "lo": lo, "hi": lo + rng.uniform(2.0, 5.0),
                "sizes_seed": rng.randint(1, 1000)}
    if kind == "adjoint":
        every = rng.randint(2, 4)
        return {"kind": kind, "model": "plummer", "n": _size(rng, 2000, 65536), "steps": every * rng.randint(1, 2) + rng.randint(0, 1), "every": every}
    if kind == "host":
        return {"kind": kind, "model": model, "n": _size(rng, 1000, 200000)}
    return {"kind": kind, "model": model, "n": _size(rng, 1000, 400000)}


def prepare(case, seed):
    b = _bodies(case, seed)
    n, kind = b.shape[1], case["kind"]
    model = case.get("model", "star_disk")
    kw = dict(theta=_THETA, eps=_EPS[model], dt=_DT[model])
    if kind == "host":
        h = b.cpu().numpy()
        bh = BarnesHut(ic.Bodies(*(h[k] for k in range(7))), timestep=kw["dt"], theta=_THETA, eps=kw["eps"])
        return {"case": case, "bh": bh}
    off = _offsets(case) if kind == "batched" else np.array([0, n], np.int64)
    ctx = Context(max_bodies=n, max_systems=len(off) - 1, compensated=case.get("compensated", 0),
                  key_order=case.get("key_order", 0), multipole=case.get("multipole", 0),
                  leaf_size=case.get("leaf_size", 1), **kw)
    ctx.set_systems(off)
    st = {"case": case, "ctx": ctx, "s": _state(b)}
    if kind == "adjoint":
        st["adj"] = Adjoint(ctx, case["steps"], checkpoint_every=case["every"], list_capacity=8192)
        # the fit's target: the bodies where they would drift to, a little off
        noise = torch.randn(3, n, generator=_gen(seed + 1), device="cuda", dtype=torch.float32)
        st["target"] = b[:3] + (case["steps"] * kw["dt"]) * b[3:6] + 0.01 * noise
        st["b"] = b
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host":
        bh = state["bh"]
        n = bh.numParticles
        bh.update()
        return {"x": bh.h_x, "y": bh.h_y, "z": bh.h_z, "vx": bh.h_vx, "vy": bh.h_vy, "vz": bh.h_vz,
                "ax": bh.d_ax[:n], "ay": bh.d_ay[:n], "az": bh.d_az[:n]}
    ctx, s = state["ctx"], state["s"]
    if kind == "forces":
        ctx.build(s)
        ctx.forces(s)
        return {"ax": s.ax, "ay": s.ay, "az": s.az}
    if kind == "energy":
        ctx.build(s)
        phi = ctx.potential(s)
        d = ctx.diagnostics(s)
        return {"phi": phi, "momentum": d["momentum"], "angular_momentum": d["angular_momentum"],
                "kinetic": float(d["kinetic"]), "mass": float(d["mass"])}
    if kind == "adjoint":
        # one evaluation of a fit: loss and gradients from the present parameters
        b = state["b"]
        for k, t in enumerate((s.x, s.y, s.z, s.vx, s.vy, s.vz)):
            t.copy_(b[k])
        loss = state["adj"].forward(s, state["target"])
        gx, gv, gm = state["adj"].backward(s)
        return {"loss": loss, "gx": gx, "gv": gv, "gm": gm, "x": s.x, "y": s.y, "z": s.z}
    if kind == "batched":
        ctx.graph_step(s, 1)
    else:
        ctx.step(s, case.get("steps", 1))
    return {"x": s.x, "y": s.y, "z": s.z, "vx": s.vx, "vy": s.vy, "vz": s.vz, "ax": s.ax, "ay": s.ay, "az": s.az}


# ---- the work a case cannot do without -----------------------------------------------------------


def _list_length(model, n):
    """Interactions per body at theta = 0.5, as the tree walks of these models count them."""
    x = math.log2(max(n, 2))
    pts = _LISTS[model]
    x = min(max(x, pts[0][0]), pts[-1][0])
    for (x0, y0), (x1, y1) in zip(pts, pts[1:]):
        if x <= x1:
            return y0 + (y1 - y0) * (x - x0) / (x1 - x0)
    return pts[-1][1]


# (log2 n, interactions per body) measured over the range
_LISTS = {
    "star_disk": ((8, 236), (10, 574), (12, 1067), (14, 1825), (16, 3007), (17, 3828), (18, 4806), (20, 7356),
                  (22, 9835), (24, 12025)),
    "binary_disk": ((8, 232), (10, 561), (12, 1050), (14, 1838), (16, 3084), (17, 3941), (18, 5000), (20, 7879),
                    (22, 11373), (24, 15996)),
    "plummer": ((8, 226), (10, 613), (12, 1077), (14, 1684), (16, 2539), (18, 2681), (20, 3021), (22, 3168),
                (24, 3310)),
}


def work(case):
    kind = case["kind"]
    if kind == "batched":
        sizes = np.diff(_offsets(case))
        n = int(sizes.sum())
        inter = float(sum(k * min(k, _list_length("star_disk", int(k))) for k in sizes))
    else:
        n = case["n"]
        inter = n * min(float(n), _list_length(case["model"], n))
    # 20 flops an interaction (3 differences, r^2, r^-3 m, 3 multiply-adds); a quadrupole term adds 46
    flops = inter * (20 + (46 if case.get("multipole") else 0))
    if kind == "forces":
        return {"bytes": 4.0 * n * 7, "flops": flops}
    if kind == "energy":
        return {"bytes": 4.0 * n * 8, "flops": inter * 13 + 25 * n}
    if kind == "host":
        return {"bytes": 4.0 * n * (10 + 9 + 6), "flops": flops + 12 * n}
    if kind == "adjoint":
        # forward, then the recompute of all but the last segment, then the reverse products
        seg = -(-case["steps"] // case["every"])
        again = (seg - 1) * case["every"]
        return {"bytes": 4.0 * n * (10 + 10 + 10) * case["steps"],
                "flops": flops * (case["steps"] + again) + inter * 44 * case["steps"]}
    steps = case.get("steps", 1)
    return {"bytes": 4.0 * n * (10 + 9) * steps, "flops": (flops + 12 * n) * steps}


# ---- 64-bit values -------------------------------------------------------------------------------


def _pairs(p, q, m, eps2, out):
    """Sums over all bodies of q for the bodies of p, block by block; out(d, r2, m) -> (k, block) terms."""
    n = p.shape[1]
    block = max(1, min(n, (1 << 26) // max(1, q.shape[1])))
    res = []
    for i in range(0, n, block):
        d = q[:, None, :] - p[:, i:i + block, None]
        r2 = (d * d).sum(0) + eps2
        res.append(out(d, r2, m, i))
    return torch.cat(res, -1)


def _acc64(x, m, eps2):
    def term(d, r2, m, i):
        f = m / (r2 * r2.sqrt())
        return (f * d).sum(-1)
    return _pairs(x, x, m, eps2, term)


def _phi64(x, m, eps2):
    def term(d, r2, m, i):
        f = m / r2.sqrt()
        k = torch.arange(f.shape[0], device=f.device)
        f[k, k + i] = 0.0
        return -f.sum(-1)
    return _pairs(x, x, m, eps2, term)


def _steps64(x, v, m, eps2, dt, steps, off=None):
    for _ in range(steps):
        if off is None:
            a = _acc64(x, m, eps2)
        else:
            a = torch.cat([_acc64(x[:, b:e], m[b:e], eps2) for b, e in zip(off[:-1], off[1:])], -1)
        v = v + dt * a
        x = x + dt * v
    return x, v, a


def _vjp64(x, m, g, eps2):
    """(gradient to x, gradient to m) of sum_i g_i . a_i(x, m)."""
    gm = torch.zeros_like(m)
    gx = torch.zeros_like(x)
    n = x.shape[1]
    block = max(1, min(n, (1 << 25) // n))
    for i in range(0, n, block):
        d = x[:, None, :] - x[:, i:i + block, None]
        r2 = (d * d).sum(0) + eps2
        gi = g[:, i:i + block, None]
        i3 = 1.0 / (r2 * r2.sqrt())
        dg = (d * gi).sum(0)
        gm += (dg * i3).sum(0)
        w = m * i3
        t = w * gi - (3.0 * w * dg / r2) * d
        gx += t.sum(1)
        gx[:, i:i + block] -= t.sum(2)
    return gx, gm


def exact(case, seed):
    """Direct sums over all pairs in 64 bits: a tree code's outputs are off from them by the opening
    angle's error in the forces, and by rounding in everything that a small time step multiplies."""
    kind = case["kind"]
    if kind == "batched":
        off = [int(k) for k in _offsets(case)]
        if sum((e - b) ** 2 for b, e in zip(off[:-1], off[1:])) > 2e11:
            return None
    else:
        off = None
        steps = case.get("steps", 1)
        if case["n"] ** 2 * steps * (4 if kind == "adjoint" else 1) > 2e11:
            return None
    b = _bodies(case, seed).double()
    model = case.get("model", "star_disk")
    eps2 = float(np.float32(_EPS[model]) * np.float32(_EPS[model]))
    dt = float(np.float32(_DT[model]))
    x, v, m = b[:3], b[3:6], b[6]
    if kind == "forces":
        a = _acc64(x, m, eps2)
        return {"ax": a[0], "ay": a[1], "az": a[2]}
    if kind == "energy":
        return {"phi": _phi64(x, m, eps2), "momentum": (m * v).sum(-1),
                "angular_momentum": (m * torch.linalg.cross(x, v, dim=0)).sum(-1),
                "kinetic": float((0.5 * m * (v * v).sum(0)).sum()), "mass": float(m.sum())}
    if kind == "adjoint":
        noise = torch.randn(3, case["n"], generator=_gen(seed + 1), device="cuda", dtype=torch.float32)
        f = _bodies(case, seed)
        target = (f[:3] + (case["steps"] * _DT[model]) * f[3:6] + 0.01 * noise).double()
        path = []
        for _ in range(case["steps"]):
            path.append(x)
            x, v, _a = _steps64(x, v, m, eps2, dt, 1)
        lx, lv, lm = 2.0 * (x - target), torch.zeros_like(v), torch.zeros_like(m)
        for p in reversed(path):
            lv = lv + dt * lx
            gx, gm = _vjp64(p, m, dt * lv, eps2)
            lx, lm = lx + gx, lm + gm
        return {"loss": float(((x - target) ** 2).sum()), "gx": lx, "gv": lv, "gm": lm, "x": x[0], "y": x[1], "z": x[2]}
    x, v, a = _steps64(x, v, m, eps2, dt, case.get("steps", 1), off)
    return {"x": x[0], "y": x[1], "z": x[2], "vx": v[0], "vy": v[1], "vz": v[2], "ax": a[0], "ay": a[1], "az": a[2]}
