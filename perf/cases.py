"""The work whose speed counts: whole calls of the step engine, as programs make them.

A case is a dict of plain values.  listed() names the standing ones, draw() gives one more
of the same ranges, prepare() what a program holds before the call, run() one call and its
outputs, work() the bytes and operations the call cannot do without, exact() the same
outputs from plain 64-bit arithmetic where a direct sum can be had in reasonable time.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-nbody_gb300"))
import nbh  # noqa: E402
from nbh import learned  # noqa: E402

EXACT_PAIRS = 1.5e11       # direct sums of more pairs than this take too long in 64 bits


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # the smallest universes, stepped and drawn one frame at a time: launches and latency count
        {"name": "frame_1000", "kind": "step", "universe": "plummer", "n": 1000, "dt": 0.01},
        # a small ball whose arrays the host owns: written, stepped and read back on every call
        # (16,384 bodies at the vote width the tuner picks for them, 32)
        {"name": "ball_io_16384", "kind": "io", "universe": "ball", "n": 16384, "dt": 0.025, "vote": 32},
        # the ordinary run: a sphere of a million bodies, launch geometry tuned once at start
        {"name": "plummer_1m", "kind": "step", "universe": "plummer", "n": 1 << 20, "dt": 0.01, "tuned": True},
        # the same, with the state owned by the host (analysis or rendering there on every step)
        {"name": "plummer_io_1m", "kind": "io", "universe": "plummer", "n": 1 << 20, "dt": 0.01},
        # a production run at a size where tree and bodies are far larger than the caches
        {"name": "plummer_16m", "kind": "step", "universe": "plummer", "n": 1 << 24, "dt": 0.01},
        # a parameter study: 256 independent universes of 1K to 64K bodies advanced together
        {"name": "ensemble_256", "kind": "ensemble", "universes": 256, "lo": 1024, "hi": 65536, "dt": 0.01},
        # a disc galaxy with a central mass, compensated sums: long runs with small increments
        {"name": "disc_precise_4m", "kind": "step", "universe": "disc", "n": 1 << 22, "dt": 0.01, "precise": True},
        # the reference's own arithmetic, work-group and constants: checking against older results
        {"name": "reference_100003", "kind": "step", "universe": "plummer", "n": 100003, "dt": 0.025, "vote": 16,
         "reference": True, "theta2": 1.5, "eps2": 0.0025},
        # the learned opening angle over one cycle of its model (8 steps, one evaluation)
        {"name": "learned_1m", "kind": "learned", "universe": "plummer", "n": 1 << 20, "dt": 0.01, "steps": 8},
        # the force error of a run: FP64 direct sum on a sample of its bodies
        {"name": "direct_1m", "kind": "direct", "universe": "plummer", "n": 1 << 20, "sample": 16384},
        # the energy balance of a run: moments and the pair potential
        {"name": "energy_200003", "kind": "energy", "universe": "plummer", "n": 200003},
        # fitting an opening-angle model to probe data
        {"name": "train_100000", "kind": "train", "n": 100000, "iters": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "io", "ensemble", "reference", "learned", "direct", "energy", "train"])
    if kind == "step":
        universe = rng.choice(["plummer", "plummer", "disc"])
        precise = universe == "disc" and rng.random() < 0.5
        c = {"kind": "step", "universe": universe, "n": _log_int(rng, 8, 1 << (22 if universe == "disc" else 24)),
             "dt": 0.01, "theta": round(rng.uniform(0.4, 0.9), 2), "vote": rng.choice([64, 64, 64, 32, 128])}
        if precise:
            c["precise"] = True
        if rng.random() < 0.3 and c["n"] <= 1 << 21:
            c["tuned"] = True
        return c
    if kind == "io":
        return {"kind": "io", "universe": rng.choice(["ball", "plummer"]), "n": _log_int(rng, 1000, 1 << 22),
                "dt": 0.01, "vote": rng.choice([64, 64, 32])}
    if kind == "ensemble":
        lo = _log_int(rng, 100, 4000)
        hi = _log_int(rng, 2 * lo, 65536)
        return {"kind": "ensemble", "universes": _log_int(rng, 2, 256), "lo": lo, "hi": hi, "dt": 0.01}
    if kind == "reference":
        return {"kind": "step", "universe": "plummer", "n": _log_int(rng, 8, 1 << 20), "dt": 0.025,
                "vote": rng.choice([16, 16, 32]), "reference": True, "theta2": 1.5, "eps2": 0.0025}
    if kind == "learned":
        return {"kind": "learned", "universe": "plummer", "n": _log_int(rng, 16384, 1 << 21), "dt": 0.01, "steps": 8}
    if kind == "direct":
        return {"kind": "direct", "universe": "plummer", "n": _log_int(rng, 1000, 1 << 20),
                "sample": _log_int(rng, 100, 16384)}
    if kind == "energy":
        return {"kind": "energy", "universe": "plummer", "n": _log_int(rng, 30000, 300000)}
    return {"kind": "train", "n": _log_int(rng, 5000, 200000), "iters": 100}


# ---- universes ------------------------------------------------------------------------------

def _direction(g, n):
    z = 2.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1.0
    phi = 2.0 * math.pi * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    s = (1.0 - z * z).sqrt()
    return torch.stack([s * phi.cos(), s * phi.sin(), z])


def _speed_fraction(g, n):
    """v / v_escape of a Plummer sphere: density ~ q^2 (1 - q^2)^3.5, by its inverted table."""
    q = torch.linspace(0.0, 1.0, 4097, device="cuda", dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1.0 - q * q) ** 3.5, 0)
    cdf = cdf / cdf[-1].clone()
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    k = torch.searchsorted(cdf, u).clamp(1, 4096)
    f = (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp_min(1e-300)
    return q[k - 1] + f.clamp(0.0, 1.0) * (q[k] - q[k - 1])


def _plummer(g, n, a=1.0):
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.998 + 1e-9
    r = a / (u ** (-2.0 / 3.0) - 1.0).sqrt()
    pos = _direction(g, n) * r
    vel = _direction(g, n) * (_speed_fraction(g, n) * math.sqrt(2.0) * (r * r + a * a) ** -0.25)
    return pos, vel, torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


def _ball(g, n):
    r = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) ** (1.0 / 3.0)
    pos = _direction(g, n) * r
    vel = 0.05 * torch.randn(3, n, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel, torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


def _disc(g, n, zd=0.1, center=0.1, halo=0.1):
    """Body 0 is the central mass; exponential disc on near-circular orbits; Plummer halo."""
    nh = int(halo * (n - 1))
    nd = n - 1 - nh
    ah = 3.0

    def enclosed(r):
        return center + (1.0 - halo) * (1.0 - (1.0 + r) * (-r).exp()) + halo * r ** 3 / (r * r + ah * ah) ** 1.5
    u = torch.rand(4, nd, generator=g, device="cuda", dtype=torch.float64).clamp(1e-12, 1.0 - 1e-12)
    R, phi = -(u[0] * u[1]).log(), 2.0 * math.pi * u[2]
    pos = torch.stack([R * phi.cos(), R * phi.sin(), zd * torch.atanh(2.0 * u[3] - 1.0)])
    vc = (enclosed(R) / R).sqrt()
    vel = torch.stack([-phi.sin(), phi.cos(), torch.zeros_like(R)]) * vc
    vel += 0.05 * vc * torch.randn(3, nd, generator=g, device="cuda", dtype=torch.float64)
    hp, hv, _ = _plummer(g, nh, ah) if nh else (pos[:, :0], vel[:, :0], None)
    zero = torch.zeros(3, 1, device="cuda", dtype=torch.float64)
    m = torch.full((n,), 1.0 / max(1, n - 1), device="cuda", dtype=torch.float64)
    m[0] = center
    return torch.cat([zero, pos, hp], 1), torch.cat([zero, vel, hv], 1), m


def _counts(case):
    """Bodies of each universe of an ensemble: log-uniform between lo and hi, a fixed choice per case."""
    r = np.random.RandomState(case["universes"])
    return np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["universes"])).astype(np.int32)


def _bodies(case, seed):
    """x y z vx vy vz m (float32 host arrays) and the universes' counts."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["kind"] == "ensemble":
        counts = _counts(case)
        pos, vel, _ = _plummer(g, int(counts.sum()))
        m = torch.from_numpy(np.repeat(1.0 / counts, counts)).cuda()
    else:
        counts = np.array([case["n"]], np.int32)
        pos, vel, m = {"plummer": _plummer, "ball": _ball, "disc": _disc}[case["universe"]](g, case["n"])
    both = torch.cat([pos, vel, m[None]]).float().cpu().numpy()
    return [both[k] for k in range(7)], counts


def _config(case):
    kw = {"theta": case.get("theta", 0.5), "eps": 0.05, "dt": case.get("dt", 0.01),
          "precise": case.get("precise", False), "theta2": case.get("theta2", 0.0), "eps2": case.get("eps2", 0.0)}
    if "vote" in case:
        kw["vote_width"] = case["vote"]
    if case.get("reference"):
        kw["arith"] = nbh.NBH_ARITH_REFERENCE
    return kw


def _samples(case, seed):
    """Probe-like data: normalised features, log angles that depend on a few of them, noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    X = torch.randn(case["n"], 12, generator=g, device="cuda")
    noise = 0.15 * torch.randn(case["n"], generator=g, device="cuda")
    Y = (-0.5 + 0.2 * torch.tanh(X[:, 0] - 0.5 * X[:, 3]) + 0.1 * X[:, 7] * X[:, 1].sigmoid() + noise).clamp(-1.2, 0.0)
    return X.cpu().numpy(), Y.cpu().numpy()


# ---- what a program holds, and one call ---------------------------------------------------------

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        X, Y = _samples(case, seed)
        return {"kind": kind, "X": X, "Y": Y, "iters": case["iters"]}
    arrays, counts = _bodies(case, seed)
    n = int(counts.sum())
    sim = nbh.Simulation(**_config(case))
    if kind == "ensemble":
        sim.load_batch(counts, *arrays)
    else:
        sim.load(*arrays)
    if case.get("tuned"):
        sim.autotune()
    state = {"kind": kind, "sim": sim, "steps": case.get("steps", 1)}
    if kind in ("step", "ensemble", "learned"):
        if kind == "learned":
            learned.install(sim, learned.load_model(learned.default_model_path()))
        state["pos"] = torch.empty(n, 4, device="cuda")
        state["vel"] = torch.empty(n, 4, device="cuda")
    elif kind == "io":
        pinned = [torch.empty(n, pin_memory=True) for _ in range(15)]
        for t, a in zip(pinned, arrays[:6]):
            t.copy_(torch.from_numpy(a))
        state["in"] = dict(zip(KEYS, (t.numpy() for t in pinned[:6])))
        state["out"] = dict(zip(KEYS, (t.numpy() for t in pinned[6:])))
        state["pinned"] = pinned
    elif kind == "direct":
        state["idx"] = np.sort(np.random.RandomState(seed & 0x7fffffff).choice(n, min(case["sample"], n), replace=False)
                               ).astype(np.int32)
    return state


def run(state):
    kind = state["kind"]
    if kind == "train":
        model = learned.train(state["X"], state["Y"], quantile=0.2, iters=state["iters"])
        return [model["params"], model["mean"], model["inv_std"], model["loss"]]
    sim = state["sim"]
    if kind == "io":
        sim.step_io(1, write=state["in"], read=state["out"])
        return [state["out"][k] for k in KEYS]
    if kind == "direct":
        return sim.direct_f64(state["idx"])
    if kind == "energy":
        return sim.diagnostics(potential=True)
    sim.step(state["steps"])
    sim.export_float4(state["pos"].data_ptr(), state["vel"].data_ptr())
    return [state["pos"], state["vel"]]


# ---- what a call cannot do without -----------------------------------------------------------

def _interactions(n, theta):
    """Accepted interactions of one body, about: every body of a small universe, and a number that
    grows with log N in a large one (measured 3,700 at a million bodies and theta 0.5 in groups of 64)."""
    return min(float(n), 150.0 * math.log2(max(2, n)) * min(2.0, (0.5 / theta) ** 2))


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["n"]
        return {"bytes": 4.0 * (13 * n + 2 * 5057 + 24), "flops": 6.0 * (12 * 64 + 64 * 64 + 64) * n * case["iters"]}
    if kind == "ensemble":
        counts = _counts(case).tolist()
    else:
        counts = [case["n"]]
    n = sum(counts)
    theta = math.sqrt(case["theta2"]) if case.get("theta2") else case.get("theta", 0.5)
    if kind == "direct":
        k = min(case["sample"], n)
        return {"bytes": 16.0 * n + 28.0 * k, "flops": 20.0 * n * k}
    if kind == "energy":
        return {"bytes": 28.0 * n, "flops": 18.0 * n * n / 2}
    flops = 20.0 * sum(c * _interactions(c, theta) for c in counts) * case.get("steps", 1)
    if kind == "io":
        return {"bytes": 4.0 * n * (7 + 9), "flops": flops}
    # state in (positions, masses, velocities, accelerations) and out, and the two exported arrays
    return {"bytes": n * (40.0 + 36.0) * case.get("steps", 1) + 32.0 * n, "flops": flops}


# ---- 64-bit values ------------------------------------------------------------------------------

def _direct(pos, m, rows, eps2):
    """Accelerations (3, len(rows)) of the bodies `rows` by the direct sum in 64 bits."""
    out = torch.empty(3, rows.numel(), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 26) // pos.shape[1])
    for a in range(0, rows.numel(), step):
        at = pos[:, rows[a:a + step]]
        d = [pos[k][None] - at[k][:, None] for k in range(3)]
        d2 = (d[0] * d[0]).addcmul_(d[1], d[1]).addcmul_(d[2], d[2]).add_(eps2)
        inv = d2.rsqrt_()
        f = (inv * inv).mul_(inv).mul_(m[None])
        for k in range(3):
            out[k, a:a + step] = d[k].mul_(f).sum(1)
    return out


def _potentials(pos, m, eps2):
    soft = plain = 0.0
    n = pos.shape[1]
    step = max(1, (1 << 26) // n)
    for a in range(0, n, step):
        at = pos[:, a:a + step]
        d = [pos[k][None] - at[k][:, None] for k in range(3)]
        d2 = (d[0] * d[0]).addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        k = torch.arange(at.shape[1], device="cuda")
        mm = m[a:a + step, None] * m[None]
        mm[k, a + k] = 0.0
        d2[k, a + k] = 1.0
        soft += float((mm / (d2 + eps2).sqrt()).sum())
        plain += float((mm / d2.sqrt()).sum())
    return -0.5 * soft, -0.5 * plain


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "learned"):
        return None
    counts = _counts(case).tolist() if kind == "ensemble" else [case["n"]]
    rows = min(case["sample"], case["n"]) if kind == "direct" else None
    pairs = float(rows) * case["n"] if kind == "direct" else sum(float(c) * c for c in counts)
    if pairs > EXACT_PAIRS:
        return None
    arrays, _ = _bodies(case, seed)
    t = torch.from_numpy(np.stack(arrays)).cuda().double()
    pos, vel, m = t[:3], t[3:6], t[6]
    n = pos.shape[1]
    eps2 = float(np.float32(case["eps2"])) if case.get("eps2") else float(np.float32(0.05) * np.float32(0.05))
    if kind == "direct":
        idx = np.sort(np.random.RandomState(seed & 0x7fffffff).choice(n, rows, replace=False))
        return [a.cpu().numpy() for a in _direct(pos, m, torch.from_numpy(idx).cuda(), eps2)]
    if kind == "energy":
        soft, plain = _potentials(pos, m, eps2)
        kinetic = float(0.5 * (m * (vel * vel).sum(0)).sum())
        cross = torch.linalg.cross(pos, vel, dim=0)
        return [{"mass": float(m.sum()), "com": [float(v) for v in (pos * m).sum(1) / m.sum()],
                 "momentum": [float(v) for v in (vel * m).sum(1)],
                 "angular_momentum": [float(v) for v in (cross * m).sum(1)], "kinetic": kinetic, "max_depth": None,
                 "potential": soft, "potential_unsoftened": plain, "total": kinetic + soft}]
    acc = torch.empty(3, n, device="cuda", dtype=torch.float64)
    at = 0
    for c in counts:
        acc[:, at:at + c] = _direct(pos[:, at:at + c], m[at:at + c], torch.arange(c, device="cuda"), eps2)
        at += c
    dt = float(np.float32(case.get("dt", 0.01)))
    pos, vel = pos + (vel + acc * (0.5 * dt)) * dt, vel + acc * dt
    if kind == "io":
        return [v.cpu().numpy() for v in torch.cat([pos, vel, acc])]
    one = torch.ones(1, n, device="cuda", dtype=torch.float64)
    return [torch.cat([pos, one]).T.contiguous(), torch.cat([vel, one]).T.contiguous()]
