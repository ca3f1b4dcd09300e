"""Performance cases of the framework: what a user's program has it do, through its public entry points.

A case is a dict of plain values.  ``kind`` says which entry points a pass goes through:

* ``round``    the reference's round on its N x 10 records: bh_load_records, then per round create_tree,
               summarize, evaluate, timestep, and the records back (the drop-in's call sequence), with the
               reference's flat far field
* ``step``     fused steps in theta mode from arrays on the device: load, step / step_graph, store
* ``batch``    the same over many independent systems of uneven size in one plan
* ``learned``  a step with the learned far-field correction
* ``direct``   the FP64 direct-sum accelerations of sampled particles (the --check sampler)
* ``train``    one training step of the correction's network: gradients of a batch, then Adam
* ``infer``    the network's forward pass over a set of feature rows

Sizes come from this repository's configurations, tests and benchmark.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "barnes-hut_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from barneshut.gb300 import learned, native  # noqa: E402

PREC = {"fp32": native.BH_PREC_FP32, "kahan": native.BH_PREC_FP32_KAHAN, "fp64": native.BH_PREC_FP64}
DEV = "cuda"


# ------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest whole call: one round of the reference's algorithm on a few thousand particles
        # (launches and latency count)
        {"name": "round_2k", "kind": "round", "n": 2000, "grid": 8, "layout": "uniform", "rounds": 1,
         "cutoff": 1e-5, "dt": 1e-4},
        # the reference GPU path's semantics on its own kind of input: generated particles over
        # [0, 499)^2, default 1000 particles per box
        {"name": "round_gpu_100k", "kind": "round", "n": 100003, "grid": 12, "layout": "generated", "rounds": 1,
         "cutoff": 0.0, "dt": 5e-3},
        # a small simulation advanced ten steps per call by the captured graph (10,000 uniform
        # particles, 16 x 16 boxes, theta 0.5)
        {"name": "sim_10k", "kind": "step", "n": 10000, "grid": 16, "layout": "uniform", "theta": 0.5,
         "eps": 1e-3, "dt": 1e-4, "prec": "kahan", "steps": 10, "graph": True, "order": "file", "group": 0,
         "dense": 0, "quad": 0},
        # an ordinary simulation, stepped eagerly, plain FP32 sums, a looser angle, ragged sizes
        {"name": "sim_131k_fp32", "kind": "step", "n": 131071, "grid": 45, "layout": "gauss", "theta": 0.7,
         "eps": 1e-4, "dt": 1e-5, "prec": "fp32", "steps": 1, "graph": False, "order": "file", "group": 0,
         "dense": 0, "quad": 0},
        # the precision study's FP64 pairs
        {"name": "sim_65k_fp64", "kind": "step", "n": 65536, "grid": 32, "layout": "cluster", "theta": 0.5,
         "eps": 1e-4, "dt": 1e-5, "prec": "fp64", "steps": 1, "graph": False, "order": "file", "group": 0,
         "dense": 0, "quad": 0},
        # the 1M cluster mixture on 256 x 256 boxes, a few steps per call
        {"name": "sim_1m", "kind": "step", "n": 1048576, "grid": 256, "layout": "cluster", "theta": 0.5,
         "eps": 1e-4, "dt": 1e-5, "prec": "kahan", "steps": 4, "graph": True, "order": "file", "group": 0,
         "dense": 0, "quad": 0},
        # the 4M cluster mixture on 512 x 512 boxes with the autotuner's usual tile, one step from the
        # state of a running simulation (the benchmark's step)
        {"name": "sim_4m", "kind": "step", "n": 4194304, "grid": 512, "layout": "cluster", "theta": 0.5,
         "eps": 1e-4, "dt": 1e-5, "prec": "kahan", "steps": 1, "graph": True, "order": "sorted", "group": 4,
         "dense": 16, "quad": 128},
        # 512 independent systems of log-uniform size in one plan, ~64 particles per box
        {"name": "batch_512", "kind": "batch", "systems": 512, "spread": 4, "nmin": 1024, "nmax": 262144, "per_box": 64,
         "theta": 0.5, "eps": 1e-4, "dt": 1e-6, "prec": "kahan", "steps": 1, "group": 2, "dense": 16,
         "quad": 128},
        # the learned correction in the step: looser angle, corrected up to the tighter one
        {"name": "learned_262k", "kind": "learned", "n": 262144, "grid": 128, "layout": "cluster", "theta": 0.8,
         "theta_lo": 0.5, "eps": 1e-4, "dt": 1e-5},
        # the accuracy check against the FP64 direct sum
        {"name": "direct_1m", "kind": "direct", "n": 1048576, "grid": 256, "targets": 1000, "eps": 1e-4},
        # training the correction: one mini-batch at train()'s default size
        {"name": "train_64k", "kind": "train", "rows": 65536},
        # the network over the pairs of an evaluation set
        {"name": "infer_1m", "kind": "infer", "rows": 1000003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["round", "step", "step", "step", "batch", "learned", "direct", "train", "infer"])
    if kind == "round":
        n = _log(rng, 500, 200000)
        generated = rng.random() < 0.5
        ppb = rng.choice([60, 250, 1000])
        grid = max(1, min(24, int(math.ceil(math.sqrt(n / (0.7 * ppb))))))
        return {"kind": kind, "n": n, "grid": grid, "layout": "generated" if generated else "uniform",
                "rounds": rng.choice([1, 2]), "cutoff": 0.0 if generated else 1e-5,
                "dt": 5e-3 if generated else 1e-4}
    if kind == "step":
        prec = rng.choice(["kahan", "kahan", "kahan", "fp32", "fp64"])
        n = _log(rng, 1000, 65536 if prec == "fp64" else 4000000)
        per_box = rng.uniform(12.0, 80.0)
        tuned = rng.random() < 0.5
        steps = rng.choice([1, 2, 10]) if n < 100000 and prec != "fp64" else 1
        return {"kind": kind, "n": n, "grid": max(2, min(512, int(round(math.sqrt(n / per_box))))),
                "layout": rng.choice(["uniform", "gauss", "cluster"]), "theta": rng.choice([0.5, 0.6, 0.7, 0.8]),
                "eps": rng.choice([1e-3, 1e-4]), "dt": 1e-5, "prec": prec, "steps": steps,
                "graph": rng.random() < 0.5, "order": rng.choice(["file", "sorted"]),
                "group": rng.choice([1, 2, 4]) if tuned else 0, "dense": rng.choice([16, 32, 64]) if tuned else 0,
                "quad": rng.choice([-1, 128]) if tuned else 0}
    if kind == "batch":
        return {"kind": kind, "systems": _log(rng, 4, 384), "spread": rng.randrange(1000), "nmin": 1024, "nmax": rng.choice([8192, 65536, 131072]),
                "per_box": 64, "theta": 0.5, "eps": 1e-4, "dt": 1e-6, "prec": "kahan", "steps": 1,
                "group": rng.choice([0, 2]), "dense": 16, "quad": 128}
    if kind == "learned":
        n = _log(rng, 4096, 262144)
        return {"kind": kind, "n": n, "grid": max(4, int(round(math.sqrt(n / 16.0)))), "layout": "cluster",
                "theta": rng.choice([0.6, 0.7, 0.8]), "theta_lo": 0.5, "eps": 1e-4, "dt": 1e-5}
    if kind == "direct":
        n = _log(rng, 2000, 1048576)
        return {"kind": kind, "n": n, "grid": max(2, int(round(math.sqrt(n / 16.0)))),
                "targets": min(n, _log(rng, 10, min(16384, max(20, 1048576000 // n)))), "eps": rng.choice([0.0, 1e-4])}
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 2000, 65536)}
    return {"kind": kind, "rows": _log(rng, 1000, 1000000)}


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _particles(layout, n, g, clusters=8):
    """(x, y, m, vx, vy) FP64 on the device, in the order of a fresh file."""
    zero = torch.zeros(n, dtype=torch.float64, device=DEV)
    if layout == "generated":  # the reference's generator: [0, 499)^2, v in (-1, 1), m in [0.5, 5)
        return (499.0 * _rand(g, n), 499.0 * _rand(g, n), 0.5 + 4.5 * _rand(g, n),
                2.0 * _rand(g, n) - 1.0, 2.0 * _rand(g, n) - 1.0)
    m = 1.0 + _rand(g, n)
    if layout == "uniform":
        return _rand(g, n), _rand(g, n), m, zero, zero.clone()
    normal = torch.randn(2, n, generator=g, device=DEV, dtype=torch.float64)
    if layout == "gauss":
        p = 0.5 + normal / 12.0
    else:  # clusters with a uniform background
        centre = 0.2 + 0.6 * _rand(g, 2, clusters)
        which = torch.randint(0, clusters, (n,), generator=g, device=DEV)
        p = centre[:, which] + 0.05 * normal
        back = _rand(g, n) < 0.2
        p = torch.where(back, _rand(g, 2, n), p)
    p = p.clamp(0.0, 1.0 - 2.0 ** -24)
    return p[0].contiguous(), p[1].contiguous(), m, zero, zero.clone()


def _square(x, y):
    """Origin and edge of the reference's square bounding box."""
    x0, y0 = float(x.min()), float(y.min())
    return x0, y0, max(float(x.max()) - x0, float(y.max()) - y0)


def _sorted(state, grid):
    """In the order a running simulation's particles have: by box, within a box by quadrant."""
    x, y = state[0], state[1]
    x0, y0, edge = _square(x, y)
    h = edge / grid / 2.0
    kx = ((x - x0) / h).floor().clamp(0, 2 * grid - 1).long()
    ky = ((y - y0) / h).floor().clamp(0, 2 * grid - 1).long()
    key = ((kx >> 1) * grid + (ky >> 1)) * 4 + (kx & 1) * 2 + (ky & 1)
    at = torch.sort(key, stable=True).indices
    return tuple(a[at].contiguous() for a in state)


def _sizes(case):
    """Particles and boxes per side of each system: the plan's shape, part of the case."""
    r = np.random.default_rng([case["spread"], 17])
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    n = np.rint(np.exp(r.uniform(lo, hi, case["systems"]))).astype(np.int64)
    return [int(v) for v in n], [max(1, int(round(math.sqrt(v / case["per_box"])))) for v in n]


def _batch(case, seed):
    n, grids = _sizes(case)
    g = _gen(seed, 3)
    uniform = np.random.default_rng([int(seed), 18]).random(len(n)) < 0.5
    parts = [_particles("uniform" if uniform[k] else "cluster", v, g, clusters=4) for k, v in enumerate(n)]
    return n, grids, tuple(torch.cat([p[c] for p in parts]) for c in range(5))


def _weights(seed):
    """Flat FP32 parameters as after some training: input weights of the features' scale, a small output."""
    r = np.random.default_rng([int(seed), 5])
    p = np.zeros(10448, dtype=np.float32)

    def block(off, rows, cols, fan_in, used_rows, used_cols, scale=1.0):
        a = np.zeros((rows, cols))
        a[:used_rows, :used_cols] = r.uniform(-1, 1, (used_rows, used_cols)) * math.sqrt(3.0 / fan_in) * scale
        p[off:off + rows * cols] = a.reshape(-1)

    block(0, 16, 64, 6, 6, 64)
    block(1088, 64, 64, 64, 64, 64)
    block(5248, 64, 64, 64, 64, 64)
    block(9408, 64, 16, 64, 64, 2, 0.1)
    for off, k in ((1024, 64), (5184, 64), (9344, 64), (10432, 2)):
        p[off:off + k] = r.uniform(-0.1, 0.1, k)
    return p


def _rows(rows, g):
    """Feature rows of (target, cell) pairs and their targets: offsets of 1.3 to 3 cell edges, second
    moments of a filled cell; the target is the quadrupole term."""
    d = 1.3 + 1.7 * _rand(g, rows)
    phi = 2.0 * math.pi * _rand(g, rows)
    u, v = d * torch.cos(phi), d * torch.sin(phi)
    q = torch.stack([1.0 / 12.0 * (0.5 + _rand(g, rows)), 0.05 * (2.0 * _rand(g, rows) - 1.0),
                     1.0 / 12.0 * (0.5 + _rand(g, rows))])
    zero = torch.zeros_like(u)
    f = torch.stack([u, v, q[0], q[1], q[2], 1.0 / d, zero, zero], dim=1)
    c = torch.complex(q[0] - q[2], -2.0 * q[1]) / torch.complex(u, -v) ** 3
    return f.float().contiguous(), torch.stack([c.real, c.imag], dim=1).float().contiguous()


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _batch(case, seed)[2]
    if kind in ("train", "infer"):
        return _rows(case["rows"], _gen(seed, 4))
    state = _particles(case.get("layout", "cluster"), case["n"], _gen(seed))
    return _sorted(state, case["grid"]) if case.get("order") == "sorted" else state


def _targets(case, seed):
    return np.sort(np.random.default_rng([int(seed), 6]).choice(case["n"], case["targets"], replace=False))


def _network(seed):
    mlp = learned.LearnedCorrection(params=_weights(seed), device=DEV)
    # moments as they are after some hundred steps
    g = _gen(seed, 7)
    used = (mlp.params != 0).float()
    mlp.m = used * 1e-3 * torch.randn(10448, generator=g, device=DEV)
    mlp.v = used * 1e-6 * (0.5 + torch.rand(10448, generator=g, device=DEV))
    mlp.step_count = 500
    return mlp


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "inputs": _inputs(case, seed)}
    if kind in ("train", "infer"):
        state["mlp"] = _network(seed)
        return state
    if kind == "round":
        x, y, m, vx, vy = state["inputs"]
        rec = torch.zeros(case["n"], 10, dtype=torch.float64, device=DEV)
        for c, v in enumerate((x, y, m, vx, vy)):
            rec[:, c] = v
        rec[:, 9] = torch.arange(case["n"], device=DEV)
        state["records"] = rec
        prm = native.make_params(1.0, case["dt"], 0.0, case["cutoff"], 0.0, 0, native.BH_PREC_FP32_KAHAN)
        state["plan"] = native.Plan([case["n"]], [case["grid"]], prm, device=DEV)
    elif kind == "batch":
        n, grids = _sizes(case)
        prm = native.make_params(1.0, case["dt"], case["eps"], 0.0, case["theta"], case["group"],
                                 PREC[case["prec"]], dense_min=case["dense"], quad_min=case["quad"])
        state["plan"] = native.Plan(n, grids, prm, device=DEV)
    elif kind == "step":
        prm = native.make_params(1.0, case["dt"], case["eps"], 0.0, case["theta"], case["group"],
                                 PREC[case["prec"]], dense_min=case["dense"], quad_min=case["quad"])
        state["plan"] = native.Plan([case["n"]], [case["grid"]], prm, device=DEV)
    elif kind == "learned":
        prm = native.make_params(1.0, case["dt"], case["eps"], 0.0, case["theta"], 0, native.BH_PREC_FP32_KAHAN,
                                 native.BH_FLAG_LEARNED, correction_theta=case["theta_lo"])
        state["plan"] = native.Plan([case["n"]], [case["grid"]], prm, device=DEV)
        state["mlp"] = learned.LearnedCorrection(params=_weights(seed), device=DEV)
        state["plan"].set_correction(state["mlp"])
    else:  # direct
        prm = native.make_params(1.0, 1e-5, case["eps"], 0.0, 0.5, 0, native.BH_PREC_FP32_KAHAN)
        state["plan"] = native.Plan([case["n"]], [case["grid"]], prm, device=DEV)
        state["plan"].load(*state["inputs"])
        state["targets"] = _targets(case, seed)
    return state


# -------------------------------------------------------------------------------------------- a pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        mlp = state["mlp"]
        loss = mlp.grad_batch(*state["inputs"])
        mlp.adam_step(2e-3)
        return {"loss": loss, "params": mlp.params, "m": mlp.m, "v": mlp.v}
    if kind == "infer":
        return state["mlp"].forward(state["inputs"][0])
    plan = state["plan"]
    if kind == "direct":
        return plan.direct_sample(state["targets"])
    if kind == "round":
        plan.load_records(state["records"])
        for _ in range(case["rounds"]):
            plan.create_tree()
            plan.summarize()
            plan.evaluate()
            plan.timestep()
        names = ("px", "py", "mass", "vx", "vy", "ax", "ay", "gx", "gy", "pid")
        return dict(zip(names, plan.store_records().unbind(1)))
    plan.load(*state["inputs"])
    if kind == "step" and not case["graph"]:
        plan.step(case["steps"])
    else:
        plan.step_graph(case.get("steps", 1))
    return plan.store()


# -------------------------------------------------------------------------------------------- work
_CROWD = {"uniform": 1.0, "generated": 1.0, "gauss": 2.5, "cluster": 3.5}  # mean occupancy a particle sees / mean


def work(case):
    """Input and output bytes once; 12 operations per particle pair and 20 per particle-cell pair of the
    method (counts estimated from the opening angle and the layout)."""
    kind = case["kind"]
    if kind == "train":
        r = case["rows"]
        return {"bytes": r * (24 + 8) + 8 * 4 * 10448, "flops": r * 3 * 2 * (6 * 64 + 2 * 64 * 64 + 64 * 2)}
    if kind == "infer":
        r = case["rows"]
        return {"bytes": r * (24 + 8) + 4 * 10448, "flops": r * 2 * (6 * 64 + 2 * 64 * 64 + 64 * 2)}
    if kind == "direct":
        return {"bytes": 24 * case["n"] + 24 * case["targets"], "flops": 12.0 * case["n"] * case["targets"]}
    if kind == "round":
        n, g = case["n"], case["grid"]
        near = n / (g * g) * min(9, g * g)
        far = max(0, g * g - 9)
        return {"bytes": 160 * n, "flops": case["rounds"] * n * (12.0 * near + 20.0 * far)}
    if kind == "batch":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        n = int(case["systems"] * (case["nmax"] - case["nmin"]) / (hi - lo))
        per, crowd, boxes = case["per_box"], 2.2, case["nmax"] / case["per_box"]
    else:
        n = case["n"]
        per, crowd, boxes = n / case["grid"] ** 2, _CROWD[case["layout"]], case["grid"] ** 2
    reach = (1.0 + 2.0 / case["theta"]) ** 2
    near = min(n, per * crowd * min(reach, boxes))
    far = 3.0 * reach * max(0.0, math.log(max(1.0, boxes / reach), 4.0))
    flops = case.get("steps", 1) * n * (12.0 * near + 20.0 * far)
    if kind == "learned":  # the band between the two angles, about a third of the far cells, 17,152 each
        flops += n * far / 3.0 * 17152.0
    return {"bytes": 88 * n, "flops": flops}


# ------------------------------------------------------------------------------------------- exact
def _direct(x, y, m, eps2, at=None, pairs=1 << 27):
    """FP64 direct-sum accelerations of the particles `at` (all of them by default)."""
    n = x.numel()
    at = torch.arange(n, device=x.device) if at is None else at
    ax, ay = torch.empty(at.numel(), dtype=x.dtype, device=x.device), torch.empty(at.numel(), dtype=x.dtype, device=x.device)
    block = max(1, pairs // n)
    for s in range(0, at.numel(), block):
        t = at[s:s + block]
        dx, dy = x[None, :] - x[t, None], y[None, :] - y[t, None]
        r2 = dx * dx + dy * dy + eps2
        w = m[None, :] / r2
        w[torch.arange(t.numel(), device=x.device), t] = 0.0
        ax[s:s + block], ay[s:s + block] = (w * dx).sum(1), (w * dy).sum(1)
    return ax, ay


def _flat_round(x, y, m, grid, cutoff):
    """Accelerations of the reference's algorithm and the particles' boxes: the neighbourhood's
    particles, and the centre of mass of every other box."""
    x0, y0, edge = _square(x, y)
    step = edge / grid
    kx = ((x - x0) / step).floor().clamp(0, grid - 1).long()
    ky = ((y - y0) / step).floor().clamp(0, grid - 1).long()
    key = kx * grid + ky
    B = grid * grid
    M = torch.zeros(B, dtype=x.dtype, device=x.device).index_add_(0, key, m)
    cx = torch.zeros_like(M).index_add_(0, key, m * x) / M.clamp(min=1e-300)
    cy = torch.zeros_like(M).index_add_(0, key, m * y) / M.clamp(min=1e-300)
    bx, by = torch.arange(B, device=x.device) // grid, torch.arange(B, device=x.device) % grid
    ax, ay = torch.zeros_like(x), torch.zeros_like(x)
    members = [torch.nonzero(key == b).flatten() for b in range(B)]
    for b in range(B):
        t = members[b]
        if not t.numel():
            continue
        near = ((bx - b // grid).abs() <= 1) & ((by - b % grid).abs() <= 1)
        src = torch.cat([members[k] for k in torch.nonzero(near).flatten().tolist()])
        far = torch.nonzero(~near & (M > 0)).flatten()
        for sx, sy, sm in ((x[src], y[src], m[src]), (cx[far], cy[far], M[far])):
            dx, dy = sx[None, :] - x[t, None], sy[None, :] - y[t, None]
            r2 = dx * dx + dy * dy
            w = torch.where(r2 > cutoff, sm[None, :] / r2, torch.zeros_like(r2))
            ax[t] += (w * dx).sum(1)
            ay[t] += (w * dy).sum(1)
    return ax, ay, kx, ky


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _mlp64(p, f):
    h = f[:, :6].double()
    for off, rows, cols, used, boff in ((0, 16, 64, 6, 1024), (1088, 64, 64, 64, 5184), (5248, 64, 64, 64, 9344)):
        h = _gelu(h @ p[off:off + rows * cols].view(rows, cols)[:used] + p[boff:boff + cols])
    return h @ p[9408:10432].view(64, 16)[:, :2] + p[10432:10434]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "infer"):
        p0 = torch.tensor(_weights(seed), device=DEV).double()
        f, t = _inputs(case, seed)
        if kind == "infer":
            return _mlp64(p0, f)
        mlp = _network(seed)
        p = p0.clone().requires_grad_(True)
        err = _mlp64(p, f) - t.double()
        loss = (err * err).sum()
        (g,) = torch.autograd.grad((err * err).mean(), p)
        m, v, k = 0.9 * mlp.m.double() + 0.1 * g, 0.999 * mlp.v.double() + 0.001 * g * g, mlp.step_count + 1
        new = p0 - 2e-3 * (m / (1.0 - 0.9 ** k)) / ((v / (1.0 - 0.999 ** k)).sqrt() + 1e-8)
        return {"loss": loss.reshape(1), "params": new, "m": m, "v": v}
    if kind == "direct":
        x, y, m = _inputs(case, seed)[:3]
        return _direct(x, y, m, case["eps"] ** 2, torch.tensor(_targets(case, seed), device=DEV))
    if kind == "round":
        if case["n"] > 250000 or case["grid"] > 32:
            return None
        x, y, m, vx, vy = _inputs(case, seed)
        for _ in range(case["rounds"]):
            ax, ay, kx, ky = _flat_round(x, y, m, case["grid"], case["cutoff"])
            vx, vy = vx + ax * case["dt"], vy + ay * case["dt"]
            x, y = x + vx * case["dt"], y + vy * case["dt"]
        zero = torch.zeros_like(x)
        return {"px": x, "py": y, "mass": m, "vx": vx, "vy": vy, "ax": zero, "ay": zero, "gx": kx.double(),
                "gy": ky.double(), "pid": torch.arange(case["n"], device=DEV).double()}
    if kind == "step" and case["n"] * case["n"] * case["steps"] <= 2 ** 35:
        # the method approximates the direct sum
        x, y, m, vx, vy = _inputs(case, seed)
        for _ in range(case["steps"]):
            ax, ay = _direct(x, y, m, case["eps"] ** 2)
            vx, vy = vx + ax * case["dt"], vy + ay * case["dt"]
            x, y = x + vx * case["dt"], y + vy * case["dt"]
        return {"x": x, "y": y, "vx": vx, "vy": vy, "ax": ax, "ay": ay}
    return None
