"""What this framework is timed on: the calls its users make, over the range of
sizes, precisions and options they make them with.

Every pass goes through the public Python interface (`create_engine`,
`create_solver`, `Ensemble`, `statistics`, `learn_loss_grad`).  FP64 engines
are timed on their force evaluation, whose result is the output; mixed-precision
engines on whole solver steps, whose result is the FP64 state a user reads.
"""
import math
import random

import numpy as np
import torch

from nbody_gb300.data import NBodyData
from nbody_gb300.engine import create_engine
from nbody_gb300.ensemble import Ensemble
from nbody_gb300.solvers import create_solver

SOFTENING = 1e-3  # of every mixed-precision configuration
DT = 1e-3


def listed():
    return [
        # the default engine on the size the reference's own parity run has:
        # the smallest force evaluation, bound by latency and idle SMs
        {"name": "direct_fp64_1024", "kind": "direct_fp64", "n": 1024, "input": "cube"},
        # the default engine on a ragged size an hour-long FP64 run would have
        {"name": "direct_fp64_20011", "kind": "direct_fp64", "n": 20011, "input": "plummer"},
        # a small cluster with unequal masses and an embedded error estimate
        # every step (7 force evaluations, buffer algebra, one readback)
        {"name": "direct_mixed_rkdp_5003", "kind": "direct_mixed", "n": 5003, "input": "cube",
         "solver": "rkdp"},
        # the headline direct-sum configuration
        {"name": "direct_mixed_rk4_131072", "kind": "direct_mixed", "n": 131072,
         "input": "plummer", "solver": "rk4"},
        # Barnes-Hut of a small system: many launches, few groups to walk
        {"name": "bh_mixed_rk4_16384", "kind": "bh_mixed", "log2n": 14, "ratio": 2.0, "order": 1,
         "solver": "rk4"},
        # the Barnes-Hut headline size, one step as the reference's bench takes it
        {"name": "bh_mixed_euler_1048576", "kind": "bh_mixed", "log2n": 20, "ratio": 2.0,
         "order": 1, "solver": "euler"},
        # quadrupole cells at the opening ratio of the 1e-4 error target
        {"name": "bh_quadrupole_euler_131072", "kind": "bh_mixed", "log2n": 17, "ratio": 4.0,
         "order": 2, "solver": "euler"},
        # the reference's own Barnes-Hut arithmetic and tree
        {"name": "bh_fp64_32768", "kind": "bh_fp64", "log2n": 15, "ratio": 2.0},
        # the learned correction at the loose opening ratio
        {"name": "bh_learned_euler_131072", "kind": "learned", "log2n": 17, "ratio": 1.1111},
        # gradients of the correction's network for one training batch
        {"name": "learn_gradient_16384", "kind": "gradient", "samples": 16384},
        # a batch of clusters of uneven size, a few adaptive steps between two
        # reads of the state
        {"name": "ensemble_512", "kind": "ensemble", "systems": 512, "steps": 4},
        # the conservation sums of a long run's check
        {"name": "statistics_50000", "kind": "statistics", "n": 50000, "softening": SOFTENING},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["direct_fp64", "direct_fp64", "direct_mixed", "direct_mixed", "bh_mixed",
                       "bh_mixed", "bh_fp64", "learned", "gradient", "ensemble", "statistics"])
    if kind == "direct_fp64":
        return {"kind": kind, "n": _log_uniform(rng, 128, 20011),
                "input": rng.choice(["cube", "plummer"])}
    if kind == "direct_mixed":
        return {"kind": kind, "n": _log_uniform(rng, 500, 120000),
                "input": rng.choice(["cube", "plummer"]),
                "solver": rng.choice(["euler", "rk4", "rkdp"]) if rng.random() < 0.5 else "rk4"}
    if kind == "bh_mixed":
        order = rng.choice([1, 1, 2])
        return {"kind": kind, "log2n": rng.randint(10, 20 if order == 1 else 17),
                "ratio": round(rng.uniform(1.1, 2.5) if order == 1 else rng.uniform(1.3, 4.0), 3),
                "order": order, "solver": rng.choice(["euler", "rk4"])}
    if kind == "bh_fp64":
        return {"kind": kind, "log2n": rng.randint(9, 15), "ratio": round(rng.uniform(1.1, 2.0), 3)}
    if kind == "learned":
        return {"kind": kind, "log2n": rng.randint(14, 17), "ratio": round(rng.uniform(1.0, 1.3), 3)}
    if kind == "gradient":
        return {"kind": kind, "samples": _log_uniform(rng, 1000, 100000)}
    if kind == "ensemble":
        return {"kind": kind, "systems": _log_uniform(rng, 16, 512), "steps": rng.randint(1, 4)}
    return {"kind": kind, "n": _log_uniform(rng, 1000, 50000),
            "softening": rng.choice([0.0, SOFTENING])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _bodies(case, seed):
    n = case["n"] if "n" in case else 1 << case["log2n"]
    if case.get("input", "plummer") == "cube":
        return NBodyData.uniform_cube(n, side=2.0, seed=seed)
    return NBodyData.plummer(n, seed=seed)


def _clusters(case, seed):
    sizes = np.random.default_rng(case["systems"]).integers(64, 4097, size=case["systems"])
    return [NBodyData.plummer(int(k), seed=seed * 100003 + i) for i, k in enumerate(sizes)]


def _batch(case, seed):
    """Features and targets as the engine's samples have them: an offset of
    1.1 to 2 cell radii, second moments, half extents, 1/|u|, centre offset."""
    rng = np.random.default_rng(seed)
    b = case["samples"]
    u = rng.normal(size=(b, 3))
    u *= (rng.uniform(1.1, 2.0, size=(b, 1)) / np.linalg.norm(u, axis=1, keepdims=True))
    h = rng.uniform(0.1, 0.6, size=(b, 3))
    q = np.concatenate([h * h / 3, 0.02 * rng.normal(size=(b, 3))], axis=1)
    o = 0.1 * rng.normal(size=(b, 3))
    x = np.concatenate([u, q, h, 1.0 / np.linalg.norm(u, axis=1, keepdims=True), o], axis=1)
    t = np.concatenate([0.1 * rng.normal(size=(b, 3)), rng.uniform(0.5, 2.0, size=(b, 1))], axis=1)
    return x.astype(np.float32), t.astype(np.float32)


def _weights(seed):
    rng = np.random.default_rng(seed + 7)
    parts = []
    for i, o in ((16, 64), (64, 64), (64, 3)):
        a = math.sqrt(6.0 / (i + o))
        parts += [rng.uniform(-a, a, size=i * o), rng.uniform(-0.1, 0.1, size=o)]
    return np.concatenate(parts).astype(np.float32)


class _DeviceArray:
    def __init__(self, mem):
        self.mem = mem  # keeps the buffer and its engine alive
        self.__cuda_array_interface__ = {"shape": (mem.size() // 8,), "typestr": "<f8",
                                         "data": (mem.device_ptr(), False), "version": 3}


def _view(mem):
    """An engine buffer as a torch tensor, without a copy."""
    return torch.as_tensor(_DeviceArray(mem), device="cuda")


def _engine(case):
    p = {"engine": "gb300", "precision": "mixed", "softening": SOFTENING}
    kind = case["kind"]
    if kind in ("direct_fp64", "bh_fp64"):
        p = {"engine": "gb300"}
    if kind == "statistics":
        p["softening"] = case["softening"]
    if kind in ("bh_fp64", "bh_mixed", "learned"):
        p.update(algo="bh", distance_to_node_radius_ratio=case["ratio"])
    if kind == "learned":
        p.update(learned=True, learned_tight_ratio=2.0, learned_judge=False)
    e = create_engine(p)
    if e is None:
        raise RuntimeError("no engine")
    if case.get("order", 1) == 2:
        e.tune_set("bh.order", 2)
    return e


def _trained(data, ratio, seed):
    """A network trained for a moment on samples of the snapshot's own tree."""
    t = create_engine({"engine": "gb300", "algo": "bh", "precision": "mixed",
                       "softening": SOFTENING, "distance_to_node_radius_ratio": ratio,
                       "learned_tight_ratio": 2.0})
    t.init(data)
    t.learn_generate(200000, seed=seed + 1)
    t.learn_train(4, batch=8192, lr=3e-3, seed=seed + 2)
    w = t.learn_get_weights()
    t.close()
    return w


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        s = Ensemble(softening=SOFTENING, tolerance=1e-8, dt_initial=DT)
        s.init(_clusters(case, seed))
        return {"kind": kind, "ensemble": s, "steps": case["steps"]}
    e = _engine(case)
    if kind == "gradient":
        x, t = _batch(case, seed)
        e.learn_set_weights(_weights(seed))
        return {"kind": kind, "engine": e, "x": x, "t": t}
    data = _bodies(case, seed)
    if not e.init(data):
        raise RuntimeError("init failed")
    state = {"kind": kind, "engine": e, "data": data}
    if kind in ("direct_fp64", "bh_fp64"):
        state["y"], state["f"] = e.get_y(), e.create_buffer(8 * e.problem_size())
        state["out"] = _view(state["f"])
    elif kind != "statistics":
        if kind == "learned":
            e.learn_set_weights(_trained(data, case["ratio"], seed))
        # threshold above any step's error: no step is subdivided
        s = create_solver({"solver": case.get("solver", "euler"), "error_threshold": 1e9,
                           "max_step": DT})
        s.set_engine(e)
        state["solver"], state["out"] = s, _view(e.get_y())
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        s = state["ensemble"]
        s.step(state["steps"])
        return list(s.get_state())
    e = state["engine"]
    if kind == "gradient":
        loss, grad = e.learn_loss_grad(state["x"], state["t"])
        return {"loss": loss, "grad": grad}
    if kind == "statistics":
        return e.statistics()
    if kind in ("direct_fp64", "bh_fp64"):
        e.fcompute(e.get_time(), state["y"], state["f"])
        return state["out"]
    state["solver"].advise(DT)
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
STAGES = {"euler": 1, "rk4": 4, "rkdp": 7}
PAIR_FLOPS = 26  # of one unordered pair, both bodies: d, r^2, r^-3, two weighted sums
CELL_FLOPS = {1: 20, 2: 50}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        # the sizes are uniform in 64 .. 4096
        pairs = case["systems"] * (4096.0 ** 3 - 64.0 ** 3) / 3 / 4032 / 2
        return {"bytes": case["systems"] * 2080 * 8 * 13.0,
                "flops": 7 * case["steps"] * PAIR_FLOPS * pairs}
    if kind == "gradient":
        b = case["samples"]
        return {"bytes": 80.0 * b, "flops": 6.0 * b * (16 * 64 + 64 * 64 + 64 * 3)}
    n = case["n"] if "n" in case else 1 << case["log2n"]
    if kind == "statistics":
        return {"bytes": 56.0 * n, "flops": 10.0 * n * n / 2}
    if kind == "direct_fp64":
        return {"bytes": 8.0 * 13 * n, "flops": PAIR_FLOPS * n * n / 2.0}
    if kind == "direct_mixed":
        k = STAGES[case["solver"]]
        return {"bytes": 8.0 * 13 * n, "flops": k * PAIR_FLOPS * n * n / 2.0}
    # cells per body grow with the ratio squared and the depth of the tree
    ratio = case["ratio"]
    cells = min(float(n), (400.0 if kind == "bh_fp64" else 39.0) * ratio * ratio * math.log2(n))
    k = STAGES[case.get("solver", "euler")]
    flops = k * n * cells * CELL_FLOPS[case.get("order", 1)]
    if kind == "learned":
        flops += 400.0 * n * 2 * (16 * 64 + 64 * 64 + 64 * 3)
    return {"bytes": 8.0 * 13 * n, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, without the framework
# ---------------------------------------------------------------------------
def _accelerations(pos, mass, eps2):
    """pos [n, 3]; chunks of rows against all bodies.  eps2 = 0: the pairs'
    r^2 is at least 1e-8."""
    n = pos.shape[0]
    acc = torch.empty_like(pos)
    rows = max(1, (1 << 26) // n)
    for i in range(0, n, rows):
        p = pos[i:i + rows]
        d = [pos[None, :, c] - p[:, c, None] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r2 = r2 + eps2 if eps2 > 0 else r2.clamp_(min=1e-8)
        w = mass / (r2 * r2.sqrt())
        for c in range(3):
            acc[i:i + rows, c] = (d[c] * w).sum(1)
    return acc


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tensors(data):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(_device())
            for a in (data.vertices, data.velocities, data.mass)]


TABLES = {
    "euler": ([[]], [1.0]),
    "rk4": ([[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6]),
    "rkdp": ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
              [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
              [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
              [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
             [5179 / 57600, 0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]),
}
RKDP_LOW = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0]


def _stages(solver, pos, vel, mass, eps2, dt):
    kp, kv = [], []
    for row in TABLES[solver][0]:
        p = pos + sum((dt * a * k for a, k in zip(row, kp) if a), torch.zeros_like(pos))
        v = vel + sum((dt * a * k for a, k in zip(row, kv) if a), torch.zeros_like(vel))
        kp.append(v)
        kv.append(_accelerations(p, mass, eps2))
    return kp, kv


def _combine(coeff, ks):
    return sum((b * k for b, k in zip(coeff, ks) if b), torch.zeros_like(ks[0]))


def _flat(a, b):
    return torch.cat([a.t().reshape(-1), b.t().reshape(-1)])


def _exact_ensemble(case, seed):
    out_p, out_v = [], []
    for d in _clusters(case, seed):
        pos, vel, mass = _tensors(d)
        dt, held = DT, False
        for _ in range(case["steps"]):
            kp, kv = _stages("rkdp", pos, vel, mass, SOFTENING ** 2, dt)
            diff = [h - lo for h, lo in zip(TABLES["rkdp"][1], RKDP_LOW)]
            err = dt * float(torch.maximum(_combine(diff, kp).abs().max(),
                                           _combine(diff, kv).abs().max()))
            ok = err <= 1e-8 or dt <= 1e-9
            if ok:
                pos = pos + dt * _combine(TABLES["rkdp"][1], kp)
                vel = vel + dt * _combine(TABLES["rkdp"][1], kv)
            grow = 0.9 * (1e-8 / err) ** 0.2 if err > 0 else 5.0
            # no growth in the step after a rejected one
            dt = min(0.1, max(1e-9, dt * min(1.0 if held else 5.0, max(0.2, grow))))
            held = not ok
        out_p.append(pos)
        out_v.append(vel)
    return [torch.cat(out_p), torch.cat(out_v)]


def _exact_gradient(case, seed):
    x, t = (torch.from_numpy(a).double() for a in _batch(case, seed))
    w = torch.from_numpy(_weights(seed)).double().requires_grad_()
    gelu = lambda z: 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
    a, at = x, 0
    for k, (i, o) in enumerate(((16, 64), (64, 64), (64, 3))):
        a = a @ w[at:at + i * o].reshape(i, o) + w[at + i * o:at + i * o + o]
        at += i * o + o
        a = gelu(a) if k < 2 else a
    uh = x[:, 0:3] * x[:, 12:13]
    xx, yy, zz, xy, xz, yz = (x[:, k:k + 1] for k in range(3, 9))
    ux, uy, uz = uh[:, 0:1], uh[:, 1:2], uh[:, 2:3]
    qu = torch.cat([xx * ux + xy * uy + xz * uz, xy * ux + yy * uy + yz * uz,
                    xz * ux + yz * uy + zz * uz], 1)
    g = a[:, 0:1] * uh + a[:, 1:2] * qu + a[:, 2:3] * x[:, 13:16]
    loss = ((g - t[:, 0:3]) ** 2).sum()
    (loss / x.shape[0]).backward()
    return {"loss": float(loss.detach()), "grad": w.grad}


def _exact_statistics(case, seed):
    pos, vel, m = _tensors(_bodies(case, seed))
    n, eps2, pe = pos.shape[0], case["softening"] ** 2, 0.0
    rows = max(1, (1 << 26) // n)
    for i in range(0, n, rows):
        p = pos[i:i + rows]
        r2 = sum((pos[None, :, c] - p[:, c, None]) ** 2 for c in range(3))
        inv = (r2 + eps2).rsqrt()
        if eps2 == 0:
            inv[r2 < 1e-8] = 0.0
        k = torch.arange(p.shape[0], device=p.device)
        inv[k, k + i] = 0.0
        pe -= float((m[i:i + rows, None] * m * inv).sum()) / 2
    mv = vel * m[:, None]
    com = (pos * m[:, None]).sum(0) / m.sum()
    return torch.tensor(mv.sum(0).tolist() + torch.linalg.cross(pos, mv).sum(0).tolist()
                        + [float((mv * vel).sum()) / 2, pe] + com.tolist() + [float(m.sum())],
                        dtype=torch.float64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "statistics":
        return _exact_statistics(case, seed)
    if case.get("log2n", 0) > 17:
        return None  # a direct sum of that size takes minutes
    pos, vel, mass = _tensors(_bodies(case, seed))
    if kind in ("direct_fp64", "bh_fp64"):
        return _flat(vel, _accelerations(pos, mass, 0.0))
    # Barnes-Hut, plain or corrected, stands for the direct sum
    solver = case.get("solver", "euler")
    kp, kv = _stages(solver, pos, vel, mass, SOFTENING ** 2, DT)
    b = TABLES[solver][1]
    return _flat(pos + DT * _combine(b, kp), vel + DT * _combine(b, kv))
