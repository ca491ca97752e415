"""Performance cases of the FARRSIGHT hot path: field evaluations, sessions and
batches through the package's public entry points.

Every case is a dict of plain values; `prepare` makes what a user's program
holds before the call, `run` is one pass, `work` what a pass cannot do without
and `exact` the FP64 result of the same inputs in plain torch.

Inputs are electrons of a nonlinear wave (density perturbations of tens of
percent, fields of order one: the trapping stage that such runs spend most of
their time in), on phase-space lattices of the sizes of the configurations or
on a ragged number of points as adaptive meshes have it.  Positions are not
wrapped into the period, as in a run.
"""
import math

import numpy as np
import torch

import multi_species_b200 as fs
from multi_species_b200 import decks

# (period, regularisation, largest speed) of the configurations: Landau
# damping, two-stream, bump-on-tail
BOXES = {"landau": (4 * math.pi, 0.05, 6.0), "two_stream": (10 * math.pi, 0.02, 8.0),
         "bump": (20 * math.pi, 0.02, 10.0)}
# Sessions step without remesh (a run of thousands of steps on these coarse
# meshes would not keep its positions remeshable); the remesh is a case of its own.
NO_REMESH = 1 << 30
# the treecode configuration: opening angle, degree, leaf size
TREE = (0.7, 8, 2000)


def listed():
    return [
        # One small self-field without allocation: a host that owns the device
        # memory calls it once per stage of a small run.  Latency.
        {"name": "noalloc_small", "kind": "noalloc", "box": "landau", "n": 2145},
        # The two-species Landau configuration's field in the reference
        # arithmetic (the default backend of a deck), 65 x 129 points twice.
        {"name": "field64_landau", "kind": "field", "box": "landau", "precision": "fp64", "n": 16770, "nt": 0},
        # Field of a two-stream state at a ragged set of other positions
        # (probes, a second species' points), reference arithmetic.
        {"name": "field64_targets", "kind": "field", "box": "two_stream", "precision": "fp64", "n": 65537,
         "nt": 33333},
        # The precision form's field at the two-stream configuration's size.
        {"name": "field32_two_stream", "kind": "field", "box": "two_stream", "precision": "fp32c", "n": 525825,
         "nt": 0},
        # The drop-in operator call with host arrays, as the reference's C++
        # program makes it, at an odd medium size.
        {"name": "field32_host", "kind": "host", "box": "two_stream", "precision": "fp32c", "n": 99991},
        # The treecode configuration's field: 3 x 1025 x 2049 points.
        {"name": "tree32_bump", "kind": "tree", "box": "bump", "precision": "fp32c", "n": 6300675},
        # The default backend of a deck with use_treecode, medium size.
        {"name": "tree64_bump", "kind": "tree", "box": "bump", "precision": "fp64", "n": 395523},
        # A served bump-on-tail request of median size: treecode steps.
        {"name": "sim_tree32", "kind": "sim", "deck": "bump", "backend": "treecode32c", "h": 6, "ph": 1, "steps": 2},
        # The two-species Landau configuration in the reference arithmetic: the
        # steps between two remeshes, and the state for the caller's diagnostics.
        {"name": "sim64_landau", "kind": "sim", "deck": "landau", "backend": "direct64", "h": 5, "ph": 1,
         "steps": 4},
        # The two-stream configuration, the steps between two remeshes.
        {"name": "sim32_two_stream", "kind": "sim", "deck": "two_stream", "backend": "direct32c", "h": 8, "ph": 1,
         "steps": 4},
        # Uneven Landau instances of one to three species stepped together.
        {"name": "batch_landau", "kind": "batch", "count": 12, "mix": 1, "steps": 2},
        # The remesh of a caller's positions at the two-stream configuration's
        # size: moved points in, the state on the fresh mesh out.
        {"name": "remesh_two_stream", "kind": "remesh", "deck": "two_stream", "backend": "direct64", "h": 8, "ph": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("noalloc", "field64", "field32", "field32", "host", "tree32", "tree64", "sim32", "sim64",
                       "batch", "remesh"))
    if kind == "noalloc":
        return {"kind": "noalloc", "box": rng.choice(("landau", "two_stream")), "n": _log(rng, 600, 32768)}
    if kind == "field64":
        n = _log(rng, 2000, 66000)
        nt = 0 if rng.random() < 0.5 else _log(rng, 500, 66000)
        return {"kind": "field", "box": rng.choice(("landau", "two_stream")), "precision": "fp64", "n": n, "nt": nt}
    if kind == "field32":
        n = _log(rng, 2000, 525000)
        nt = 0 if rng.random() < 0.7 else _log(rng, 500, 200000)
        return {"kind": "field", "box": rng.choice(tuple(BOXES)), "precision": "fp32c", "n": n, "nt": nt}
    if kind == "host":
        return {"kind": "host", "box": rng.choice(("landau", "two_stream")), "precision": "fp32c",
                "n": _log(rng, 2000, 300000)}
    if kind == "tree32":
        return {"kind": "tree", "box": "bump", "precision": "fp32c", "n": _log(rng, 100000, 6300000)}
    if kind == "tree64":
        return {"kind": "tree", "box": "bump", "precision": "fp64", "n": _log(rng, 10000, 400000)}
    if kind == "sim32":
        return {"kind": "sim", "deck": "two_stream", "backend": "direct32c", "h": rng.randint(5, 7),
                "ph": rng.randint(0, 2), "steps": rng.choice((1, 2, 4, 8))}
    if kind == "sim64":
        return {"kind": "sim", "deck": rng.choice(("landau", "two_stream")), "backend": "direct64",
                "h": rng.randint(4, 5), "ph": rng.randint(0, 2), "steps": rng.choice((1, 2, 4, 8))}
    if kind == "remesh":
        return {"kind": "remesh", "deck": rng.choice(("landau", "two_stream")), "backend": "direct64",
                "h": rng.randint(4, 8), "ph": rng.randint(0, 1)}
    return {"kind": "batch", "count": rng.randint(3, 12), "mix": rng.randint(2, 500), "steps": rng.choice((1, 2))}


# ---------------------------------------------------------------- inputs
def _electrons(case, seed, n, device):
    """x, q of n electrons of a nonlinear wave: positions and velocities on a
    rank-1 lattice of the box, moved along their orbits for a moment and
    displaced by the wave; weights from the velocity distribution.  FP64."""
    L, _, vmax = BOXES[case["box"]]
    g = torch.Generator().manual_seed(seed)
    u = torch.rand(6, generator=g, dtype=torch.float64)
    u = [float(v) for v in u]
    i = torch.arange(n, dtype=torch.float64, device=device)
    X = torch.remainder(i * 0.6180339887498949 + u[0], 1.0) * L
    v = vmax * (2.0 * torch.remainder((i + 0.5) / n + u[1], 1.0) - 1.0)
    if case["box"] == "landau":
        f = torch.exp(-0.5 * v * v)
    elif case["box"] == "two_stream":
        f = v * v * torch.exp(-0.5 * v * v)
    else:
        f = 0.9 * torch.exp(-0.5 * v * v) + 0.2 * torch.exp(-2.0 * (v - 4.5) ** 2)
    f = f / math.sqrt(2 * math.pi)
    k = 2 * math.pi / L
    q = -(2 * vmax * L / n) * f * (1.0 + (0.2 + 0.2 * u[2]) * torch.cos(k * X))
    x = X + v * (0.5 + u[3]) + (0.2 + 0.2 * u[4]) / k * torch.sin(k * X + 2 * math.pi * u[5])
    return x, q


def _targets(case, seed, device):
    L = BOXES[case["box"]][0]
    g = torch.Generator().manual_seed(seed + 7919)
    return (torch.rand(case["nt"], generator=g, dtype=torch.float64) * 1.2 * L - 0.1 * L).to(device)


def _deck(case, seed):
    g = torch.Generator().manual_seed(seed)
    a, b = (float(t) for t in torch.rand(2, generator=g, dtype=torch.float64))
    if case["deck"] == "two_stream":
        d = decks.two_stream(h=case["h"], ph=case["ph"])
    elif case["deck"] == "landau":
        d = decks.landau_two_species(h=case["h"], ph=case["ph"])
    else:
        d = decks.bump_on_tail(h=case["h"], ph=case["ph"])
    d["remesh_period"] = NO_REMESH
    for s in d["species_list"]:
        if s["m"] < 100:
            s["amp"] = 0.3 + 0.2 * a
            s["pth"] = s["pth"] * (0.95 + 0.1 * b)
    return d


def _batch_decks(case, seed):
    """The members' sizes, boxes and species are the case's; the waves the seed's."""
    g = torch.Generator().manual_seed(seed)
    ds = decks.landau_batch(count=case["count"], seed=case["mix"])
    for d in ds:
        d["remesh_period"] = NO_REMESH
        a = float(torch.rand(1, generator=g, dtype=torch.float64))
        for s in d["species_list"]:
            if s["m"] < 100:
                s["amp"] = 0.3 + 0.2 * a
    return ds


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sim":
        sim = fs.Simulation(_deck(case, seed), case["backend"])
        return {"kind": kind, "sim": sim, "steps": case["steps"]}
    if kind == "remesh":
        d = _deck(case, seed)
        sim = fs.Simulation(d, case["backend"])
        g = torch.Generator().manual_seed(seed + 104729)
        t, a = (float(u) for u in torch.rand(2, generator=g, dtype=torch.float64))
        st, k = sim.state(), 2 * math.pi / d["xmax"]
        # a moment of free motion and a kick by the wave
        xs = st["xs"] + (0.2 + 0.3 * t) * st["ps"]
        ps = st["ps"] + (0.1 + 0.2 * a) * np.sin(k * st["xs"])
        return {"kind": kind, "sim": sim, "xs": xs, "ps": ps}
    if kind == "batch":
        b = fs.Batch()
        ids = [b.add(d) for d in _batch_decks(case, seed)]
        return {"kind": kind, "batch": b, "ids": ids, "steps": case["steps"]}
    L, eps, _ = BOXES[case["box"]]
    if kind == "host":
        x, q = (a.numpy() for a in _electrons(case, seed, case["n"], "cpu"))
        return {"kind": kind, "field": fs.E_MQ_DirectSum_B200(L, eps, case["precision"]), "x": x, "q": q}
    x, q = _electrons(case, seed, case["n"], "cuda")
    s = {"kind": kind, "x": x, "q": q, "n": case["n"], "L": L, "eps": eps}
    if kind == "noalloc":
        s["t"], s["nt"] = x, case["n"]
    elif kind == "tree":
        s["field"] = fs.E_MQ_Treecode_B200(L, eps, *TREE, precision=case["precision"])
        s["t"], s["nt"] = x, case["n"]
    else:
        s["field"] = fs.E_MQ_DirectSum_B200(L, eps, case["precision"])
        s["t"], s["nt"] = (_targets(case, seed, "cuda"), case["nt"]) if case["nt"] else (x, case["n"])
    s["es"] = torch.zeros(s["nt"], dtype=torch.float64, device="cuda")
    s["stream"] = torch.cuda.Stream()
    torch.cuda.synchronize()  # the inputs are there before the caller's stream reads them
    return s


def run(s):
    kind = s["kind"]
    if kind == "sim":
        s["sim"].step(s["steps"])
        return s["sim"].state()
    if kind == "remesh":
        s["sim"].import_xp(s["xs"], s["ps"])
        s["sim"].remesh()
        return s["sim"].state()
    if kind == "batch":
        s["batch"].step(s["steps"])
        return [s["batch"].state(i) for i in s["ids"]]
    if kind == "host":
        return s["field"].evaluate(s["x"], s["x"], s["q"])
    es, t, x, q = (s[k].data_ptr() for k in ("es", "t", "x", "q"))
    if kind == "noalloc":
        fs.field_eval_noalloc(s["L"], s["eps"], es, x, q, s["n"], s["stream"].cuda_stream)
    else:
        s["field"].evaluate_device(es, t, s["nt"], x, q, s["n"], s["stream"].cuda_stream)
    return s["es"]


# ---------------------------------------------------------------- what a pass needs
# FP64 operations of one pair in the reference's arithmetic and order (a
# division, a rounding, a square root and a reciprocal, each one operation)
PAIR64 = 17


def _points(case):
    if case["kind"] == "batch":
        ds = _batch_decks(case, 0)
    else:
        ds = [_deck(case, 0)]
    return [decks.deck_points(d) for d in ds]


def work(case):
    kind = case["kind"]
    if kind in ("sim", "batch"):
        # per step: the state once in and once out, and what the field needs
        ns, steps = _points(case), case["steps"]
        n = sum(ns)
        flops = 30.0 * n
        if case.get("backend") == "direct64":
            flops += 4.0 * PAIR64 * sum(m * m for m in ns)
        return {"bytes": steps * 2 * 40.0 * n, "flops": steps * flops}
    if kind == "remesh":
        # positions in, state out; per point an interpolation, per leaf a 9 x 9 solve
        n = sum(_points(case))
        return {"bytes": 80.0 * n, "flops": 40.0 * n + 600.0 * n / 4}
    n, nt = case["n"], case.get("nt") or case["n"]
    if case.get("precision") == "fp64" and kind != "tree":
        return {"bytes": 16.0 * n + 16.0 * nt, "flops": float(PAIR64) * n * nt}
    # a smooth kernel's sum needs each input and each output once
    return {"bytes": 16.0 * n + 8.0 * nt + (8.0 * nt if nt != n else 0.0), "flops": 60.0 * (n + nt)}


# ---------------------------------------------------------------- 64 bits
def _direct(t, x, q, L, eps):
    """E at t: sum_j -q_j z L (1/sqrt(L^2 + 4 eps^2) - 1/sqrt(4 z^2 L^2 + 4 eps^2)),
    z = (t - x_j)/L less its nearest integer."""
    c = 1 / math.sqrt(L * L + 4 * eps * eps)
    out = torch.empty_like(t)
    step = max(1, (1 << 28) // max(1, x.numel()))
    for a in range(0, t.numel(), step):
        z = (t[a:a + step, None] - x[None, :]).div_(L)
        z.sub_(torch.round(z))
        z.mul_(L)
        w = (z * z).mul_(4).add_(4 * eps * eps).rsqrt_().neg_().add_(c).mul_(z)
        out[a:a + step] = -(w @ q)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sim", "batch", "remesh") or case["n"] > 600000:
        return None
    L, eps, _ = BOXES[case["box"]]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "host":
        x, q = (a.to(device) for a in _electrons(case, seed, case["n"], "cpu"))
        return _direct(x, x, q, L, eps).cpu().numpy()
    x, q = _electrons(case, seed, case["n"], device)
    t = _targets(case, seed, device) if case.get("nt") else x
    return _direct(t, x, q, L, eps)
