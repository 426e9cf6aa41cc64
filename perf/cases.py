"""The work a user of the engine has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (robotfd_b200) on seeded synthetic
curves of the generator the tests and the benchmark use: "walk" curves (a random walk and a
noisy arc-length resampling of it) and "spline" curves (a Catmull-Rom path through random
waypoints and a time-warped noisy copy).  Sizes are those of the workloads the benchmark and
the tests name (2,000 x 1,900 points in 2D, 200,000 x 200,000 in 3D, uneven batches with
lognormal lengths around 2,000 clipped to [100, 50,000]) and of the range in between.

The kinds of calls, by what they stand for:
  decide    the tolerance a track keeps, found by the user's own bisection: one reachability
            question after another (Context.decide, host curves), where latency counts
  noalloc   the same without allocation, on device memory (decide_noalloc), as a control loop
            asks it: each answer is read before the next question
  drop_in   compute_distance_parallel: the reference's call, stop rule and formulas
  bounds    the discrete and the vertex-edge distance (Context.bounds)
  pair      one pair in device memory, to 2^-33 relative: the plain method, or with the learned
            bracket and the coarse upper bound (the benchmark's long-pair form)
  batch     uneven pairs in one call (Context.distance_batch): plain or learned, FP64 or the
            FP32 filter, host or device curves
  matrix    all pairwise distances of a set of curves (Context.distance_matrix)
  gradients forward and backward pass of the bracket network (Model.gradients)

A solve returns its numbers (distance, discrete, vertex-edge and endpoint distance, bracket)
and its probe count and flags.  The cells_* counters are left out: they count the kernels'
work, speculative tiles included, and differ from run to run.
"""
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import robotfd_b200 as rfd

VALUES = ("distance", "dfd", "vefd", "endpoint", "lb", "ub")
WALK, SPLINE = 0, 1


def listed():
    return [
        # two short plans compared: the smallest call
        {"name": "bounds_short", "kind": "bounds", "style": WALK, "dims": 2, "n1": 61, "n2": 52},
        # tolerances of recorded tracks of ordinary length, second curve the shorter
        {"name": "decide_track", "kind": "decide", "style": SPLINE, "dims": 3, "n1": 5003,
         "n2": 4100, "from": 0.1, "to": 2.0, "steps": 12},
        # the allocation-free form inside a running loop
        {"name": "noalloc_loop", "kind": "noalloc", "style": WALK, "dims": 3, "n1": 1281,
         "n2": 1100, "from": 0.1, "to": 4.0, "steps": 12},
        # the reference's own call on its 2D workload
        {"name": "drop_in_2d", "kind": "drop_in", "style": WALK, "dims": 2, "n1": 2000, "n2": 1900},
        # both bounds of two long recorded tracks
        {"name": "bounds_long", "kind": "bounds", "style": SPLINE, "dims": 2, "n1": 60000,
         "n2": 45001},
        # one ordinary pair solved by the plain method
        {"name": "pair_plain", "kind": "pair", "style": SPLINE, "dims": 3, "n1": 20000,
         "n2": 19003, "learned": False, "coarse": 0},
        # a dense track against a sparse plan: one curve much the longer
        {"name": "pair_thin", "kind": "pair", "style": WALK, "dims": 2, "n1": 50000, "n2": 1039,
         "learned": False, "coarse": 0},
        # the benchmark's long pair: learned bracket, coarse upper bound
        {"name": "pair_long", "kind": "pair", "style": SPLINE, "dims": 3, "n1": 200000,
         "n2": 200000, "learned": True, "coarse": 6},
        # many short pairs, the plain method with the reference's stop rule, host curves
        {"name": "batch_short", "kind": "batch", "pairs": 256, "median": 400, "sigma": 0.6,
         "longest": 2000, "learned": False, "filter": False, "device": False, "precise": False},
        # an uneven batch as the benchmark's, a quarter of its pairs, curves in device memory
        {"name": "batch_uneven", "kind": "batch", "pairs": 1024, "median": 2000, "sigma": 1.0,
         "longest": 50000, "learned": True, "filter": False, "device": True, "precise": True},
        # the mixed-precision form of a smaller one, host curves
        {"name": "batch_filter", "kind": "batch", "pairs": 192, "median": 2000, "sigma": 0.7,
         "longest": 20000, "learned": True, "filter": True, "device": False, "precise": True},
        # one gradient of the bracket network on 4,096 labelled pairs
        {"name": "gradients", "kind": "gradients", "rows": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decide", "decide", "noalloc", "drop_in", "bounds", "pair", "pair", "batch",
                       "batch", "matrix", "gradients"])
    style, dims = rng.choice([WALK, SPLINE]), rng.choice([2, 3])
    if kind in ("decide", "noalloc"):
        most = 20000 if kind == "decide" else 8000
        n1 = _log_int(rng, 100, most)
        # curves of like length: the bisection starts on both sides of their distance
        return {"kind": kind, "style": style, "dims": dims, "n1": n1,
                "n2": min(most, max(40, round(n1 * rng.uniform(0.6, 1.6)))), "from": 0.1,
                "to": 4.0, "steps": rng.randint(10, 16)}
    if kind == "drop_in":
        return {"kind": kind, "style": style, "dims": dims, "n1": _log_int(rng, 100, 8000),
                "n2": _log_int(rng, 100, 8000)}
    if kind == "bounds":
        return {"kind": kind, "style": style, "dims": dims, "n1": _log_int(rng, 40, 60000),
                "n2": _log_int(rng, 40, 60000)}
    if kind == "pair":
        if rng.random() < 0.5:
            return {"kind": kind, "style": SPLINE, "dims": 3, "n1": _log_int(rng, 20000, 200000),
                    "n2": _log_int(rng, 20000, 200000), "learned": True, "coarse": 6}
        return {"kind": kind, "style": style, "dims": dims, "n1": _log_int(rng, 1000, 20000),
                "n2": _log_int(rng, 1000, 20000), "learned": False, "coarse": 0}
    if kind == "batch":
        learned = rng.random() < 0.7
        return {"kind": kind, "pairs": _log_int(rng, 12, 700), "median": _log_int(rng, 300, 2500),
                "sigma": round(rng.uniform(0.3, 1.0), 2), "longest": 20000, "learned": learned,
                "filter": learned and rng.random() < 0.4, "device": rng.random() < 0.5,
                "precise": learned or rng.random() < 0.5}
    if kind == "matrix":
        return {"kind": kind, "curves": rng.randint(5, 32), "median": _log_int(rng, 100, 1200)}
    return {"kind": "gradients", "rows": _log_int(rng, 64, 4096)}


# ---------------------------------------------------------------- inputs

def _scale(style):
    return (1.0, 0.05) if style == WALK else (100.0, 0.1)


def _pair(case, seed):
    scale, noise = _scale(case["style"])
    return rfd.gen_pair(case["style"], case["dims"], case["n1"], case["n2"], scale, noise, seed, 1)


def _batch(case, seed):
    """Uneven pairs: dimension and style at even odds, lognormal lengths (the benchmark's mix)."""
    g = np.random.default_rng(seed)
    n = case["pairs"]
    sizes = np.exp(math.log(case["median"]) + case["sigma"] * g.standard_normal((n, 2)))
    sizes = np.clip(np.rint(sizes), 100, case["longest"]).astype(int)
    dims, styles = g.integers(2, 4, n), g.integers(0, 2, n)

    def one(k):
        scale, noise = _scale(int(styles[k]))
        return rfd.gen_pair(int(styles[k]), int(dims[k]), int(sizes[k, 0]), int(sizes[k, 1]),
                            scale, noise, seed, k)

    with ThreadPoolExecutor(max(1, min(16, os.cpu_count() or 1))) as ex:
        return list(ex.map(one, range(n)))


def _bisect(case, right_end):
    """Radii asked and the right ends answered, narrowing [from, to] around the tolerance."""
    lo, hi, asked, got = case["from"], case["to"], [], []
    for _ in range(case["steps"]):
        r = 0.5 * (lo + hi)
        right = right_end(r)
        asked.append(r)
        got.append(right)
        if right == 1.0:
            hi = r
        else:
            lo = r
    return np.array(asked), np.array(got)


def _curve_set(case, seed):
    """Noisy resamplings of one walk at different rates: tracks of the same route."""
    g = np.random.default_rng(seed)
    curves = []
    for k in range(case["curves"]):
        n = int(np.clip(round(case["median"] * math.exp(0.4 * g.standard_normal())), 20, 4000))
        base, track = rfd.gen_pair(WALK, 2, case["median"], n, 1.0, 0.05, seed, 3)
        curves.append(np.ascontiguousarray(track + 0.3 * g.standard_normal(track.shape)))
    return curves


def _network_rows(case, seed):
    """Feature rows (centred, scaled to at most 1, zero padding) and targets in the labels' range."""
    g = np.random.default_rng(seed)
    x = np.zeros((case["rows"], rfd.FEATURE_WIDTH), dtype=np.float32)
    x[:, :rfd.N_FEATURES] = np.clip(0.4 * g.standard_normal((case["rows"], rfd.N_FEATURES)), -1, 1)
    t = (-1.7 + 1.2 * g.standard_normal(case["rows"])).astype(np.float32)
    return x, t


_MODEL = None


def _model():
    global _MODEL
    if _MODEL is None:
        _MODEL = rfd.Model.pretrained(0)
    return _MODEL


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": rfd.default_context()}
    if kind in ("decide", "drop_in", "bounds"):
        s["P"], s["Q"] = _pair(case, seed)
    elif kind in ("noalloc", "pair"):
        P, Q = _pair(case, seed)
        s["dP"], s["dQ"] = torch.from_numpy(P).cuda(), torch.from_numpy(Q).cuda()
        if kind == "noalloc":
            s["out"] = torch.empty(1, dtype=torch.float64, device="cuda")
        elif case["learned"]:
            s["model"] = _model()
    elif kind == "batch":
        pairs = _batch(case, seed)
        if case["device"]:
            dev = [(torch.from_numpy(p).cuda(), torch.from_numpy(q).cuda()) for p, q in pairs]
            s["keep"] = dev
            s["Ps"] = [(p.data_ptr(), len(p), p.shape[1]) for p, _ in dev]
            s["Qs"] = [(q.data_ptr(), len(q), q.shape[1]) for _, q in dev]
        else:
            s["Ps"], s["Qs"] = [p for p, _ in pairs], [q for _, q in pairs]
        s["kw"] = {"precise": case["precise"],
                   "memory": rfd.RFD_MEM_DEVICE if case["device"] else rfd.RFD_MEM_HOST,
                   "precision": rfd.RFD_PREC_FP32_FILTER if case["filter"] else rfd.RFD_PREC_FP64}
        if case["learned"]:
            s["kw"]["model"] = _model()
    elif kind == "matrix":
        s["curves"] = _curve_set(case, seed)
    else:
        x, t = _network_rows(case, seed)
        s["x"], s["t"], s["model"] = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), _model()
    torch.cuda.synchronize()  # the context works on a stream of its own
    return s


def _numbers(results):
    return (np.array([[r[k] for k in VALUES] for r in results]),
            np.array([[r["probes"], r["flags"]] for r in results], dtype=np.int64))


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "decide":
        return _bisect(case, lambda r: ctx.decide(state["P"], state["Q"], r)[1])
    if kind == "noalloc":
        dP, dQ, out = state["dP"], state["dQ"], state["out"]
        stream = torch.cuda.current_stream().cuda_stream

        def ask(r):
            rfd.decide_noalloc(dP.data_ptr(), len(dP), dQ.data_ptr(), len(dQ), case["dims"], r,
                               stream, out.data_ptr())
            return out.item()

        return _bisect(case, ask)
    if kind == "drop_in":
        return rfd.compute_distance_parallel(state["P"], state["Q"])
    if kind == "bounds":
        return np.array(ctx.bounds(state["P"], state["Q"], quirks=False))
    if kind == "pair":
        dP, dQ = state["dP"], state["dQ"]
        return _numbers([ctx.distance_device(dP.data_ptr(), len(dP), dQ.data_ptr(), len(dQ),
                                             case["dims"], precise=True, model=state.get("model"),
                                             coarse_ub=case["coarse"])])
    if kind == "batch":
        return _numbers(ctx.distance_batch(state["Ps"], state["Qs"], **state["kw"]))
    if kind == "matrix":
        return ctx.distance_matrix(state["curves"], precise=True)
    return state["model"].gradients(state["x"].data_ptr(), state["t"].data_ptr(), case["rows"])


# ---------------------------------------------------------------- necessary work

def _sweep_flops(n1, n2, d, probes):
    """One vertex-edge sweep and `probes` decisions along a path through the grid: no method
    evaluates fewer cells than one per row and column it passes."""
    return (n1 + n2) * ((24 * d + 2) + probes * (12 * d + 22))


def work(case):
    kind = case["kind"]
    if kind == "gradients":
        w = rfd.Model.num_params()
        return {"bytes": 4 * case["rows"] * (rfd.FEATURE_WIDTH + 1) + 8 * w,
                "flops": 6 * case["rows"] * w}
    if kind == "matrix":
        n, m = case["curves"], case["median"]
        pairs = n * (n - 1) // 2
        return {"bytes": 16 * n * m + 8 * n * n,
                "flops": pairs * ((2 * m) * 9 + _sweep_flops(m, m, 2, 1))}
    if kind == "batch":
        m = case["median"] * math.exp(0.5 * case["sigma"] ** 2)
        return {"bytes": int(case["pairs"] * (2 * m * 20 + 64)),
                "flops": int(case["pairs"] * (2 * m * 10 + _sweep_flops(m, m, 2.5, 1)))}
    n1, n2, d = case["n1"], case["n2"], case["dims"]
    data = 8 * d * (n1 + n2) + 64
    if kind in ("decide", "noalloc"):
        return {"bytes": case["steps"] * data,
                "flops": case["steps"] * (n1 + n2) * (12 * d + 22)}
    probes = 0 if kind == "bounds" else 1 if case.get("learned") else 25
    return {"bytes": data, "flops": (n1 + n2) * (3 * d + 3) + _sweep_flops(n1, n2, d, probes)}


# ---------------------------------------------------------------- 64-bit values by other means

def _diagonals(n, m):
    for k in range(n + m - 1):
        i = np.arange(max(0, k - m + 1), min(n, k + 1))
        yield i, k - i


def _discrete(P, Q):
    """Discrete Frechet distance, an anti-diagonal at a time."""
    n, m = len(P), len(Q)
    one, two = np.full(n + 1, np.inf), np.full(n + 1, np.inf)  # value of row i at index i + 1
    for i, j in _diagonals(n, m):
        best = np.minimum(np.minimum(one[i], one[i + 1]), two[i])
        if i[0] == 0 and j[0] == 0:
            best = np.zeros(1)
        cur = np.full(n + 1, np.inf)
        cur[i + 1] = np.maximum(np.sum((P[i] - Q[j]) ** 2, axis=1), best)
        one, two = cur, one
    return math.sqrt(one[n])


def _point_segment(x, a, b):
    ab = b - a
    t = np.clip(np.sum((x - a) * ab, axis=1) / np.sum(ab * ab, axis=1), 0.0, 1.0)
    return np.sum((x - a - t[:, None] * ab) ** 2, axis=1)


def _vertex_edge(P, Q, seed):
    """Vertex-edge distance: paths from cell to cell, an edge crossed costing the distance of
    its vertex to its segment."""
    R, C = len(P) - 1, len(Q) - 1
    up, along = np.full(R + 1, np.inf), np.full(R + 1, np.inf)
    along[0] = seed
    for i, j in _diagonals(R, C):
        reach = np.minimum(up[i], along[i])
        right = _point_segment(P[i + 1], Q[j], Q[j + 1])
        top = _point_segment(Q[j + 1], P[i], P[i + 1])
        nu, na = np.full(R + 1, np.inf), np.full(R + 1, np.inf)
        nu[i + 1] = np.maximum(right, reach)
        na[i] = np.maximum(top, reach)
        up, along = nu, na
    return math.sqrt(min(up[R], along[R - 1]))


def _free(x, a, b, r):
    d, m = b - a, a - x
    A, B = np.sum(d * d, axis=1), 2.0 * np.sum(m * d, axis=1)
    disc = B * B - 4.0 * A * (np.sum(m * m, axis=1) - r * r)
    s = np.sqrt(np.maximum(disc, 0.0))
    lo, hi = (-B - s) / (2.0 * A), (-B + s) / (2.0 * A)
    empty = (disc < 0.0) | (hi < 0.0) | (lo > 1.0)
    return np.where(empty, np.inf, np.clip(lo, 0.0, 1.0)), np.where(empty, -np.inf, np.clip(hi, 0.0, 1.0))


def _right_end(P, Q, r):
    """Upper end of the reachable part of the last cell's right edge (p_n against the last
    segment of Q); -2 when none is reachable."""
    R, C = len(P) - 1, len(Q) - 1
    up, along = np.full(R + 1, np.inf), np.full(R + 1, np.inf)  # first reachable point, inf: none
    along[0] = 0.0
    last = -2.0
    for i, j in _diagonals(R, C):
        below, beside = up[i], along[i]
        lo, hi = _free(P[i + 1], Q[j], Q[j + 1], r)
        start = np.where(np.isfinite(beside), lo, np.maximum(lo, below))
        start = np.where(start <= hi, start, np.inf)
        tlo, thi = _free(Q[j + 1], P[i], P[i + 1], r)
        side = np.where(np.isfinite(below), tlo, np.maximum(tlo, beside))
        side = np.where(side <= thi, side, np.inf)
        nu, na = np.full(R + 1, np.inf), np.full(R + 1, np.inf)
        nu[i + 1], na[i] = start, side
        if i[-1] == R - 1 and j[-1] == C - 1:
            last = float(hi[-1]) if np.isfinite(start[-1]) else -2.0
        up, along = nu, na
    return last


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradients":
        return _exact_gradients(*_network_rows(case, seed))
    if kind not in ("decide", "noalloc", "drop_in", "bounds"):
        return None
    calls = case["steps"] if kind in ("decide", "noalloc") else 2 if kind == "bounds" else 40
    if calls * (case["n1"] + case["n2"]) > 60000:
        return None  # longer than this takes here
    P, Q = _pair(case, seed)
    if kind in ("decide", "noalloc"):
        return _bisect(case, lambda r: _right_end(P, Q, r))
    seed_sq = max(float(np.sum((P[0] - Q[0]) ** 2)), float(np.sum((P[-1] - Q[-1]) ** 2)))
    if kind == "bounds":
        return np.array([_discrete(P, Q), _vertex_edge(P, Q, seed_sq)])
    lb, ub = math.sqrt(seed_sq), _discrete(P, Q)
    while ub - lb > 2.0 ** -40 * ub:
        mid = 0.5 * (lb + ub)
        if not lb < mid < ub:
            break
        if _right_end(P, Q, mid) == 1.0:
            ub = mid
        else:
            lb = mid
    return 0.5 * (lb + ub)


def _exact_gradients(x, t):
    """Loss and gradients of the 400-256-256-256-2 network (tanh-form GELU, pinball loss at 0.05
    and 0.95), parameters laid out layer by layer, weights [out][in] then biases."""
    dims, p, at, layers = (400, 256, 256, 256, 2), _model().get_params().astype(np.float64), 0, []
    for a, b in zip(dims[:-1], dims[1:]):
        layers.append((p[at:at + a * b].reshape(b, a), p[at + a * b:at + a * b + b]))
        at += a * b + b
    c0, c1 = math.sqrt(2.0 / math.pi), 0.044715
    h, zs, hs = x.astype(np.float64), [], [x.astype(np.float64)]
    for k, (w, b) in enumerate(layers):
        z = h @ w.T + b
        zs.append(z)
        h = 0.5 * z * (1.0 + np.tanh(c0 * (z + c1 * z ** 3))) if k < 3 else z
        hs.append(h)
    tau = np.array([0.05, 0.95])
    u = t.astype(np.float64)[:, None] - h
    loss = float(np.sum(u * (tau - (u < 0.0))) / len(x))
    d = -(tau - (u < 0.0)) / len(x)
    parts = []
    for k in range(3, -1, -1):
        w, _ = layers[k]
        parts = [(d.T @ hs[k]).ravel(), d.sum(axis=0)] + parts
        if k:
            z = zs[k - 1]
            th = np.tanh(c0 * (z + c1 * z ** 3))
            d = (d @ w) * (0.5 * (1.0 + th) + 0.5 * z * (1.0 - th ** 2) * c0 * (1.0 + 3.0 * c1 * z * z))
    return np.concatenate(parts), loss
