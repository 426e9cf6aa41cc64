"""Where a walk does not pay (wide bands, small grids, thin pairs) the strips take over: the same
results on every route, and not much later than on the strips alone (RFD_WALK=0)."""
import os
import time

import numpy as np
import pytest

KEYS = ("distance", "dfd", "vefd", "endpoint", "lb", "ub", "probes", "flags", "cells_nominal")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def strips(built):
    os.environ["RFD_WALK"] = "0"
    try:
        c = built.Context(0)
    finally:
        del os.environ["RFD_WALK"]
    yield c
    c.close()


def curves(built, kind, d, n1, n2, seed=7):
    g = np.random.default_rng(seed)
    if kind == "indep":    # two walks that have nothing to do with each other
        return np.cumsum(g.standard_normal((n1, d)), 0), np.cumsum(g.standard_normal((n2, d)), 0)
    if kind == "noise":    # every point near every other
        return g.standard_normal((n1, d)), g.standard_normal((n2, d))
    if kind == "loops":    # thirty turns of the same circle: many bands beside the true one
        def turn(n):
            t = 2 * np.pi * np.linspace(0, 30, n)
            return np.stack([np.cos(t), np.sin(t)] + [0.003 * t] * (d - 2), 1) + \
                0.01 * g.standard_normal((n, d))
        return turn(n1), turn(n2)
    return built.gen_pair(0, d, n1, n2, 1.0, 0.05, seed, 1)


@pytest.mark.parametrize("kind", ["walk", "indep", "noise", "loops"])
@pytest.mark.parametrize("d,n1,n2", [(2, 97, 96), (3, 98, 97), (2, 300, 260), (2, 470, 480),
                                     (3, 620, 640), (2, 1281, 1100), (2, 90, 1500), (3, 2300, 2100)])
def test_routes_agree(ctx, strips, built, kind, d, n1, n2):
    import torch
    P, Q = curves(built, kind, d, n1, n2)
    a, b = ctx.distance(P, Q, precise=True), strips.distance(P, Q, precise=True)
    assert [a[k] for k in KEYS] == [b[k] for k in KEYS]
    assert ctx.bounds(P, Q, quirks=False) == strips.bounds(P, Q, quirks=False)
    dP, dQ = torch.from_numpy(P).cuda(), torch.from_numpy(Q).cuda()
    out = torch.empty(1, dtype=torch.float64, device="cuda")
    for r in a["distance"] * np.array([0.9, 1 + 1e-4, 2.0, 10.0]):
        want = strips.decide(P, Q, r)
        assert ctx.decide(P, Q, r) == want
        built.decide_noalloc(dP.data_ptr(), n1, dQ.data_ptr(), n2, d, r,
                             torch.cuda.current_stream().cuda_stream, out.data_ptr())
        assert out.item() == want[1]


@pytest.mark.parametrize("kind", ["indep", "loops"])
@pytest.mark.parametrize("kw", [dict(), dict(coarse_ub=4), dict(max_probes=6, graph=True)])
def test_routes_agree_in_calls_of_several(ctx, strips, built, kind, kw):
    """Calls whose pairs are given up in different phases, among pairs that are walked to the end."""
    g = np.random.default_rng(3)
    for n, top in ((6, 460), (12, 1500), (170, 400)):
        pairs = [curves(built, kind if k % 3 else "walk", 2 + k % 2, *(int(v) for v in g.integers(60, top, 2)),
                        seed=k) for k in range(n)]
        Ps, Qs = [p for p, _ in pairs], [q for _, q in pairs]
        a = ctx.distance_batch(Ps, Qs, precise=True, **kw)
        b = strips.distance_batch(Ps, Qs, precise=True, **{**kw, "graph": False})
        assert [[x[k] for k in KEYS] for x in a] == [[x[k] for k in KEYS] for x in b]


def least(f, g, reps=40):
    """Least times of two calls, taken in turn."""
    t = [[], []]
    for _ in range(reps + 1):
        for k, h in enumerate((f, g)):
            t0 = time.perf_counter()
            h()
            t[k].append(time.perf_counter() - t0)
    return min(t[0][1:]), min(t[1][1:])


@pytest.mark.parametrize("kind,n1,n2", [("indep", 300, 260), ("indep", 600, 610), ("noise", 600, 610),
                                        ("loops", 1281, 1100)])
def test_wide_bands_cost_little_more_than_the_strips(ctx, strips, built, kind, n1, n2):
    """Before the walk kept to a share of the strips' time: 5, 11, 8 and 15 times as long.  (Other
    users of the host can disturb calls for a second or two: up to four tries.)"""
    P, Q = curves(built, kind, 2, n1, n2)
    for _ in range(4):
        a, b = least(lambda: ctx.bounds(P, Q, quirks=False), lambda: strips.bounds(P, Q, quirks=False))
        if a < 2.5 * b:
            return
        time.sleep(1.0)
    assert a < 2.5 * b


def test_thin_pairs_run_on_the_strips_at_once(ctx, strips, built):
    """A call with nothing to walk makes the strips' launches and no others."""
    P, Q = built.gen_pair(0, 2, 12000, 400, 1.0, 0.1, 5, 0)
    R, S = built.gen_pair(0, 2, 300, 260, 1.0, 0.1, 5, 1)
    count = []
    for c in (ctx, strips):
        c.phase_times(1)
        for X, Y in ((P, Q), (R, S)):
            c.decide(X, Y, 1.0)
            count.append(c.phase_times()["launches"])
        c.bounds(P, Q, quirks=False)
        count.append(c.phase_times()["launches"])
        c.phase_times(0)
    assert count[:3] == count[3:]


def test_vefd_ahead_of_a_given_up_dfd_is_kept(ctx, strips, built):
    """A group sweeps the VE-FD before the DFD; where it then gives the DFD up (a stretch of this pair
    is wide) the strips sweep the DFD only."""
    P, Q = built.gen_pair(1, 2, 60000, 45001, 100.0, 0.1, 970302523, 1)
    ms, got = [], []
    for c in (ctx, strips):
        c.phase_times(1)
        t = []
        for _ in range(6):
            got.append(c.bounds(P, Q, quirks=False))
            t.append(c.phase_times(1)["vefd_ms"])
        c.phase_times(0)
        ms.append(min(t))
    assert len(set(got)) == 1
    assert ms[0] < 0.3 * ms[1]
