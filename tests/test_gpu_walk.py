"""Walk sweeps (rfd_walk.cuh) against the oracle and against the strips (RFD_WALK=0): sizes around
the 32-cell blocks, grids of one piece and of many, bands that are not thin (given up in part
or whole), both orientations and formulas, and a batch whose last pairs share the CTAs."""
import numpy as np
import pytest

import oracle

KEYS = ("distance", "dfd", "vefd", "endpoint", "lb", "ub", "probes", "flags", "cells_nominal")


@pytest.fixture(scope="module")
def strips(built):
    import os
    os.environ["RFD_WALK"] = "0"
    try:
        c = built.Context(0)
    finally:
        del os.environ["RFD_WALK"]
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("style,d,n1,n2", [
    (0, 2, 32, 33), (0, 3, 33, 32), (0, 2, 34, 65), (1, 3, 65, 64), (0, 2, 129, 128),
    (1, 2, 321, 40), (0, 3, 97, 700), (0, 2, 1025, 1023), (1, 3, 1500, 1400), (0, 2, 3000, 500),
    (1, 2, 1500, 40),   # a spacing far below the distance: a wide band
    (1, 2, 2794, 44),   # ... along the block rows: long passes, pieces without rows
    (0, 2, 44, 2794),
    (1, 3, 4100, 6007)])
def test_walk_equals_strips_and_oracle(ctx, strips, built, style, d, n1, n2):
    P, Q = built.gen_pair(style, d, n1, n2, 100.0 if style else 1.0, 0.1, 91, n1)
    a, b = ctx.distance(P, Q, precise=True), strips.distance(P, Q, precise=True)
    assert [a[k] for k in KEYS] == [b[k] for k in KEYS]
    if n1 * n2 < 2_000_000:
        want = oracle.distance(P, Q, stop_mode=1, quirks=False, threads=oracle.max_threads())
        assert (a["distance"], a["dfd"], a["vefd"]) == (want["distance"], want["dfd"], want["vefd"])
    assert ctx.bounds(P, Q, quirks=False) == strips.bounds(P, Q, quirks=False)
    # decisions from below the endpoint bound to far above the distance, right ends included
    for r in np.geomspace(0.3 * a["distance"], 1.5 * a["dfd"], 9):
        for formula in (built.RFD_FORMULA_FUSED, built.RFD_FORMULA_MATERIALISED):
            assert ctx.decide(P, Q, r, formula=formula) == strips.decide(P, Q, r, formula=formula)


@pytest.mark.gpu
def test_walk_on_repeated_points(ctx, strips, built):
    """Zero-length segments are free at every radius: no chunk or edge of one may be skipped."""
    P, Q = built.gen_pair(0, 2, 900, 800, 1.0, 0.05, 92, 0)
    P, Q = P.copy(), Q.copy()
    g = np.random.default_rng(5)
    for X in (P, Q):
        for k in g.integers(1, len(X), 60):
            X[k] = X[k - 1]
    a, b = ctx.distance(P, Q, precise=True), strips.distance(P, Q, precise=True)
    assert [a[k] for k in KEYS] == [b[k] for k in KEYS]
    for r in np.geomspace(0.2 * a["distance"], 2 * a["distance"], 7):
        assert ctx.decide(P, Q, r) == strips.decide(P, Q, r)


@pytest.mark.gpu
@pytest.mark.parametrize("precise", [True, False])
def test_walk_batches_share_the_ctas(ctx, strips, built, precise):
    """More pairs than half the CTAs, a few long ones first, searches past the first probes."""
    g = np.random.default_rng(6)
    pairs = []
    for k in range(180):
        n1, n2 = (int(v) for v in g.integers(40, 400, 2)) if k % 45 else (5000, 4300)
        pairs.append(built.gen_pair(int(g.integers(0, 2)), int(g.integers(2, 4)), n1, n2,
                                    1.0 if k % 2 else 100.0, 0.1, 93, k))
    Ps, Qs = [p for p, _ in pairs], [q for _, q in pairs]
    for kw in (dict(), dict(coarse_ub=4) if precise else dict(max_probes=5), dict(graph=True)):
        a = ctx.distance_batch(Ps, Qs, precise=precise, **kw)
        b = strips.distance_batch(Ps, Qs, precise=precise, **{**kw, "graph": False})
        for x, y in zip(a, b):
            assert [x[k] for k in KEYS] == [y[k] for k in KEYS]
    a = ctx.distance_batch(Ps, Qs, precise=precise, graph=True)  # the captured call, replayed
    assert [x["distance"] for x in a] == [
        x["distance"] for x in strips.distance_batch(Ps, Qs, precise=precise)]
