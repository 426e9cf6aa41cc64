"""Tree rounds (two or three probes of a search decided at once, for pairs with one long and one
short curve) against the search probe by probe (RFD_WALK=0), alone and in batches whose pairs
come and go: every reported value, probe and nominal cell counts included (the evaluated ones
depend on the order in which strips end)."""
import numpy as np
import pytest

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
@pytest.mark.parametrize("style,d,n1,n2", [(0, 2, 9000, 40), (1, 3, 64, 8192), (0, 3, 12000, 1025),
                                           (0, 2, 30000, 1300)])
def test_lone_thin_pair(ctx, strips, built, style, d, n1, n2):
    P, Q = built.gen_pair(style, d, n1, n2, 100.0 if style else 1.0, 0.1, 94, n1)
    for kw in (dict(precise=True), dict(precise=False), dict(precise=True, max_probes=4),
               dict(precise=True, max_probes=8, graph=True)):
        a, b = ctx.distance(P, Q, **kw), strips.distance(P, Q, **kw)
        assert {k: a[k] for k in KEYS if k in a} == {k: b[k] for k in KEYS if k in b}


@pytest.mark.gpu
@pytest.mark.parametrize("model", [False, True])
def test_thin_pairs_in_a_batch(ctx, strips, built, model):
    g = np.random.default_rng(8)
    pairs = []
    for k in range(40):
        n1, n2 = (int(v) for v in g.integers(40, 900, 2))
        if k % 4 == 0:
            n1 = int(g.integers(8192, 16000))
        pairs.append(built.gen_pair(int(g.integers(0, 2)), 2 + k % 2, n1, n2, 1.0, 0.1, 95, k))
    Ps, Qs = [p for p, _ in pairs], [q for _, q in pairs]
    # a bracket around the distance, above it, and below it
    plain = strips.distance_batch(Ps, Qs, precise=True)
    for kw in (dict(), dict(max_probes=6)):
        if model:
            w = np.array([r["distance"] for r in plain]) * g.uniform(0.9, 1.1, len(plain))
            kw["brackets"] = np.stack([w * 0.97, w * 1.03], axis=1)
        a = ctx.distance_batch(Ps, Qs, precise=True, **kw)
        b = strips.distance_batch(Ps, Qs, precise=True, **kw)
        for x, y in zip(a, b):
            assert {k: x[k] for k in KEYS if k in x} == {k: y[k] for k in KEYS if k in y}
