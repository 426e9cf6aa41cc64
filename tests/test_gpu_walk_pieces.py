"""Walk sweeps of a group of CTAs (rfd_walk.cuh) against the strips (RFD_WALK=0), where the pieces of
the grid are cut in uncommon ways."""
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


def check(ctx, strips, P, Q):
    a, b = ctx.distance(P, Q, precise=True), strips.distance(P, Q, precise=True)
    assert [a[k] for k in KEYS] == [b[k] for k in KEYS]
    assert ctx.bounds(P, Q, quirks=False) == strips.bounds(P, Q, quirks=False)
    for r in np.geomspace(0.5 * a["distance"], 1.2 * a["dfd"], 5):
        assert ctx.decide(P, Q, r) == strips.decide(P, Q, r)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("dwell,n,m", [(400, 2500, 1400), (1000, 4000, 2600), (700, 1500, 760)])
def test_band_far_along_the_first_row(ctx, strips, built, d, dwell, n, m):
    """A track that waits at its start: the band runs along the first block row past the first
    piece's share of it."""
    P, Q = built.gen_pair(0, d, n, m - dwell, 1.0, 0.05, 96, n)
    g = np.random.default_rng(dwell)
    Q = np.concatenate([Q[0] + 0.01 * g.standard_normal((dwell, d)), Q])
    check(ctx, strips, P, Q)
    check(ctx, strips, Q, P)


@pytest.mark.gpu
@pytest.mark.parametrize("style,d,n1,n2", [
    (0, 2, 449, 449), (0, 3, 609, 609), (1, 2, 929, 929), (0, 2, 1025, 850), (0, 2, 850, 1025),
    (0, 2, 1889, 1600), (1, 3, 2049, 2049), (0, 2, 2049, 2049), (1, 3, 20001, 19003)])
def test_grids_of_different_piece_counts(ctx, strips, built, style, d, n1, n2):
    """Sizes whose DFD grid, a row and a column more than the VE-FD's, has a piece more."""
    P, Q = built.gen_pair(style, d, n1, n2, 100.0 if style else 1.0, 0.1, 97, n1)
    check(ctx, strips, P, Q)


@pytest.mark.gpu
def test_last_pairs_of_a_batch_of_like_pairs(strips, built):
    """A batch without leading pairs, whose last ten searches share the CTAs: groups that start their
    pieces by the chunks' bounds, in a workspace that an earlier call has filled.  (The curves lie
    far from the origin, where zeros would say that no chunk is in reach.)"""
    pairs = [built.gen_pair(0, 2, 900 + k % 7, 800 + k % 5, 1.0, 0.05, 98, k) for k in range(300)]
    Ps, Qs = [p + 1000.0 for p, _ in pairs], [q + 1000.0 for _, q in pairs]
    b = strips.distance_batch(Ps, Qs, precise=True)
    d = np.array([r["distance"] for r in b])
    wide = np.arange(300) % 30 == 0
    brackets = np.stack([d * np.where(wide, 0.6, 1 - 1e-12), d * np.where(wide, 1.3, 1 + 1e-12)], axis=1)
    c = built.Context(0)
    try:
        for fill in (0.0, 3.0):
            big = [np.full((40000, 2), fill) + 1e-3 * np.arange(40000)[:, None] * (fill > 0)
                   for _ in range(40)]
            c.distance_batch(big[:20], big[20:], precise=True, max_probes=1)
            for kw in (dict(brackets=brackets), dict(brackets=brackets, graph=True), dict()):
                a = c.distance_batch(Ps, Qs, precise=True, **kw)
                w = strips.distance_batch(Ps, Qs, precise=True, **{**kw, "graph": False})
                assert [[x[k] for k in KEYS] for x in a] == [[x[k] for k in KEYS] for x in w]
    finally:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,m", [(33, 32), (65, 45), (97, 57), (161, 21), (577, 27), (33, 12)])
def test_vefd_of_whole_last_block_rows(ctx, strips, built, n, m):
    """The last block row has 32 rows and the level grows past dead sweeps: what the last row last
    handed up is not the last cell's value unless the sweep came that far."""
    for seed in range(60):
        g = np.random.default_rng(1000 * n + seed)
        d = 2 + seed % 2
        if seed % 3:
            P, Q = np.cumsum(g.standard_normal((n, d)), 0), np.cumsum(g.standard_normal((m, d)), 0)
        else:
            t, u = 2 * np.pi * np.linspace(0, 3, n), 2 * np.pi * np.linspace(0, 3, m)
            P, Q = (np.stack([np.cos(v), np.sin(v)] + [0.1 * v] * (d - 2), 1) +
                    0.2 * g.standard_normal((len(v), d)) for v in (t, u))
        assert ctx.bounds(P, Q, quirks=False) == strips.bounds(P, Q, quirks=False)
        assert ctx.bounds(Q, P, quirks=False) == strips.bounds(Q, P, quirks=False)
