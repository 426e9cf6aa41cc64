"""Fed DFD strips (weights computed by feeder warps, rows along the shorter curve) against the
strips whose warp computes both (RFD_DFD_SKEW=1) and against the oracle: sizes around the 32-row
strips and 32-column tiles, both orientations, the coarse bound's inflated weights, boundary rings
of two rows, and several pairs in one launch."""
import os

import numpy as np
import pytest

import oracle


def context(built, **env):
    env = {"RFD_WALK": "0", **env}
    os.environ.update(env)
    try:
        return built.Context(0)
    finally:
        for k in env:
            del os.environ[k]


@pytest.fixture(scope="module")
def both(built):
    c = [context(built), context(built, RFD_DFD_RING_ROWS="2"), context(built, RFD_DFD_SKEW="1")]
    yield c
    for x in c:
        x.close()


SIZES = [(2, 2), (2, 64), (33, 31), (31, 33), (32, 32), (64, 65), (65, 1), (1, 97), (65, 65), (66, 64), (97, 200), (129, 300),
         (300, 129), (1000, 40), (40, 3000), (4097, 2300)]


@pytest.mark.gpu
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("n1,n2", SIZES)
def test_fed_strips(both, built, d, n1, n2):
    P, Q = built.gen_pair(1, d, max(n1, 2), max(n2, 2), 100.0, 0.1, 96, n1)
    P, Q = P[:n1].copy(), Q[:n2].copy()
    if n1 * n2 < 200_000 and min(n1, n2) > 1:
        want = oracle.distance(P, Q, stop_mode=1, quirks=False)["dfd"]
    else:
        want = both[2].distance(P, Q, precise=True, max_probes=1)["dfd"]
    for c in both:
        assert c.distance(P, Q, precise=True, max_probes=1)["dfd"] == want
    for k in (2, 6):
        a = [c.distance(P, Q, precise=True, max_probes=1, coarse_ub=k)["dfd"] for c in both]
        assert a[0] == a[1] == a[2]


@pytest.mark.gpu
@pytest.mark.parametrize("coarse", [0, 3])
def test_fed_strips_of_several_pairs(both, built, coarse):
    g = np.random.default_rng(11)
    pairs = [built.gen_pair(k % 2, 2 + k % 2, *(int(v) for v in g.integers(2, 700, 2)), 1.0, 0.1, 97, k)
             for k in range(24)]
    Ps, Qs = [p for p, _ in pairs], [q for _, q in pairs]
    kw = dict(precise=True, max_probes=1, coarse_ub=coarse)
    a = [[r["dfd"] for r in c.distance_batch(Ps, Qs, **kw)] for c in both]
    assert a[0] == a[1] == a[2]
    assert a[0] == [r["dfd"] for r in both[0].distance_batch(Ps, Qs, **{**kw, "graph": True})]


@pytest.mark.gpu
@pytest.mark.parametrize("npairs,longest", [(9, 60000), (40, 9000), (500, 900)])
def test_batches_on_either_side_of_the_rows_rule(built, both, npairs, longest):
    """Four or eight rows a lane, by the strips of the call, against eight skewed."""
    g = np.random.default_rng(npairs)
    pairs = []
    for k in range(npairs):
        n1 = int(g.integers(longest // 2, longest))
        pairs.append(built.gen_pair(k % 2, 2 + k % 2, n1, int(g.integers(2, 300)), 1.0, 0.1, 98, k))
    Ps, Qs = [p for p, _ in pairs], [q for _, q in pairs]
    a = [[r["dfd"] for r in c.distance_batch(Ps, Qs, precise=True, max_probes=1)] for c in both]
    assert a[0] == a[1] == a[2]
