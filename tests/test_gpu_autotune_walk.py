"""The autotuners beside the walk sweeps and the fed DFD strips: they time the strips that they tune,
and a tuned context keeps the fed strips where those are the faster ones."""
import os

import pytest

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


def test_autotuners_time_the_strips(strips, built):
    """The walk takes a tenth of these strips' time, so a tuner that timed it would show."""
    P, Q = built.gen_pair(0, 2, 8000, 7600, 1.0, 0.1, 31, 0)
    R, S = built.gen_pair(1, 3, 2000, 1900, 100.0, 0.1, 31, 1)
    c = built.Context(0)
    try:
        for name, pair in (("autotune", (P, Q)), ("autotune_search", (R, S))):
            kw = dict(precise=True) if name == "autotune_search" else {}
            a = getattr(c, name)([pair[0]], [pair[1]], reps=2, **kw)
            b = getattr(strips, name)([pair[0]], [pair[1]], reps=2, **kw)
            assert min(a["ms"].values()) > 0.5 * min(b["ms"].values()), name
    finally:
        c.close()


def test_a_tuned_context_keeps_the_fed_strips(built):
    """The coarse bound's sweep of 30,000 points: 1.3 ms with fed strips, 2.9 without."""
    P, Q = built.gen_pair(1, 3, 30000, 29000, 100.0, 0.1, 32, 0)
    R, S = built.gen_pair(1, 3, 900, 800, 100.0, 0.1, 32, 1)
    ms = []
    for tune in (False, True):
        c = built.Context(0)
        try:
            if tune:
                c.autotune([R], [S], reps=1)
            best = 1e9
            for _ in range(20):
                c.phase_times(1)
                c.distance(P, Q, precise=True, coarse_ub=6, max_probes=1)
                best = min(best, c.phase_times(0)["dfd_ms"])
            ms.append(best)
        finally:
            c.close()
    assert ms[1] < 1.5 * ms[0], ms
