"""CPU model of the walk sweeps' rules (rfd_walk.cuh), against the plain cell recurrences.

Row rule: the decision's row of 32 columns by a carry chain of bits (walk_row) equals the
recurrence cell by cell, on tie-heavy intervals.

Group rule: pieces of a grid that start from everything that could be live (or from part of it),
are walked again from their predecessor's end until a block row's list meets its record (up to
one constant for the min-max kinds), and so on by rounds, end with the serial sweep's result.
"""
import numpy as np
import pytest

DEAD = 4.0
BIG = float(np.finfo(np.float32).max)


# ------------------------------------------------------------------ row rule

def serial_row(rl, ru, tl, tu, F, x):
    """One row: F live values handed up per column, x entering on the left (DEAD: none)."""
    out = np.empty(len(F))
    for j in range(len(F)):
        bl, ll = x < 2.0, F[j] < 2.0
        right_free, top_free = rl[j] >= 0.0, tl[j] >= 0.0
        up = DEAD
        if right_free and (bl or F[j] <= ru[j]):
            up = rl[j] if bl else max(rl[j], F[j])
        nxt = DEAD
        if top_free and (ll or x <= tu[j]):
            nxt = tl[j] if ll else max(tl[j], x)
        out[j], x = up, nxt
    return out, x


def bit_row(rl, ru, tl, tu, F, x):
    """walk_row<K_DEC>: returns the same, and whether the column-by-column way was taken."""
    n, full = 32, 0xffffffff
    mr = sum(1 << j for j in range(n) if rl[j] >= 0.0)
    mt = sum(1 << j for j in range(n) if tl[j] >= 0.0)
    V = sum(1 << j for j in range(n) if F[j] < 2.0)
    live_in = x < 2.0
    prev = [x if j == 0 else tl[j - 1] for j in range(n)]
    late = sum(1 << j for j in range(n) if tu[j] < prev[j])
    gen = V & mt
    X = ((mt + gen + int(live_in)) ^ mt ^ gen) & full
    passing = X & ~V & mt & full
    slow = bool(passing & (late | (passing << 1)))
    y = [tl[j] if (V >> j) & 1 or not tl[j] < prev[j] else prev[j] for j in range(n)]
    Y = mt & (V | X)
    if slow:
        y = [tl[j] if (mt >> j) & 1 and (V >> j) & 1 else DEAD for j in range(n)]
        while True:
            xs = [x if live_in else DEAD] + y[:-1]
            yn = []
            for j in range(n):
                up = (V >> j) & 1
                ends = not (mt >> j) & 1 or (not up and tu[j] < xs[j])
                yn.append(DEAD if ends else tl[j] if up or not tl[j] < xs[j] else xs[j])
            moved = yn != y
            y = yn
            if not moved:
                break
        X = sum(1 << j for j in range(n) if xs[j] < 2.0)
        Y = sum(1 << j for j in range(n) if y[j] < 2.0)
    out = np.full(n, DEAD)
    for j in range(n):
        xl = (X >> j) & 1
        if (mr >> j) & 1 and (xl or not ru[j] < F[j]):
            out[j] = rl[j] if xl or not rl[j] < F[j] else F[j]
    return out, (y[31] if Y >> 31 else DEAD), slow


@pytest.mark.parametrize("levels,empty", [(3, 0.1), (3, 0.5), (8, 0.2), (1000, 0.05), (1000, 0.4)])
def test_row_of_bits_equals_recurrence(levels, empty):
    g = np.random.default_rng(levels + int(100 * empty))
    slow = 0
    for _ in range(1500):
        def interval():
            a = np.sort(g.integers(0, levels + 1, (2, 32)) / levels, axis=0)
            gone = g.random(32) < empty
            return np.where(gone, -1.0, a[0]), np.where(gone, -2.0, a[1])
        (rl, ru), (tl, tu) = interval(), interval()
        F = np.where(g.random(32) < g.random(), g.integers(0, levels + 1, 32) / levels, DEAD)
        x = g.integers(0, levels + 1) / levels if g.random() < 0.5 else DEAD
        want, xw = serial_row(rl, ru, tl, tu, F, x)
        got, xg, s = bit_row(rl, ru, tl, tu, F, x)
        slow += s
        assert np.array_equal(want, got) and xw == xg
    assert 0 < slow < 1500


# ------------------------------------------------------------------ group rule

class Grid:
    """Random cell values; block rows of `b` rows.  kind 'dec', 'vefd' or 'dfd'."""

    def __init__(self, g, kind, rows, cols, b):
        self.kind, self.rows, self.cols, self.b = kind, rows, cols, b
        q = g.integers(4, 30)
        shape = (rows, cols)
        # a band of likely live cells around a random monotone path
        path = np.minimum.accumulate(np.sort(g.integers(0, cols, rows))[::-1])[::-1]
        far = np.abs(np.arange(cols)[None, :] - path[:, None])
        p = np.clip(1.1 - far / g.uniform(1.5, 6.0), 0.02, 0.98)
        self.live_r, self.live_t = g.random(shape) < p, g.random(shape) < p
        a = np.sort(g.integers(0, q + 1, (2,) + shape) / q, axis=0)
        c = np.sort(g.integers(0, q + 1, (2,) + shape) / q, axis=0)
        self.rl, self.ru, self.tl, self.tu = a[0], a[1], c[0], c[1]
        self.dead = DEAD if kind == "dec" else BIG
        self.nbr = -(-rows // b)

    def walk(self, i, F, start):
        """Block row i from the row below F; start: what row 0 enters column 0 with."""
        res = self.dead
        for r in range(i * self.b, min((i + 1) * self.b, self.rows)):
            x = start if r == 0 else self.dead
            out = np.full(self.cols, self.dead)
            for j in range(self.cols):
                br, bt = self.live_r[r, j], self.live_t[r, j]
                if self.kind == "dec":
                    bl, ll = x < 2.0, F[j] < 2.0
                    up = nx = self.dead
                    if br and (bl or F[j] <= self.ru[r, j]):
                        up = self.rl[r, j] if bl else max(self.rl[r, j], F[j])
                    if bt and (ll or x <= self.tu[r, j]):
                        nx = self.tl[r, j] if ll else max(self.tl[r, j], x)
                else:
                    m = min(F[j], x)
                    if self.kind == "vefd":
                        up = max(self.rl[r, j], m) if br else self.dead
                        nx = max(self.tl[r, j], m) if bt else self.dead
                    else:
                        nx = max(self.tl[r, j], m) if bt else self.dead
                        up = min(nx, x)
                out[j] = up
                last, x = x, nx
            F = out
        end = min(F[-1], x) if self.kind != "dfd" else x
        return F, (end if self.kind != "dec" else (F[-1] if F[-1] < 2.0 else DEAD))

    def everything(self, i):
        """What could be live in the row below block row i."""
        r = i * self.b - 1
        if self.kind != "dfd":
            return np.where(self.live_r[r], self.rl[r], self.dead)
        w = np.where(self.live_t[r], self.tl[r], self.dead)
        return np.minimum(w, np.concatenate([[self.dead], w[:-1]]))

    def bottom(self):
        F = np.full(self.cols, self.dead)
        if self.kind == "dfd":
            F[0] = 0.0
        return F


def group(grid, pieces, drop, g):
    """The rounds of walk_sweep; drop: chance that a start loses some of its entries."""
    dead, start0 = grid.dead, (grid.dead if grid.kind == "dfd" else 0.0)
    cuts = [grid.nbr * m // pieces for m in range(pieces + 1)]
    recs, ends, result, part, empty = {}, [], [], [], []
    least = []
    for m in range(pieces):
        F = grid.bottom() if m == 0 else grid.everything(cuts[m])
        lost = m > 0 and g.random() < drop
        if lost:
            F = np.where(g.random(grid.cols) < 0.5, F, dead)
        for i in range(cuts[m], cuts[m + 1]):
            F, end = grid.walk(i, F, start0)
            recs[i] = F
            if not np.any(F < dead) and i + 1 < grid.nbr:
                end = dead
                for k in range(i + 1, cuts[m + 1]):
                    recs[k] = None
                break
        ends.append(F)
        result.append(end)
        part.append(lost)
        empty.append(cuts[m + 1] < grid.nbr and not np.any(F < dead))
        v = np.min(F) if cuts[m + 1] < grid.nbr else end
        least.append(v if v < dead else 0.0)
    if empty[0] or any(e and not p for e, p in zip(empty, part)):
        return dead, least, part, 0
    first_end, first_res, first_empty = list(ends), list(result), list(empty)
    const = [0.0] * pieces
    changed, rounds = [True] * pieces, 0
    met = [True] * pieces
    while True:
        rounds += 1
        new_ends, new_changed = list(ends), [False] * pieces
        for m in range(1, pieces):
            if not changed[m - 1]:
                continue
            F, c, hit, end = ends[m - 1], 0.0, False, dead
            if np.any(F < dead):
                for i in range(cuts[m], cuts[m + 1]):
                    F, end = grid.walk(i, F, start0)
                    r = recs[i]
                    if i + 1 < grid.nbr and r is not None:
                        if grid.kind == "dec":
                            hit = np.array_equal(F, r)
                        else:
                            c = max([v for v, q in zip(F, r) if v != q], default=0.0)
                            hit = np.array_equal(F, np.maximum(c, r)) and \
                                np.array_equal(F < dead, r < dead)
                    if hit or not np.any(F < dead):
                        break
            if not np.any(F < dead) and cuts[m + 1] < grid.nbr:
                end = dead
            if hit:
                new_ends[m], result[m], empty[m] = first_end[m], first_res[m], first_empty[m]
                const[m], new_changed[m], met[m] = c, not met[m], True
            else:
                new_ends[m], result[m], const[m] = F, end, 0.0
                empty[m] = cuts[m + 1] < grid.nbr and not np.any(F < dead)
                new_changed[m], met[m] = True, False
        ends, changed = new_ends, new_changed
        moved = [m for m in range(pieces) if changed[m]]
        hollow = [m for m in range(pieces) if empty[m]]
        if not moved:
            if hollow or not result[-1] < dead:
                return dead, least, part, rounds
            return (result[-1] if grid.kind == "dec" else max(max(const), result[-1])), least, part, rounds
        if hollow and hollow[0] <= moved[0]:
            return dead, least, part, rounds


@pytest.mark.parametrize("kind", ["dec", "vefd", "dfd"])
@pytest.mark.parametrize("drop", [0.0, 0.5])
def test_pieces_by_rounds_equal_serial_sweep(kind, drop):
    g = np.random.default_rng({"dec": 1, "vefd": 2, "dfd": 3}[kind] + int(10 * drop))
    alive = early = 0
    for _ in range(250):
        rows, cols, b = int(g.integers(8, 40)), int(g.integers(6, 24)), int(g.integers(1, 4))
        grid = Grid(g, kind, rows, cols, b)
        F, want = grid.bottom(), grid.dead
        for i in range(grid.nbr):
            F, want = grid.walk(i, F, grid.dead if kind == "dfd" else 0.0)
            if not np.any(F < grid.dead) and i + 1 < grid.nbr:
                want = grid.dead
                break
        pieces = int(g.integers(2, max(3, grid.nbr // 2 + 1)))
        got, least, part, rounds = group(grid, min(pieces, grid.nbr), drop, g)
        assert got == want
        alive += want < grid.dead
        early += rounds <= 1
        if kind != "dec" and want < grid.dead and not any(part):
            assert max(least) <= want  # the pieces' least values bound the result from below
    assert alive > 20 and early > 20
