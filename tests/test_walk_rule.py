"""CPU model of the walk sweeps' rules (rfd_walk.cuh), against the plain cell recurrences.

Block rule: the decision's rows of a block by carry chains of bits, as far as no value stands in
the way of another (walk_bits), equal the recurrence cell by cell, on tie-heavy intervals.

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


def bit_block(rl, ru, tl, tu, F, xin):
    """walk_bits<K_DEC> on rows 0 .. nr - 1: the rows settled by bits, what they hand on up (values)
    and to the right (one value a row)."""
    n, full, nr = 32, 0xffffffff, len(rl)

    def bits(a):
        return sum(1 << j for j in range(n) if a[j])
    V = bits(F < 2.0)
    above = bits((F < 2.0) & (F > 0.0))
    rows = []
    for r in range(nr):
        mr, mt = bits(rl[r] >= 0.0), bits(tl[r] >= 0.0)
        gen = V & mt
        X = ((mt + gen + int(xin[r] < 2.0)) ^ mt ^ gen) & full
        ok = mr & (X | V)
        held = above & ~X
        ends = bits((rl[r] >= 0.0) & (ru[r] < 1.0))
        rows.append((X, ok, X & ~V & mt, mt & (X | V), ok & held & ends))
        above = ok & (bits((rl[r] >= 0.0) & (rl[r] > 0.0)) | held)
        V = ok

    def run(c, r):
        """Largest start from row r down to where column c's run began."""
        f = 0.0
        while True:
            if r < 0:
                return max(f, F[c])
            f = max(f, rl[r][c])
            if rows[r][0] >> c & 1:
                return f
            r -= 1
    out, nok = [], nr
    for r, (X, ok, passing, Y, risk) in enumerate(rows):
        ends = bits((tl[r] >= 0.0) & (tu[r] < 1.0)) | 1 << 31
        x, before, clash = DEAD, -2, False
        if passing & ends:
            for c in range(n):
                if passing >> c & 1:
                    frm = x if before == c - 1 else xin[r] if c == 0 else tl[r][c - 1]
                    clash |= tu[r][c] < frm
                    x, before = max(tl[r][c], frm), c
        for c in range(n):
            if risk >> c & 1:
                clash |= ru[r][c] < run(c, r - 1)
        if clash:
            nok = r
            break
        out.append((x if before == 31 else tl[r][31]) if Y >> 31 & 1 else DEAD)
    up = F if nok == 0 else np.array(
        [run(c, nok - 1) if rows[nok - 1][1] >> c & 1 else DEAD for c in range(n)])
    return nok, up, out


@pytest.mark.parametrize("levels,empty,cut", [(3, 0.1, 0.1), (3, 0.5, 0.4), (8, 0.2, 0.02),
                                              (1000, 0.05, 0.01), (1000, 0.4, 0.3)])
def test_block_of_bits_equals_recurrence(levels, empty, cut):
    g = np.random.default_rng(levels + int(100 * empty))
    whole = clashed = 0
    for _ in range(300):
        nr = int(g.integers(1, 33))

        def interval():
            a = np.sort(g.integers(0, levels + 1, (2, nr, 32)) / levels, axis=0)
            gone, open_ = g.random((nr, 32)) < empty, g.random((2, nr, 32)) >= cut
            lo, hi = np.where(open_[0], 0.0, a[0]), np.where(open_[1], 1.0, a[1])
            return np.where(gone, -1.0, lo), np.where(gone, -2.0, hi)
        (rl, ru), (tl, tu) = interval(), interval()
        F = np.where(g.random(32) < g.random(), g.integers(0, levels + 1, 32) / levels, DEAD)
        xin = np.where(g.random(nr) < g.random(), g.integers(0, levels + 1, nr) / levels, DEAD)
        r = 0
        while r < nr:
            n, up, out = bit_block(rl[r:], ru[r:], tl[r:], tu[r:], F, xin[r:])
            whole += r == 0 and n == nr
            for k in range(n):
                F, x = serial_row(rl[r + k], ru[r + k], tl[r + k], tu[r + k], F, xin[r + k])
                assert x == out[k]
            assert np.array_equal(F, up)
            r += n
            if r < nr:  # a row with its values
                G, x = serial_row(rl[r], ru[r], tl[r], tu[r], F, xin[r])
                F = G
                clashed += 1
                r += 1
    assert whole > 0 and clashed > 0


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
