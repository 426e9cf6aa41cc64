"""The pieces of a walk's grid (rfd_walk_cut.h, compiled for the host): where the band of an earlier
sweep cuts the block rows among the members of a group, and a CPU model of sweeps that follow one
another with such cuts, against the plain recurrences."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "robotfd_b200", "csrc")
SHIM = r"""
#include "rfd_walk_cut.h"
extern "C" int pieces_of(int size, int nbr, int nbc) { return rfd::walk_pieces(size, nbr, nbc); }
// (top: the largest row asked for)
extern "C" int cut_row(int q, int pieces, int n, int nbr, int nbc, const int* hi, int* top) {
  return rfd::walk_cut_row(q, pieces, n, nbr, nbc, [&](int i) {
    if (i > *top) *top = i;
    return hi[i];
  });
}
extern "C" void piece(int cut_pieces, int row0, int row1, int m, int pieces, int nbr, int* rows) {
  rfd::walk_piece(rfd::WalkCut{cut_pieces, row0, row1}, m, pieces, nbr, rows, rows + 1);
}
"""


@pytest.fixture(scope="module")
def cuts(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk_cut")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o",
                    str(d / "shim.so"), str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def band(g, nbr, nbc):
    """Last chunk of every block row's list, for a band that runs up and right; often far along one
    row."""
    hi = np.sort(g.integers(0, nbc, nbr))
    hi[g.integers(0, nbr + 1):] = nbc - 1     # along a row, then straight up
    u = g.random()
    if u < 0.3:
        hi[:] = nbc - 1                       # along row 0
    elif u < 0.6:
        hi[:] = hi // 4                       # straight up, then along the last row
    return hi.astype(np.int32)


def rows_of(cuts, pieces, n, nbr, nbc, hi):
    """First rows of the pieces, and the largest row whose record was looked at."""
    h, top = hi.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), ctypes.c_int(-1)
    rows = [cuts.cut_row(q, pieces, n, nbr, nbc, h, ctypes.byref(top)) for q in range(1, pieces)]
    return [0] + rows + [nbr], top.value


def blocks(n):
    return (n + 31) // 32


def test_first_piece_has_the_first_row(cuts):
    """Only the first piece enters the grid where a path does: however far the band runs along block
    row 0, that row stays with it, and no other piece looks at the row below the grid."""
    g = np.random.default_rng(1)
    along = 0
    for _ in range(3000):
        n, m = sorted((int(v) for v in g.integers(40, 9600, 2)), reverse=True)
        nbr, nbc, size = blocks(n - 1), blocks(m - 1), int(g.integers(1, 149))
        pieces = cuts.pieces_of(size, nbr, nbc)
        assert 1 <= pieces <= max(1, min(size, nbr // 2))
        hi = band(g, nbr, nbc)
        rows, _ = rows_of(cuts, pieces, n, nbr, nbc, hi)
        assert rows == sorted(rows) and rows[0] == 0 and rows[-1] == nbr
        assert all(1 <= r <= nbr for r in rows[1:])
        along += pieces > 1 and hi[0] >= (nbr + nbc) // pieces
    assert along > 300


def test_cuts_ask_only_for_rows_with_a_record(cuts):
    """The last block row of a grid has no record, and a DFD's last row is one that the VE-FD's
    and the decisions' grid can lack: no cut of either grid may depend on them."""
    g = np.random.default_rng(2)
    more = 0
    for _ in range(3000):
        n, m = sorted((int(v) for v in g.integers(130, 4000, 2)), reverse=True)
        if g.random() < 0.3:
            n = n // 32 * 32 + 1
            m = min(m, n)
        size = int(g.integers(2, 149))
        seg, dfd = (blocks(n - 1), blocks(m - 1)), (blocks(n), blocks(m))
        more += dfd[0] > seg[0]
        hi = np.append(band(g, *seg), 0).astype(np.int32)
        for nbr, nbc in (seg, dfd):
            pieces = cuts.pieces_of(size, nbr, nbc)
            rows, top = rows_of(cuts, pieces, n, nbr, nbc, hi)
            assert top <= seg[0] - 2
            for junk in (-2**31, 2**31 - 1):
                hi[seg[0] - 1:] = junk
                assert rows_of(cuts, pieces, n, nbr, nbc, hi)[0] == rows
            assert rows == sorted(rows) and all(0 < r < nbr for r in rows[1:-1])
    assert more > 300


def piece(cuts, cut, m, pieces, nbr):
    rows = (ctypes.c_int * 2)()
    cuts.piece(*cut, m, pieces, nbr, rows)
    return rows[0], rows[1]


def cut_of(cuts, m, pieces, n, nbr, nbc, hi):
    """walk_cut: what member m keeps of the cuts of a grid."""
    if m >= pieces:
        return (pieces, nbr, nbr)
    rows, _ = rows_of(cuts, pieces, n, nbr, nbc, hi)
    return (pieces, rows[m], rows[m + 1])


def tiles(parts, pieces, nbr):
    return ([a for a, _ in parts[:pieces]] == [0] + [b for _, b in parts[:pieces - 1]] and
            parts[pieces - 1][1] == nbr and all(a <= b for a, b in parts) and
            all(a == b for a, b in parts[pieces:]))


def test_pieces_of_sweeps_in_a_row_tile_the_grid(cuts):
    """VE-FD, DFD and decision sweeps of sizes that change the number of pieces between the kinds,
    as a group runs them: cuts kept from one sweep to the next, made again where the number of
    pieces differs; also cuts that are not made again (equal parts)."""
    g = np.random.default_rng(3)
    changed = 0
    sizes = [(609, 609), (1889, 1600), (2049, 2049), (20001, 19003), (1025, 850), (449, 449)]
    while len(sizes) < 2000:
        n = int(g.integers(130, 6000))
        n = n // 32 * 32 + 1 if g.random() < 0.5 else n
        sizes.append((n, int(g.integers(64, n + 1))))
    for n, m in sizes:
        size = int(g.choice([2, 5, 12, 32, 148, 296]))
        hi = band(g, blocks(n), blocks(m))
        state = [(0, 0, 0)] * size
        for kind in ("vefd", "dfd", "dfd", "vefd", "dec", "dec"):
            k = 0 if kind == "dfd" else 1
            nbr, nbc = blocks(n - k), blocks(m - k)
            pieces = cuts.pieces_of(size, nbr, nbc)
            stale = state[0][0] > 0 and state[0][0] != pieces
            changed += stale
            assert tiles([piece(cuts, state[q], q, pieces, nbr) for q in range(size)], pieces, nbr)
            if stale:
                state = [cut_of(cuts, q, pieces, n, nbr, nbc, hi) for q in range(size)]
            parts = [piece(cuts, state[q], q, pieces, nbr) for q in range(size)]
            assert tiles(parts, pieces, nbr)
            assert parts[0][1] > 0
            if pieces > 1 and g.random() < 0.8:  # the sweep found the band
                hi = band(g, blocks(n), blocks(m))
                state = [cut_of(cuts, q, pieces, n, nbr, nbc, hi) for q in range(size)]
    assert changed > 100


# ------------------------------------------------------------------ sweeps that share their records

class Member:
    cut, near = (0, 0, 0), None


def sweep(cuts, grid, members, records, b, n):
    """walk_sweep's rounds with the members' pieces (cut where an earlier sweep's band ran, starts only
    near it, pieces without rows left out); records: lo, hi of every block row as last walked."""
    dead, start0 = grid.dead, (grid.dead if grid.kind == "dfd" else 0.0)
    nbr, nbc = grid.nbr, -(-grid.cols // b)
    pieces = cuts.pieces_of(len(members), nbr, nbc)

    def hi():
        return np.array([r[1] if r else 2**30 for r in records], dtype=np.int32)

    def cut_all():
        for m, q in enumerate(members):
            q.cut = cut_of(cuts, m, pieces, n, nbr, nbc, hi())
            q.near = records[q.cut[1] - 1] if 0 < m < pieces else None
    if members[0].cut[0] not in (0, pieces):
        cut_all()
    part = [piece(cuts, q.cut, m, pieces, nbr) for m, q in enumerate(members)][:pieces]
    on = [m for m in range(pieces) if part[m][0] < part[m][1]]
    assert on[0] == 0 and part[on[-1]][1] == nbr

    def live(F):
        return np.nonzero(F < dead)[0] // b

    def note(i, F):
        if len(live(F)) and i + 1 < nbr:
            records[i] = (int(live(F)[0]), int(live(F)[-1]))
    recs, ends, res, lossy, empty = {}, {}, {}, {}, {}
    for m in on:
        i0, i1 = part[m]
        F = grid.bottom() if m == 0 else grid.everything(i0)
        lossy[m] = m > 0 and members[m].near is not None
        if lossy[m]:
            lo, up = members[m].near
            c = np.arange(grid.cols) // b
            F = np.where((c >= lo - 2) & (c <= up + 2), F, dead)
        end = dead
        for i in range(i0, i1):
            F, end = grid.walk(i, F, start0)
            recs[i] = F
            note(i, F)
            if not np.any(F < dead) and i + 1 < nbr:
                end = dead
                recs.update({k: None for k in range(i + 1, i1)})
                break
        ends[m], res[m], empty[m] = F, end, i1 < nbr and not np.any(F < dead)
    if empty[0] or any(empty[m] and not lossy[m] for m in on):
        return dead
    first = {m: (ends[m], res[m], empty[m]) for m in on}
    const, met = {m: 0.0 for m in on}, {m: True for m in on}
    changed = {m: True for m in on}
    while True:
        new = {m: False for m in on}
        old = dict(ends)
        for p, m in zip(on, on[1:]):
            if not changed[p]:
                continue
            F, c, hit, end = old[p], 0.0, False, dead
            for i in range(*part[m]):
                if not np.any(F < dead):
                    break
                F, end = grid.walk(i, F, start0)
                note(i, F)
                r = recs[i]
                if i + 1 < nbr and r is not None:
                    if grid.kind == "dec":
                        hit = np.array_equal(F, r)
                    else:
                        c = max([v for v, q in zip(F, r) if v != q], default=0.0)
                        hit = np.array_equal(F, np.maximum(c, r)) and \
                            np.array_equal(F < dead, r < dead)
                if hit:
                    break
            if hit:
                ends[m], res[m], empty[m] = first[m]
                const[m], new[m], met[m] = c, not met[m], True
            else:
                gone = part[m][1] < nbr and not np.any(F < dead)
                ends[m], res[m], empty[m] = F, dead if gone else end, gone
                const[m], new[m], met[m] = 0.0, True, False
        changed = new
        moved = [m for m in on if changed[m]]
        hollow = [m for m in on if empty[m]]
        if not moved or (hollow and hollow[0] <= moved[0]):
            break
    last = res[on[-1]]
    if hollow or not last < dead:
        return dead
    cut_all()
    return last if grid.kind == "dec" else max(max(const.values()), last)


@pytest.mark.parametrize("along", [False, True])
def test_sweeps_in_a_row_equal_serial_sweeps(cuts, along):
    """VE-FD, DFD and decisions of grids that follow the same path, blocks of two cells a side (so
    that small grids have pieces), records and cuts carried on: every result is the serial
    sweep's.  along: the path runs far along the first or the last block rows."""
    from tests.test_walk_rule import Grid

    class Small(Grid):
        def __init__(self, g, kind, rows, cols, path):
            super().__init__(g, kind, rows, cols, 2)
            p = np.clip(path[:rows], 0, cols - 1)
            low = np.concatenate([[0], p[:-1]])
            c = np.arange(cols)[None, :]
            far = np.maximum(np.maximum(low[:, None] - c, c - p[:, None]), 0)
            live = g.random((rows, cols))
            self.live_r = self.live_t = live < np.where(far == 0, 0.995, 0.6 / (1 + far))

    class Scaled:
        """The header's block of 32 cells against the model's of 2."""
        def __getattr__(self, name):
            return getattr(cuts, name)

        def cut_row(self, q, pieces, n, nbr, nbc, h, top):
            return cuts.cut_row(q, pieces, 32 * ((n - 1 + 1) // 2) + 1, nbr, nbc, h, top)
    g = np.random.default_rng(4 + along)
    alive = 0
    for _ in range(60):
        n, m = sorted((int(v) for v in g.integers(30, 90, 2)), reverse=True)
        n = n // 2 * 2 + 1 if g.random() < 0.6 else n
        path = np.sort(g.integers(0, m, n))
        if along:
            k = int(g.integers(1, n))
            path[k:] = m - 1
            if g.random() < 0.5:
                path = np.where(np.arange(n) < n - 1, 0, m - 1)
            elif g.random() < 0.5:
                path[:] = m - 1
        members, records = [Member() for _ in range(int(g.integers(2, 9)))], [None] * (n + 1)
        for kind in ("vefd", "dfd", "vefd", "dec", "dec"):
            k = 0 if kind == "dfd" else 1
            grid = Small(g, kind, n - k, m - k, path)
            F, want = grid.bottom(), grid.dead
            for i in range(grid.nbr):
                F, want = grid.walk(i, F, grid.dead if kind == "dfd" else 0.0)
                if not np.any(F < grid.dead) and i + 1 < grid.nbr:
                    want = grid.dead
                    break
            assert sweep(Scaled(), grid, members, records, 2, n) == want, (kind, n, m)
            alive += want < grid.dead
    assert alive > 60
