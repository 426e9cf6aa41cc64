"""The pieces of a walk's grid (rfd_walk_cut.h, compiled for the host): where the band of an earlier
sweep cuts the block rows among the members of a group."""
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
