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
extern "C" int cut_row(int q, int pieces, int nbr, int nbc, const int* hi) {
  return rfd::walk_cut_row(q, pieces, nbr, nbc, [&](int i) { return hi[i]; });
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
    if g.random() < 0.3:
        hi[:] = nbc - 1                       # along row 0
    return hi.astype(np.int32)


def rows_of(cuts, pieces, nbr, nbc, hi):
    h = hi.ctypes.data_as(ctypes.POINTER(ctypes.c_int))
    return [0] + [cuts.cut_row(q, pieces, nbr, nbc, h) for q in range(1, pieces)] + [nbr]


def test_first_piece_has_the_first_row(cuts):
    """Only the first piece enters the grid where a path does: however far the band runs along block
    row 0, that row stays with it, and no other piece looks at the row below the grid."""
    g = np.random.default_rng(1)
    along = 0
    for _ in range(3000):
        nbr, nbc, size = int(g.integers(2, 300)), int(g.integers(1, 300)), int(g.integers(1, 149))
        if nbr < nbc:
            nbr, nbc = nbc, nbr
        pieces = cuts.pieces_of(size, nbr, nbc)
        assert 1 <= pieces <= max(1, min(size, nbr // 2))
        hi = band(g, nbr, nbc)
        rows = rows_of(cuts, pieces, nbr, nbc, hi)
        assert rows == sorted(rows) and rows[0] == 0 and rows[-1] == nbr
        assert all(1 <= r <= nbr for r in rows[1:])
        along += pieces > 1 and hi[0] >= (nbr + nbc) // pieces
    assert along > 300
