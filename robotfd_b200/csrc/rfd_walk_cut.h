// How the block rows of a walk's grid are shared out among the members of a group (rfd_walk.cuh),
// compiled for host and device.
#pragma once

#if defined(__CUDACC__)
#define RFD_WHD __host__ __device__ __forceinline__
#else
#define RFD_WHD inline
#endif

namespace rfd {

// The number of pieces of a grid of nbr x nbc blocks: at most `size`, of two block rows or more and
// of at least kWalkStretch blocks of a thin band (shorter ones end before the band has forgotten
// their start).
constexpr int kWalkStretch = 10;
constexpr int kWalkFew = 6;  // a grid of a few blocks: at most so many, rows and columns together
RFD_WHD int walk_pieces(int size, int nbr, int nbc) {
  int n = size < nbr / 2 ? size : nbr / 2;
  const int by_length = (nbr + nbc) / kWalkStretch;
  n = n < by_length ? n : by_length;
  return n > 1 ? n : 1;
}

// First block row of piece q (0 < q < pieces) where an earlier sweep's band ran: block row i ended
// about i + hi(i) blocks along it, and pieces take equal stretches, so piece q starts with the
// first row that ends past q / pieces of the way.  Row 0 stays with piece 0, which alone has the
// sweep's true start (a band that runs far along row 0 would leave it none), and the last row with
// the last piece: a grid's last row hands nothing on and has no record.  n: points of the longer
// curve; hi is asked for rows 1 .. (n - 1 + 31) / 32 - 2 only, which every kind of sweep that
// found a band has recorded (the DFD's grid can have a block row more than the others').
// (A larger q asks more of every row, so the bisection's rows are in order in q whatever hi holds.)
template <class Hi>
RFD_WHD int walk_cut_row(int q, int pieces, int n, int nbr, int nbc, Hi hi) {
  const long long want = (long long)(nbr + nbc) * q / pieces;
  int a = 1, b = ((n - 1 + 31) >> 5) - 1;
  while (a < b) {
    const int mid = (a + b) >> 1;
    if ((long long)mid + hi(mid) >= want) b = mid;
    else a = mid + 1;
  }
  return a;
}

// A member's cut: rows row0 .. row1 - 1 of a grid cut in `pieces` (0: not cut yet).  Every member has
// the same `pieces`, those past the last piece too.
struct WalkCut {
  int pieces, row0, row1;
};

// Block rows i0 .. i1 - 1 of piece m of a grid of nbr block rows (none for members past the last
// piece).  A cut holds for its own number of pieces only - the DFD's grid, a row and a column
// larger, can have one more than the VE-FD's - and otherwise all members take equal parts, so that
// the pieces of a sweep always tile the grid.
RFD_WHD void walk_piece(const WalkCut& c, int m, int pieces, int nbr, int* i0, int* i1) {
  if (m >= pieces) {
    *i0 = *i1 = nbr;
  } else if (pieces > 1 && c.pieces == pieces) {
    *i0 = c.row0;
    *i1 = m + 1 < pieces ? c.row1 : nbr;
  } else {
    *i0 = (int)((long long)nbr * m / pieces);
    *i1 = (int)((long long)nbr * (m + 1) / pieces);
  }
}

}  // namespace rfd
