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

}  // namespace rfd
