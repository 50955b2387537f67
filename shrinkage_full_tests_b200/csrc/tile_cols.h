// tile_cols.h — which columns of an image a group of four lines reads.
// Plain C++ (no CUDA types), so that the ranges can be checked on the host.
#pragma once

#ifdef __CUDACC__
#define SRK_HD __host__ __device__
#else
#define SRK_HD
#endif

namespace srk {

// Columns [lo, hi) of a staged window.
struct ColSpan {
  int lo, hi;
};

// The window of a group whose lines are the tile columns xg .. xg + 3 starts
// `halo` columns before xg (1: central differences, 0: cotangents).  Outputs
// are valid for the tile columns [e, e + S) only, and a group's first and last
// lines may lie outside them (its blocks of four start at a multiple of four).
// The columns that only those lines would read are left out: the buffer of a
// column slab ends with the columns that its valid outputs need.
SRK_HD constexpr ColSpan window_span(int xg, int e, int S, int halo) {
  const int first = xg > e ? xg : e;                    // first and one past the last valid line
  const int last = xg + 4 < e + S ? xg + 4 : e + S;
  return ColSpan{first - xg, last - xg + 2 * halo};
}

// Window columns [lo, hi) of `need` that lie in an image of N columns, window
// column 0 being the image column gx0.  Empty: lo == hi.
SRK_HD constexpr ColSpan clip_span(ColSpan need, int gx0, int N) {
  const int in0 = need.lo > -gx0 ? need.lo : -gx0;
  const int lo = in0 < need.hi ? in0 : need.hi;
  const int in1 = need.hi < N - gx0 ? need.hi : N - gx0;
  return ColSpan{lo, in1 > lo ? in1 : lo};
}

}  // namespace srk
