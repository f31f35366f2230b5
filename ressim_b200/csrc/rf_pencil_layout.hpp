// rf_pencil_layout.hpp — memory layout of the pressure solve along grid lines (rf_pencil.cu): how the
// columns are split over a cluster's CTAs, the step order's rows, and one CTA's shared memory.  Host
// and device code share these definitions; the CPU tests compile them with g++.
#pragma once

#include <cstddef>

#ifdef __CUDACC__
#define RF_PEN_HD __host__ __device__
#else
#define RF_PEN_HD
#endif

namespace rf {

constexpr int kPenChunk = 8;  // steps copied at a time (4 or 2 where 8 do not fit)
constexpr int kPenGuard = 2;  // zero rows before and after a CTA's steps

RF_PEN_HD constexpr size_t pen_up16(size_t b) { return (b + 15) / 16 * 16; }
RF_PEN_HD inline int pen_first_col(int c, int cs, int ny) {
  return int(unsigned(c) * unsigned(ny) / unsigned(cs));
}
RF_PEN_HD inline int pen_steps(int nx, int jc, int nz) { return nx + jc + nz - 2; }
// A step's rows: the lines rounded up to four, so that every row starts on a 16-byte boundary.
RF_PEN_HD constexpr int pen_stride(int lines) { return (lines + 3) / 4 * 4; }
// Bytes of one ring place: records, inputs (forward: right-hand side, backward: y), reciprocals.
template <class T>
RF_PEN_HD constexpr unsigned pen_place(int stride) {
  return unsigned(stride) * (5u * unsigned(sizeof(T)) + 8u);
}
// Steps of a sweep, whole chunks.
RF_PEN_HD inline int pen_rounded(int steps, int chunk) { return (steps + chunk - 1) / chunk * chunk; }

// Shared memory of one CTA (byte offsets); `wells` listed rows with `entries` entries.
struct PenLayout {
  size_t place, rows, ghost, nbr, mbar, full, red, bad, well_in, well_y, well_x, at, slot, ptr, piv, code, val, total;
};
template <class T>
RF_PEN_HD inline PenLayout pen_layout(int nx, int nz, int cols, int cs, int chunk, int nvw, int wells, int entries) {
  PenLayout o;
  size_t p = 0;
  auto take = [&](size_t bytes) {
    const size_t at = p;
    p += pen_up16(bytes);
    return at;
  };
  const int stride = pen_stride(cols * nz);
  o.place = take(2 * size_t(chunk) * pen_place<T>(stride));          // two chunks of copied rows
  o.rows = take(2 * size_t(chunk) * size_t(stride) * sizeof(T));     // two chunks of results
  o.ghost = take((2 * size_t(nz) + 1) * sizeof(T));                  // the neighbouring CTA's column, twice; a zero
  o.nbr = take(cs > 1 ? size_t(nx + nz - 1) * nz * sizeof(T) : 0);
  o.mbar = take(cs > 1 ? 2 * size_t(nx + nz - 1) * 8 : 0);
  o.full = take(2 * 8);
  o.red = take(4 * size_t(nvw) * sizeof(double));
  o.bad = take(2 * sizeof(int));  // two flags, read together
  // The places above are the same in every CTA of a cluster: CTAs store to one another's by their own
  // offsets (nbr, mbar, red, bad).  Below, each CTA's own wells.
  o.well_in = take(size_t(wells) * sizeof(T));
  o.well_y = take(size_t(wells) * sizeof(T));
  o.well_x = take(size_t(wells) * sizeof(T));
  o.piv = take(size_t(wells) * sizeof(T));
  o.at = take(size_t(wells) * 2 * sizeof(int));
  o.slot = take(size_t(wells) * sizeof(int));
  o.ptr = take(2 * (size_t(wells) + 1) * sizeof(int));
  o.val = take(size_t(entries) * sizeof(T));
  o.code = take(size_t(entries) * sizeof(unsigned short));
  o.total = p;
  return o;
}

}  // namespace rf
