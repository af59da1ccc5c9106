// Row form of the pull table: 36 bytes per node instead of 72.
//
// In the reference's node order the fluid nodes of one row of cells (fixed y,
// z) are numbered consecutively along x, so the sources of the directions
// with the same (e_y, e_z), the cells x - 1, x, x + 1 of one neighbouring
// row, are up to three consecutive nodes: one base index and a bit per cell
// give all three.  Per node nine words, [9][stride]:
//   word 0..3   base of the rows (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)
//   word 4..7   source of the directions 11..14 (one per diagonal row)
//   word 8      bit q - 1: the source cell of direction q is fluid (clear:
//               halfway bounce-back, the source is the node's own slot of
//               opp q); kRowLo / kRowHi: the sources at x - 1 (x + 1) do not
//               follow this form and are in the int32 table
// The own row's sources are p - 1 and p + 1.  A node's kRowLo, kRowHi mark
// the periodic wrap along x (2 of the nx cells of a row) and, with other
// node orders, whatever else does not follow: the builder checks every entry
// against the int32 table, so the form is right for any order and small
// enough to pay where few nodes are marked.
#pragma once

#include "lbm_internal.h"

namespace lbm {

constexpr uint32_t kRowLo = 1u << 18, kRowHi = 1u << 19;
// Direction of the source at x - 1 + c (c = 0, 1, 2) in neighbouring row r.
__host__ __device__ constexpr int row_dir(int r, int c) {
  return r == 0 ? (c == 0 ? 7 : c == 1 ? 3 : 8)
       : r == 1 ? (c == 0 ? 9 : c == 1 ? 4 : 10)
       : r == 2 ? (c == 0 ? 15 : c == 1 ? 5 : 16)
                : (c == 0 ? 17 : c == 1 ? 6 : 18);
}
__host__ __device__ constexpr bool row_dirs_ok() {
  for (int r = 0; r < 4; r++)
    for (int c = 0; c < 3; c++)
      if (cx(row_dir(r, c)) != 1 - c || cy(row_dir(r, c)) != cy(row_dir(r, 1)) ||
          cz(row_dir(r, c)) != cz(row_dir(r, 1)))
        return false;
  return cx(1) == 1 && cx(2) == -1;
}
static_assert(row_dirs_ok(), "row_dir lists the directions of a row from x - 1 to x + 1");

#ifdef __CUDACC__
// node(q, m, fluid) for q = 1..18: the source node m of direction q (any
// value when the source cell is solid) and whether it is fluid.  `words` are
// the nine words of node p; entries of marked nodes come from the int32
// table (flat indices q * stride + m).
template <typename F>
__device__ __forceinline__ void row_sources(const int32_t (&w)[9], const int32_t* __restrict__ table, int stride,
                                            int p, F&& node) {
  const uint32_t bits = (uint32_t)w[8];
  auto fluid = [&](int q) { return (bits >> (q - 1)) & 1u; };
  int32_t lo[5], hi[5];
  lo[4] = p - 1;
  hi[4] = p + 1;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int32_t mid = w[r] + (int32_t)fluid(row_dir(r, 0));
    node(row_dir(r, 1), mid, fluid(row_dir(r, 1)));
    lo[r] = w[r];
    hi[r] = mid + (int32_t)fluid(row_dir(r, 1));
  }
#pragma unroll
  for (int q = 11; q <= 14; q++) node(q, w[q - 7], fluid(q));
  if (bits & kRowLo) {
#pragma unroll
    for (int r = 0; r < 5; r++) {
      const int q = r < 4 ? row_dir(r, 0) : 1;
      lo[r] = __ldg(table + (size_t)(q - 1) * stride + p) - q * stride;
    }
  }
  if (bits & kRowHi) {
#pragma unroll
    for (int r = 0; r < 5; r++) {
      const int q = r < 4 ? row_dir(r, 2) : 2;
      hi[r] = __ldg(table + (size_t)(q - 1) * stride + p) - q * stride;
    }
  }
#pragma unroll
  for (int r = 0; r < 5; r++) {
    const int ql = r < 4 ? row_dir(r, 0) : 1, qh = r < 4 ? row_dir(r, 2) : 2;
    node(ql, lo[r], fluid(ql));
    node(qh, hi[r], fluid(qh));
  }
}
// The pull slots of node p with the words w: slot[q] = q * stride + m, or
// opp(q) * stride + p behind a wall.
__device__ __forceinline__ void row_slots(const int32_t (&w)[9], const int32_t* __restrict__ table, int stride, int p,
                                          int32_t (&slot)[kQ]) {
  row_sources(w, table, stride, p, [&](int q, int32_t m, uint32_t fluid) {
    slot[q] = fluid ? q * stride + m : opp(q) * stride + p;
  });
}
__device__ __forceinline__ void row_slots(const int32_t* __restrict__ rows, const int32_t* __restrict__ table,
                                          int stride, int p, int32_t (&slot)[kQ]) {
  int32_t w[9];
#pragma unroll
  for (int i = 0; i < 9; i++) w[i] = __ldg(rows + (size_t)i * stride + p);
  row_slots(w, table, stride, p, slot);
}
#endif

}  // namespace lbm
