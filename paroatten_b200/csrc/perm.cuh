// Decoder of the six (F,H,W) axis orders: maps a position in a head's reordered token
// sequence to the token it came from.  Order ids follow paroattention/cogvideox.py:38-45.
#pragma once
#include <cstdint>

namespace paro {

// Quotients by an extent of the grid, for dividends below 2^31: with p = 31 + ceil(log2 d) and m = ceil(2^p / d), which
// fits 32 bits, m * d exceeds 2^p by less than d, so j * m / 2^p exceeds j / d by less than 1 / d.  (Two instructions; a
// division by a run-time integer takes about twenty, and a row takes two of them.)
struct FastDiv {
  uint32_t m;
  int p, d;
};
inline FastDiv fast_div(int d) {
  int log2 = 0;
  while (log2 < 31 && (1u << log2) < (uint32_t)d) ++log2;
  const int p = 31 + log2;
  return FastDiv{(uint32_t)(((1ull << p) + (uint32_t)d - 1) / (uint32_t)d), p, d};
}
__device__ __forceinline__ int quotient(const FastDiv& f, int j) { return (int)(((uint64_t)(uint32_t)j * f.m) >> f.p); }

// The extents of the token grid.
struct GridDims {
  FastDiv f, y, x;
};
inline GridDims grid_dims(int F, int Hh, int W) { return GridDims{fast_div(F), fast_div(Hh), fast_div(W)}; }

struct PermDecoder {
  FastDiv div1, div2;      // of the middle and the fastest of the reordered axes
  int axis0, axis1, axis2; // which of (f, y, x) each reordered axis is, slowest first
  int Hh, W;

  __device__ PermDecoder(int order_id, const GridDims& g) : Hh(g.y.d), W(g.x.d) {
    // 0 FHW, 1 FWH, 2 HWF, 3 HFW, 4 WHF, 5 WFH: two bits per order, the middle and the fastest axis
    const int o = (order_id >= 0 && order_id < 6) ? order_id : 0;
    axis1 = (1 | 2 << 2 | 2 << 4 | 0 << 6 | 1 << 8 | 0 << 10) >> (2 * o) & 3;
    axis2 = (2 | 1 << 2 | 0 << 4 | 2 << 6 | 0 << 8 | 1 << 10) >> (2 * o) & 3;
    axis0 = 3 - axis1 - axis2;
    div1 = axis1 == 0 ? g.f : axis1 == 1 ? g.y : g.x;
    div2 = axis2 == 0 ? g.f : axis2 == 1 ? g.y : g.x;
  }

  // j: position among the reordered video tokens; returns the source token index and its
  // (f, y, x) grid coordinate.
  __device__ __forceinline__ int source(int j, int& f, int& y, int& x) const {
    const int t = quotient(div2, j), c2 = j - t * div2.d;
    const int c0 = quotient(div1, t), c1 = t - c0 * div1.d;
    f = axis0 == 0 ? c0 : axis1 == 0 ? c1 : c2;
    y = axis0 == 1 ? c0 : axis1 == 1 ? c1 : c2;
    x = axis0 == 2 ? c0 : axis1 == 2 ? c1 : c2;
    return (f * Hh + y) * W + x;
  }
};

}  // namespace paro
