// Index arithmetic of the Selector gather (gather_reduce.cu): which tile of
// rows and columns a CTA takes and what each of its threads loads and stores.
// Compiled for the host too, over pointer-like types that check every access.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define ESR_HD __host__ __device__ __forceinline__
#else
#define ESR_HD inline
#endif

namespace gather {

constexpr int kCols = 1024;  // vectors of one row a tile takes at most

// Local element -> (row, column) of a tile without a division: j / d for
// j < 2^16 and 1 <= d < 2^16 is umulhi(j, ceil(2^32 / d)) exactly (the
// rounding error of the quotient, j * (d - 1) / (d * 2^32), stays below 1/d).
struct FastDiv {
  uint32_t d, magic;
};

inline FastDiv fast_div(uint32_t d) { return FastDiv{d, d > 1 ? (uint32_t)((((uint64_t)1 << 32) + d - 1) / d) : 0u}; }

template <int D>
ESR_HD uint32_t div_by(uint32_t j, FastDiv f) {
  if (D > 0) return j / (uint32_t)(D > 0 ? D : 1);
#ifdef __CUDA_ARCH__
  return f.d > 1 ? __umulhi(j, f.magic) : j;
#else
  return f.d > 1 ? (uint32_t)(((uint64_t)j * f.magic) >> 32) : j;
#endif
}

// Columns and rows of a tile of about `vectors` vectors, of rows of `vpr`
// vectors (whole rows where a row has at most kCols).
inline int tile_width(int64_t vpr) { return (int)(vpr < kCols ? vpr : kCols); }
inline int tile_rows(int width, int vectors) { return width >= vectors ? 1 : vectors / width; }

template <class T>
ESR_HD T load_index(const T *p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}

// The part of thread `thread` of THREADS in tile (bx, by): y[row] = x[idx[row]].
// It requests U indices, then U vectors, THREADS apart, before it stores them.
// A row whose index is not below n_in is left alone; false if there was one.
// O: type of a vector's offset in x (32 bits where x is small enough).
template <class V, int D, int U, class O, int THREADS, class X, class I, class Y>
ESR_HD bool copy_part(X x, uint32_t n_in, O vpr, I idx, int64_t m, Y y, int rows_per_tile, FastDiv cols, int64_t col0,
                      uint32_t bx, uint32_t by, uint32_t thread) {
  const int64_t row0 = (int64_t)bx * rows_per_tile;
  const O c0 = D > 0 ? O(0) : (O)(col0 + (int64_t)by * kCols);
  const uint32_t rows = (uint32_t)(m - row0 < rows_per_tile ? m - row0 : rows_per_tile);
  const uint32_t width = D > 0 ? (uint32_t)D : (uint32_t)((int64_t)vpr - (int64_t)c0 < cols.d ? (int64_t)vpr - (int64_t)c0 : cols.d);
  const O row_len = D > 0 ? (O)D : vpr;
  const uint32_t count = rows * width;  // (a row cut into column blocks: one row a tile, no division)
  const bool cut = D == 0 && (int64_t)vpr > kCols;
  const I ti = idx + row0;
  const Y ty = y + (row0 * (int64_t)row_len + (int64_t)c0);
  bool ok = true;
  for (uint32_t j0 = thread; j0 < count; j0 += U * THREADS) {
    uint32_t s[U], c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t j = j0 + u * THREADS;
      const uint32_t r = cut ? 0u : div_by<D>(j, cols);
      c[u] = j - r * width;
      // (past the tile: no row, so nothing is loaded; its column may lie past
      // the end of x)
      s[u] = j < count ? (uint32_t)load_index(ti + r) : 0xffffffffu;
    }
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s[u] < n_in) v[u] = x[(O)s[u] * row_len + c0 + c[u]];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t j = j0 + u * THREADS;
      if (j < count) {
        if (s[u] < n_in) ty[j] = v[u];
        else ok = false;
      }
    }
  }
  return ok;
}

}  // namespace gather
