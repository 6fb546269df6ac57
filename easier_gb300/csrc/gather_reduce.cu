// Selector gather, Reducer segmented reduce, aggregators and dot products.
//
// Everything here is deterministic: there are no floating-point atomics.
// Segmented reductions run one thread per row and walk the segment in
// ascending order, which is the order the reference's CPU scatter_reduce_
// accumulates in, so sums are bitwise equal to it.
#include <cmath>
#include <cstdint>
#include <mutex>

#include "esr_internal.h"
#include "gather_tile.cuh"
#include "reduce_util.cuh"
#include "soft64.cuh"

namespace {

constexpr int kThreads = 256;

using gather::div_by;
using gather::fast_div;
using gather::FastDiv;

// ---------------------------------------------------------------- gather --
// Bound: HBM, given enough loads in flight (index -> row is a chain of two
// dependent loads) and few enough instructions a vector.  A CTA takes a tile
// of whole rows (or of up to gather::kCols vectors of long rows, blockIdx.y) of
// about U * kThreads vectors; a thread requests U indices, then U row
// vectors, strided so that every store and index load is coalesced.  In a
// tile of whole rows vector j goes to offset j, and its (row, column) is a
// 16-bit division (FastDiv).  A 64-bit division per vector and one load in
// flight a thread, as before, took 59 us for 5.87 M rows of 12 bytes (this
// form 37, whole rows a thread as below 25: 4.7 TB/s of the bytes it must
// move).
template <typename V, int D, int U, typename O>
__global__ void __launch_bounds__(kThreads)
gather_kernel(const V *__restrict__ x, uint32_t n_in, O vpr, const int32_t *__restrict__ idx, int64_t m,
              V *__restrict__ y, int rows_per_tile, FastDiv cols, int64_t col0) {
  if (!gather::copy_part<V, D, U, O, kThreads>(x, n_in, vpr, idx, m, y, rows_per_tile, cols, col0, blockIdx.x,
                                               blockIdx.y, threadIdx.x))
    esr::raise_status(ESR_DEV_IDX_RANGE);
}

// Rows of D (3) vectors: a thread takes U whole rows, whose vectors go through
// shared memory to coalesced stores.  A third of the index work of the kernel
// above: 28 -> 25 us for 5.87 M rows of three floats.
template <typename V, int D, int U, typename O>
__global__ void __launch_bounds__(kThreads)
gather_rows_kernel(const V *__restrict__ x, uint32_t n_in, const int32_t *__restrict__ idx, int64_t m,
                   V *__restrict__ y) {
  __shared__ V s_row[kThreads * D];
  __shared__ uint8_t s_ok[kThreads];
  const int64_t row0 = (int64_t)blockIdx.x * (U * kThreads);
  uint32_t s[U];
  V v[U][D];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t e = row0 + u * kThreads + threadIdx.x;
    s[u] = e < m ? (uint32_t)__ldg(idx + e) : 0u;
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int c = 0; c < D; ++c)
      if (s[u] < n_in) v[u][c] = x[(O)s[u] * D + c];
  V *const warp_rows = s_row + (threadIdx.x & ~31) * D;
  uint8_t *const warp_ok = s_ok + (threadIdx.x & ~31);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < U; ++u) {  // each warp stages its own 32 rows
    const int64_t e0 = row0 + u * kThreads + (threadIdx.x & ~31);
    const bool here = e0 + lane < m, ok = here && s[u] < n_in;
    if (here && !ok) esr::raise_status(ESR_DEV_IDX_RANGE);
    __syncwarp();
    if (ok) {
#pragma unroll
      for (int c = 0; c < D; ++c) warp_rows[lane * D + c] = v[u][c];
    }
    warp_ok[lane] = ok;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const int j = lane + 32 * c;
      if (warp_ok[j / D]) y[e0 * D + j] = warp_rows[j];
    }
  }
}

template <typename V, int D, int U>
void launch_gather_rows(const V *x, int64_t n_in, const int32_t *idx, int64_t m, V *y, cudaStream_t st) {
  const unsigned g = (unsigned)((m + U * kThreads - 1) / (U * kThreads));
  const uint32_t nin = n_in > ((int64_t)1 << 31) ? (uint32_t)1 << 31 : (uint32_t)n_in;
  if (n_in * D < ((int64_t)1 << 31)) gather_rows_kernel<V, D, U, uint32_t><<<g, kThreads, 0, st>>>(x, nin, idx, m, y);
  else gather_rows_kernel<V, D, U, int64_t><<<g, kThreads, 0, st>>>(x, nin, idx, m, y);
}

template <typename V, int D, int U>
void launch_gather_u(const V *x, int64_t n_in, int64_t vpr, const int32_t *idx, int64_t m, V *y, cudaStream_t st) {
  const int width = gather::tile_width(vpr), rows = gather::tile_rows(width, U * kThreads);
  const int64_t gx = (m + rows - 1) / rows;
  // indices are int32: none of them reaches 2^31
  const uint32_t nin = n_in > ((int64_t)1 << 31) ? (uint32_t)1 << 31 : (uint32_t)n_in;
  for (int64_t c0 = 0; c0 < vpr; c0 += (int64_t)65535 * gather::kCols) {
    int64_t gy = (vpr - c0 + gather::kCols - 1) / gather::kCols;
    if (gy > 65535) gy = 65535;
    const dim3 g((unsigned)gx, (unsigned)gy);
    if (n_in * vpr < ((int64_t)1 << 31))
      gather_kernel<V, D, U, uint32_t><<<g, kThreads, 0, st>>>(x, nin, (uint32_t)vpr, idx, m, y, rows, fast_div(width), c0);
    else
      gather_kernel<V, D, U, int64_t><<<g, kThreads, 0, st>>>(x, nin, vpr, idx, m, y, rows, fast_div(width), c0);
  }
}

template <typename V>
int launch_gather(const void *x, int64_t n_in, int64_t row_bytes, const int32_t *idx, int64_t m, void *y,
                  cudaStream_t st) {
  const int64_t vpr = row_bytes / (int64_t)sizeof(V);
  const V *xv = (const V *)x;
  V *yv = (V *)y;
  // four vectors a thread once that still gives every SM eight CTAs
  const bool wide = m * vpr >= (int64_t)152 * 8 * 4 * kThreads;
  if (vpr == 1) {
    if (wide) launch_gather_u<V, 1, 4>(xv, n_in, vpr, idx, m, yv, st);
    else launch_gather_u<V, 1, 1>(xv, n_in, vpr, idx, m, yv, st);
  } else if (vpr == 3) {
    if (wide) launch_gather_rows<V, 3, 2>(xv, n_in, idx, m, yv, st);
    else launch_gather_rows<V, 3, 1>(xv, n_in, idx, m, yv, st);
  } else {
    if (wide) launch_gather_u<V, 0, 4>(xv, n_in, vpr, idx, m, yv, st);
    else launch_gather_u<V, 0, 1>(xv, n_in, vpr, idx, m, yv, st);
  }
  ESR_LAUNCH_CHECK("esr_gather");
  return ESR_OK;
}

// ----------------------------------------------------------- segreduce --
template <typename T>
__device__ __forceinline__ bool is_nan(T v) {
  return v != v;
}

// 0 + v without an add (the FP64 pipe is GB300's scarce one): v, with -0
// turned into +0
__device__ __forceinline__ double plus_zero(double v) {
  return __double_as_longlong(v) == (long long)0x8000000000000000ull ? 0.0 : v;
}
__device__ __forceinline__ float plus_zero(float v) { return __fadd_rn(0.f, v); }
__device__ __forceinline__ int32_t plus_zero(int32_t v) { return v; }
__device__ __forceinline__ int64_t plus_zero(int64_t v) { return v; }

template <typename T, int OP>
__device__ __forceinline__ T seg_combine(T acc, T v, bool first) {
  if (OP == ESR_REDUCE_SUM || OP == ESR_REDUCE_MEAN) return first ? plus_zero(v) : ops<T>::add(acc, v);
  if (OP == ESR_REDUCE_PROD) return first ? v : ops<T>::mul(acc, v);
  if (first || is_nan(v)) return v;
  if (OP == ESR_REDUCE_AMAX) return (acc < v) ? v : acc;
  return (v < acc) ? v : acc;
}

// The largest of the warp's values (a warp-uniform trip count: FP64
// instructions that are predicated off for every lane still take their pipe).
__device__ __forceinline__ int32_t warp_most(int32_t v) { return __reduce_max_sync(0xffffffffu, v); }

// One thread per row (of D columns, or of one of them), its entries in
// ascending order.  Bound: HBM, given enough loads in flight: a row is a chain
// row bounds -> perm -> value, so a thread requests R rows' bounds, then up to
// U positions of each, then their values, before it adds them in order;
// longer segments go on U entries at a time.  Load::entry(k) gives an entry's
// position, fetch() loads what lies there, follow() what that points to, value()
// turns it into the terms.
// Rows without entries reach the store with `none` set.  (Staging the entries
// through shared memory so that perm loads coalesce was slower: 131 us against
// 52 for a plain loop per (row, column) at 1.96 M rows of 3 entries x 3 FP32
// columns; a thread per row takes 24, 5.2 TB/s.)
// Every thread of the warp calls it.
template <typename T, int OP, int D, int U, int R, class Load, class Store>
__device__ __forceinline__ void seg_rows(const Load &load, const Store &store, const int32_t *__restrict__ rowptr,
                                         const int64_t (&row)[R], const int64_t (&col)[R], const bool (&mine)[R]) {
  int32_t b[R], e[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    b[q] = mine[q] ? __ldg(rowptr + row[q]) : 0;
    e[q] = mine[q] ? __ldg(rowptr + row[q] + 1) : 0;
  }
  typename Load::Held h[R][U];
  int32_t src[R][U];
#pragma unroll
  for (int q = 0; q < R; ++q)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < e[q] - b[q]) src[q][u] = load.entry(b[q] + u);
#pragma unroll
  for (int q = 0; q < R; ++q)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < e[q] - b[q]) load.fetch(src[q][u], col[q], h[q][u]);
#pragma unroll
  for (int q = 0; q < R; ++q)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < e[q] - b[q]) load.follow(h[q][u]);
#pragma unroll
  for (int q = 0; q < R; ++q) {
    T acc[D];
#pragma unroll
    for (int c = 0; c < D; ++c) acc[c] = T(0);
    const int32_t most = warp_most(e[q] - b[q]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= most) break;
      if (u < e[q] - b[q]) {
        T v[D];
        load.value(h[q][u], v);
#pragma unroll
        for (int c = 0; c < D; ++c) acc[c] = seg_combine<T, OP>(acc[c], v[c], u == 0);
      }
    }
    for (int32_t done = U; done < most; done += U) {
      const int32_t left = e[q] - b[q] - done;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < left) src[q][u] = load.entry(b[q] + done + u);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < left) load.fetch(src[q][u], col[q], h[q][u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u < left) load.follow(h[q][u]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u >= most - done) break;
        if (u < left) {
          T v[D];
          load.value(h[q][u], v);
#pragma unroll
          for (int c = 0; c < D; ++c) acc[c] = seg_combine<T, OP>(acc[c], v[c], false);
        }
      }
    }
    if (!mine[q]) continue;
    if (OP == ESR_REDUCE_MEAN && b[q] < e[q]) {
#pragma unroll
      for (int c = 0; c < D; ++c) acc[c] = ops<T>::div_count(acc[c], (int64_t)(e[q] - b[q]));
    }
    store(row[q], col[q], acc, b[q] >= e[q]);
  }
}

// t[perm[k], c .. c + D)
template <typename T, int D>
struct SegLoad {
  struct Held {
    T v[D];
  };
  const T *t;
  int64_t cols;
  const int32_t *perm;
  __device__ __forceinline__ int32_t entry(int32_t k) const { return perm ? __ldg(perm + k) : k; }
  __device__ __forceinline__ void fetch(int32_t src, int64_t c0, Held &h) const {
    const T *p = t + ((int64_t)src * (D > 1 ? (int64_t)D : cols) + c0);
#pragma unroll
    for (int c = 0; c < D; ++c) h.v[c] = __ldg(p + c);
  }
  __device__ __forceinline__ void follow(Held &) const {}
  __device__ __forceinline__ void value(const Held &h, T (&v)[D]) const {
#pragma unroll
    for (int c = 0; c < D; ++c) v[c] = h.v[c];
  }
};

template <typename T, int D>
struct SegStore {
  T *out;
  int64_t cols;
  bool fill;  // rows without entries get zero (otherwise they keep `out`)
  __device__ __forceinline__ void operator()(int64_t i, int64_t c0, const T (&acc)[D], bool none) const {
    T *p = out + (i * (D > 1 ? (int64_t)D : cols) + c0);
    if (!none || fill) {
#pragma unroll
      for (int c = 0; c < D; ++c) p[c] = acc[c];
    }
  }
};

// Narrow rows (1..4 columns): a thread takes R whole rows, kThreads apart.
template <typename T, int OP, int D, int R>
__global__ void __launch_bounds__(kThreads)
segreduce_kernel(const T *__restrict__ t, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ perm,
                 int64_t n, T *__restrict__ out, int fill) {
  int64_t row[R], col[R];
  bool mine[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    row[q] = ((int64_t)blockIdx.x * R + q) * kThreads + threadIdx.x;
    col[q] = 0;
    mine[q] = row[q] < n;
  }
  seg_rows<T, OP, D, 4, R>(SegLoad<T, D>{t, 1, perm}, SegStore<T, D>{out, 1, fill != 0}, rowptr, row, col, mine);
}

// Wider rows: a CTA takes `rows` consecutive rows times up to kThreads columns
// (blockIdx.y), a thread one (row, column).
template <typename T, int OP>
__global__ void __launch_bounds__(kThreads)
segreduce_cols_kernel(const T *__restrict__ t, int64_t cols, const int32_t *__restrict__ rowptr,
                      const int32_t *__restrict__ perm, int64_t n, T *__restrict__ out, int rows, FastDiv width,
                      int64_t col0, int fill) {
  const int64_t row0 = (int64_t)blockIdx.x * rows;
  const int64_t c0 = col0 + (int64_t)blockIdx.y * kThreads;
  const uint32_t w = (uint32_t)(cols - c0 < width.d ? cols - c0 : width.d);
  const uint32_t r = cols > kThreads ? 0u : div_by<0>(threadIdx.x, width), c = threadIdx.x - r * w;
  const int64_t row[1] = {row0 + r}, col[1] = {c0 + c};
  const bool mine[1] = {r < (uint32_t)rows && row0 + r < n && c < w};
  seg_rows<T, OP, 1, 4, 1>(SegLoad<T, 1>{t, cols, perm}, SegStore<T, 1>{out, cols, fill != 0}, rowptr, row, col, mine);
}

template <typename T, int OP, int D>
void launch_seg_rows(const T *t, const int32_t *rowptr, const int32_t *perm, int64_t n, T *out, int fill,
                     cudaStream_t st) {
  // two rows a thread once that still gives every SM eight CTAs
  if (n >= (int64_t)152 * 8 * 2 * kThreads)
    segreduce_kernel<T, OP, D, 2><<<(unsigned)((n + 2 * kThreads - 1) / (2 * kThreads)), kThreads, 0, st>>>(
        t, rowptr, perm, n, out, fill);
  else
    segreduce_kernel<T, OP, D, 1><<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st>>>(t, rowptr, perm, n,
                                                                                                  out, fill);
}

template <typename T, int OP>
void launch_seg_op(const T *t, int64_t cols, const int32_t *rowptr, const int32_t *perm, int64_t n, T *out, int fill,
                   cudaStream_t st) {
  switch (cols) {
    case 1: return launch_seg_rows<T, OP, 1>(t, rowptr, perm, n, out, fill, st);
    case 2: return launch_seg_rows<T, OP, 2>(t, rowptr, perm, n, out, fill, st);
    case 3: return launch_seg_rows<T, OP, 3>(t, rowptr, perm, n, out, fill, st);
    case 4: return launch_seg_rows<T, OP, 4>(t, rowptr, perm, n, out, fill, st);
    default: break;
  }
  const int width = (int)(cols < kThreads ? cols : kThreads);
  const int rows = kThreads / width;
  for (int64_t c0 = 0; c0 < cols; c0 += (int64_t)65535 * kThreads) {
    int64_t gy = (cols - c0 + kThreads - 1) / kThreads;
    if (gy > 65535) gy = 65535;
    segreduce_cols_kernel<T, OP><<<dim3((unsigned)((n + rows - 1) / rows), (unsigned)gy), kThreads, 0, st>>>(
        t, cols, rowptr, perm, n, out, rows, fast_div(width), c0, fill);
  }
}

template <typename T>
int launch_segreduce(int op, const void *t, int64_t cols, const int32_t *rowptr, const int32_t *perm,
                     int64_t n, void *out, cudaStream_t st) {
  const int fill = (op & ESR_REDUCE_FILL) ? 1 : 0;
  const T *tv = (const T *)t;
  T *ov = (T *)out;
  switch (op & ~ESR_REDUCE_FILL) {
    case ESR_REDUCE_SUM: launch_seg_op<T, ESR_REDUCE_SUM>(tv, cols, rowptr, perm, n, ov, fill, st); break;
    case ESR_REDUCE_PROD: launch_seg_op<T, ESR_REDUCE_PROD>(tv, cols, rowptr, perm, n, ov, fill, st); break;
    case ESR_REDUCE_MEAN: launch_seg_op<T, ESR_REDUCE_MEAN>(tv, cols, rowptr, perm, n, ov, fill, st); break;
    case ESR_REDUCE_AMAX: launch_seg_op<T, ESR_REDUCE_AMAX>(tv, cols, rowptr, perm, n, ov, fill, st); break;
    case ESR_REDUCE_AMIN: launch_seg_op<T, ESR_REDUCE_AMIN>(tv, cols, rowptr, perm, n, ov, fill, st); break;
    default:
      return esr::fail(ESR_ERR_ARG, "unknown reduce op");
  }
  ESR_LAUNCH_CHECK("esr_segreduce");
  return ESR_OK;
}

// -------------------------------------------------------------- linsys --
// y = reducer(selector(x) * Ae) + x * Av straight from the Selector's index
// and the Reducer's CSR, one pass instead of five through memory, with the
// same rounded operations in the same order (bitwise the five).  One thread
// a row, four entries' loads in flight, all of x's before the first product
// (the sum's branches hold loads back); bound in FP64 by latency and the FP64
// pipe together (two operations an entry, one a row: 72% busy), by HBM in FP32.
// 998,001-row P1 grid, FP64: 84 us as five steps; 35 with eight entries and x
// loaded product by product; 31 so.  The row's own product runs on the integer
// pipe; the entries' there too: 33.  Two rows a thread: 39.
__device__ __forceinline__ float linsys_product(float a, float b) { return ops<float>::mul(a, b); }
__device__ __forceinline__ double linsys_product(double a, double b) { return soft64::product(a, b); }

template <typename T>
struct LinsysLoad {
  struct Held {
    int32_t col;
    T ae, x;
  };
  const T *x, *ae;
  const int32_t *col, *perm;
  __device__ __forceinline__ int32_t entry(int32_t k) const { return perm ? __ldg(perm + k) : k; }
  __device__ __forceinline__ void fetch(int32_t src, int64_t, Held &h) const {
    h.col = __ldg(col + src);
    h.ae = __ldg(ae + src);
  }
  __device__ __forceinline__ void follow(Held &h) const { h.x = __ldg(x + h.col); }
  __device__ __forceinline__ void value(const Held &h, T (&v)[1]) const {
    v[0] = ops<T>::mul(h.x, h.ae);
  }
};

template <typename T>
struct LinsysStore {
  const T *x, *av;
  T *y;
  __device__ __forceinline__ void operator()(int64_t i, int64_t, const T (&acc)[1], bool) const {
    y[i] = ops<T>::add(acc[0], linsys_product(__ldg(x + i), __ldg(av + i)));
  }
};

template <typename T>
__global__ void __launch_bounds__(kThreads)
linsys_kernel(const T *__restrict__ x, const T *__restrict__ ae, const T *__restrict__ av,
              const int32_t *__restrict__ col, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ perm,
              int64_t n, T *__restrict__ y) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t row[1] = {i}, none[1] = {0};
  const bool mine[1] = {i < n};
  seg_rows<T, ESR_REDUCE_SUM, 1, 4, 1>(LinsysLoad<T>{x, ae, col, perm}, LinsysStore<T>{x, av, y}, rowptr, row, none,
                                       mine);
}

template <typename T>
int launch_linsys(const void *x, const void *ae, const void *av, const int32_t *col, const int32_t *rowptr,
                  const int32_t *perm, int64_t n, void *y, cudaStream_t st) {
  linsys_kernel<T><<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, st>>>(
      (const T *)x, (const T *)ae, (const T *)av, col, rowptr, perm, n, (T *)y);
  ESR_LAUNCH_CHECK("esr_linsys_apply");
  return ESR_OK;
}

// ---------------------------------------------------------- aggregate --
// Two launches (one for short inputs): blocks reduce strided parts into
// partials, then one block per column reduces the partials in block order.
// Bound: HBM / L2 for max and min, the FP64 pipe (one DADD or DFMA a value)
// for sums.  Extrema are taken on order-preserving integer keys: a double
// compare costs the FP64 pipe what an add does, integer compares run beside
// it.  A block covers kAggUnroll * W values at a time, W the largest multiple
// of `cols` up to kThreads, so a thread stays in one column of coalesced,
// independent loads.  8 M doubles: sum 31 -> 22 us, norm 48 -> 20, max 67 ->
// 16 (first launch, cold cache); the final launch's latency (6 us alone) is
// hidden in part by launching it early.
constexpr int kAggUnroll = 8;
constexpr int kAggMaxBlocks = 152 * 4;
constexpr int64_t kAggSingle = 8192;  // values one block takes alone: the second launch costs more

// acc_t A: load(T) -> A, combine(A, A), identity(), store(A) -> T
template <typename T, int AGG>
struct Agg;

template <typename A, int AGG>
struct AggSum {  // sum, prod, norm in A = double (floating T) or int64
  static __device__ __forceinline__ A identity() { return AGG == ESR_AGG_PROD ? A(1) : A(0); }
  static __device__ __forceinline__ A combine(A a, A b) {
    return AGG == ESR_AGG_PROD ? ops<A>::mul(a, b) : ops<A>::add(a, b);
  }
};

template <typename T, int AGG>
struct AggFloat : AggSum<double, AGG> {
  using A = double;
  static __device__ __forceinline__ A add(A a, T v) {
    if (AGG == ESR_AGG_NORM) return fma((double)v, (double)v, a);
    return AggSum<double, AGG>::combine(a, (double)v);
  }
  static __device__ __forceinline__ T store(A a) { return (T)(AGG == ESR_AGG_NORM ? sqrt(a) : a); }
};

// bits of a float / double -> signed integers in the values' order, every
// NaN at the end that wins (max: the top, min: the bottom)
template <typename I, typename U, int AGG>
struct AggKey {
  using A = I;
  static constexpr I kMag = (I)(~(U)0 >> 1);
  static constexpr I kLow = (I)((U)1 << (8 * sizeof(U) - 1));
  static constexpr I kWin = AGG == ESR_AGG_MAX ? kMag : kLow;
  static __device__ __forceinline__ I identity() { return AGG == ESR_AGG_MAX ? kLow : kMag; }
  static __device__ __forceinline__ I combine(I a, I b) {
    return AGG == ESR_AGG_MAX ? (a < b ? b : a) : (b < a ? b : a);
  }
  static __device__ __forceinline__ I key(I bits, U inf) {
    const I k = bits ^ ((bits >> (8 * sizeof(I) - 1)) & kMag);
    return ((U)bits << 1) > (inf << 1) ? kWin : k;
  }
  static __device__ __forceinline__ I bits(I k) { return k ^ ((k >> (8 * sizeof(I) - 1)) & kMag); }
};

template <int AGG>
struct AggExtF64 : AggKey<int64_t, uint64_t, AGG> {
  using K = AggKey<int64_t, uint64_t, AGG>;
  static __device__ __forceinline__ int64_t add(int64_t a, double v) {
    return K::combine(a, K::key(__double_as_longlong(v), 0x7ff0000000000000ull));
  }
  static __device__ __forceinline__ double store(int64_t k) { return __longlong_as_double(K::bits(k)); }
};

template <int AGG>
struct AggExtF32 : AggKey<int32_t, uint32_t, AGG> {
  using K = AggKey<int32_t, uint32_t, AGG>;
  static __device__ __forceinline__ int32_t add(int32_t a, float v) {
    return K::combine(a, K::key(__float_as_int(v), 0x7f800000u));
  }
  static __device__ __forceinline__ float store(int32_t k) { return __int_as_float(K::bits(k)); }
};

template <typename T, int AGG>
struct AggInt : AggSum<int64_t, AGG> {
  using A = int64_t;
  static __device__ __forceinline__ A add(A a, T v) { return AggSum<int64_t, AGG>::combine(a, (int64_t)v); }
  static __device__ __forceinline__ T store(A a) { return (T)a; }
};

template <typename T, int AGG>
struct AggIntExt : AggKey<int64_t, uint64_t, AGG> {
  static __device__ __forceinline__ int64_t add(int64_t a, T v) {
    return AggKey<int64_t, uint64_t, AGG>::combine(a, (int64_t)v);
  }
  static __device__ __forceinline__ T store(int64_t a) { return (T)a; }
};

constexpr bool is_ext(int agg) { return agg == ESR_AGG_MAX || agg == ESR_AGG_MIN; }
template <bool C, class X, class Y>
struct Pick { using type = X; };
template <class X, class Y>
struct Pick<false, X, Y> { using type = Y; };
template <int AGG>
struct Agg<float, AGG> : Pick<is_ext(AGG), AggExtF32<AGG>, AggFloat<float, AGG>>::type {};
template <int AGG>
struct Agg<double, AGG> : Pick<is_ext(AGG), AggExtF64<AGG>, AggFloat<double, AGG>>::type {};
template <int AGG>
struct Agg<int32_t, AGG> : Pick<is_ext(AGG), AggIntExt<int32_t, AGG>, AggInt<int32_t, AGG>>::type {};
template <int AGG>
struct Agg<int64_t, AGG> : Pick<is_ext(AGG), AggIntExt<int64_t, AGG>, AggInt<int64_t, AGG>>::type {};

// Combines the accumulators of threads t, t + w, t + 2w, ... < rows * w into
// thread t < w.  One column: the first warp adds eight values a lane, then
// shuffles (13 adds a block where a shuffle tree over eight warps issues 45;
// the FP64 pipe is the bound of sums).
template <class G>
__device__ __forceinline__ typename G::A agg_block(typename G::A acc, int rows, int w, typename G::A *s) {
  const int t = threadIdx.x;
  s[t] = acc;
  __syncthreads();
  if (w == 1) {
    if (t < 32) {
      for (int k = 32; k < kThreads; k += 32) acc = G::combine(acc, s[t + k]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc = G::combine(acc, __shfl_down_sync(0xffffffffu, acc, o));
    }
    return acc;
  }
  int top = 1;
  while (top < rows) top <<= 1;
  for (int h = top >> 1; h > 0; h >>= 1) {
    if (t < h * w && t + h * w < rows * w) s[t] = G::combine(s[t], s[t + h * w]);
    __syncthreads();
  }
  return s[t < w ? t : 0];
}

// blocks x columns: partial[b * cols + c]; a single block stores the result
template <typename T, int AGG>
__global__ void __launch_bounds__(kThreads, 4)
agg_partial_kernel(const T *__restrict__ t, int64_t n, int64_t cols, typename Agg<T, AGG>::A *__restrict__ partial,
                   T *__restrict__ out) {
  using G = Agg<T, AGG>;
  __shared__ typename G::A s[kThreads];
  cudaTriggerProgrammaticLaunchCompletion();  // the final launch may queue up; it waits for this grid's end
  typename G::A acc = G::identity();
  int rows = 1, w = kThreads;
  int64_t c = threadIdx.x;
  if (cols <= kThreads) {
    w = (int)cols;
    rows = kThreads / w;
    const int64_t W = (int64_t)rows * w, total = n * cols, step = (int64_t)gridDim.x * kAggUnroll * W;
    if ((int)threadIdx.x < W)
      for (int64_t base = (int64_t)blockIdx.x * kAggUnroll * W + threadIdx.x; base < total; base += step) {
        T v[kAggUnroll];
#pragma unroll
        for (int u = 0; u < kAggUnroll; ++u)
          if (base + u * W < total) v[u] = t[base + u * W];
#pragma unroll
        for (int u = 0; u < kAggUnroll; ++u)
          if (base + u * W < total) acc = G::add(acc, v[u]);
      }
  } else {  // wide rows: one column a thread, kThreads columns a block (blockIdx.y)
    c += (int64_t)blockIdx.y * kThreads;
    const int64_t step = (int64_t)gridDim.x * kAggUnroll;
    if (c < cols)
      for (int64_t r = (int64_t)blockIdx.x * kAggUnroll; r < n; r += step) {
        T v[kAggUnroll];
#pragma unroll
        for (int u = 0; u < kAggUnroll; ++u)
          if (r + u < n) v[u] = t[(r + u) * cols + c];
#pragma unroll
        for (int u = 0; u < kAggUnroll; ++u)
          if (r + u < n) acc = G::add(acc, v[u]);
      }
  }
  const typename G::A tot = agg_block<G>(acc, rows, w, s);
  if ((int)threadIdx.x >= w || c >= cols) return;
  // (empty input: sum and norm 0, prod 1; the host rejects empty max / min)
  if (gridDim.x == 1) out[c] = n > 0 || !is_ext(AGG) ? G::store(tot) : T(0);
  else partial[(int64_t)blockIdx.x * cols + c] = tot;
}

template <typename T, int AGG>
__global__ void __launch_bounds__(kThreads)
agg_final_kernel(const typename Agg<T, AGG>::A *__restrict__ partial, int nblocks, int64_t cols,
                 T *__restrict__ out) {
  using G = Agg<T, AGG>;
  __shared__ typename G::A s[kThreads];
  cudaGridDependencySynchronize();
  const int64_t c = blockIdx.x;
  typename G::A acc = G::identity();
#pragma unroll 4
  for (int b = threadIdx.x; b < nblocks; b += kThreads) acc = G::combine(acc, partial[b * cols + c]);
  const typename G::A tot = agg_block<G>(acc, kThreads, 1, s);
  if (threadIdx.x == 0) out[c] = G::store(tot);
}

// Scratch a call may be asked for by the static array's limit (one slot of
// 12 bytes per column and 8,192 rows, at most 1,024)
int64_t agg_limit_bytes(int64_t n, int64_t cols) {
  int64_t b = (n + 8191) / 8192;
  b = b < 1 ? 1 : b > 1024 ? 1024 : b;
  return b * (cols < 1 ? 1 : cols) * 12;
}

// Row blocks of the first launch: enough values each to pay for a block, at
// most four blocks an SM, and partials within ESR_AGG_NOALLOC_SCRATCH_BYTES
// or what the limit above already allows.
int64_t agg_blocks(int64_t n, int64_t cols) {
  if (cols < 1) cols = 1;
  if (n * cols <= kAggSingle) return 1;
  int64_t b;
  if (cols <= kThreads) {
    const int64_t per = (int64_t)kAggUnroll * (kThreads / cols) * cols;
    b = (n * cols + per - 1) / per;
  } else {
    b = (n + kAggUnroll - 1) / kAggUnroll;
    const int64_t fill = kAggMaxBlocks / ((cols + kThreads - 1) / kThreads);
    if (b > fill) b = fill;
  }
  if (b > kAggMaxBlocks) b = kAggMaxBlocks;
  int64_t room = (int64_t)ESR_AGG_NOALLOC_SCRATCH_BYTES;
  if (agg_limit_bytes(n, cols) > room) room = agg_limit_bytes(n, cols);
  if (b > room / (8 * cols)) b = room / (8 * cols);
  return b < 1 ? 1 : b;
}

template <typename T, int AGG>
int launch_agg_t(const void *t, int64_t n, int64_t cols, void *out, void *ws, cudaStream_t st) {
  using A = typename Agg<T, AGG>::A;
  const int64_t nb = agg_blocks(n, cols);
  const unsigned gy = cols <= kThreads ? 1u : (unsigned)((cols + kThreads - 1) / kThreads);
  A *partial = (A *)ws;
  agg_partial_kernel<T, AGG><<<dim3((unsigned)nb, gy), kThreads, 0, st>>>((const T *)t, n, cols, partial, (T *)out);
  ESR_LAUNCH_CHECK("esr_aggregate/partial");
  if (nb == 1) return ESR_OK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cols);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, agg_final_kernel<T, AGG>, (const A *)partial, (int)nb, cols, (T *)out);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate/final");
  return ESR_OK;
}

template <typename T>
int launch_agg(int agg, const void *t, int64_t n, int64_t cols, void *out, void *ws, cudaStream_t st) {
  switch (agg) {
    case ESR_AGG_SUM: return launch_agg_t<T, ESR_AGG_SUM>(t, n, cols, out, ws, st);
    case ESR_AGG_PROD: return launch_agg_t<T, ESR_AGG_PROD>(t, n, cols, out, ws, st);
    case ESR_AGG_NORM:
      if constexpr (sizeof(T) == 0 || T(0.5) == T(0)) return esr::fail(ESR_ERR_UNSUPPORTED, "norm of an integer tensor");
      else return launch_agg_t<T, ESR_AGG_NORM>(t, n, cols, out, ws, st);
    case ESR_AGG_MAX: return launch_agg_t<T, ESR_AGG_MAX>(t, n, cols, out, ws, st);
    case ESR_AGG_MIN: return launch_agg_t<T, ESR_AGG_MIN>(t, n, cols, out, ws, st);
    default: return esr::fail(ESR_ERR_ARG, "unknown aggregator");
  }
}

// ----------------------------------------------------------------- dot --
template <typename T>
__global__ void __launch_bounds__(kThreads)
dot_kernel(const T *__restrict__ a, const T *__restrict__ b, int64_t n, double *__restrict__ partial,
           unsigned int *__restrict__ counter, double *__restrict__ out) {
  double acc = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    acc = fma((double)a[i], (double)b[i], acc);
  __shared__ double s_red[kThreads / 32];
  double tot = esr::block_sum_fixed<kThreads>(acc, s_red);
  if (esr::last_block_done(tot, partial, counter)) {
    double v = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) v += __ldcg(partial + k);
    double all = esr::block_sum_fixed<kThreads>(v, s_red);
    if (threadIdx.x == 0) {
      *out = all;
      *counter = 0u;
    }
  }
}

constexpr int kDotMaxBlocks = 152 * 4;

int dot_blocks(int64_t n) {
  int64_t g = (n + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > kDotMaxBlocks) g = kDotMaxBlocks;
  return (int)g;
}

}  // namespace

ESR_DEFINE_STATUS_READER(esr_status_gather_reduce)

extern "C" int esr_gather(const void *x, int64_t n_in, int64_t row_bytes, const int32_t *idx, int64_t m,
                          void *y, void *stream) {
  if (m < 0 || n_in < 0 || row_bytes < 0) return esr::fail(ESR_ERR_ARG, "esr_gather: negative size");
  if (m == 0 || row_bytes == 0) return ESR_OK;
  if (!x || !idx || !y) return esr::fail(ESR_ERR_ARG, "esr_gather: null pointer");
  cudaStream_t st = esr::as_stream(stream);
  const uintptr_t al = (uintptr_t)x | (uintptr_t)y;
  if (row_bytes % 16 == 0 && al % 16 == 0) return launch_gather<uint4>(x, n_in, row_bytes, idx, m, y, st);
  if (row_bytes % 8 == 0 && al % 8 == 0) return launch_gather<uint2>(x, n_in, row_bytes, idx, m, y, st);
  if (row_bytes % 4 == 0 && al % 4 == 0) return launch_gather<uint32_t>(x, n_in, row_bytes, idx, m, y, st);
  return launch_gather<uint8_t>(x, n_in, row_bytes, idx, m, y, st);
}

extern "C" int esr_segreduce(int dtype, int op, const void *t, int64_t row_elems, const int32_t *rowptr,
                             const int32_t *perm, int64_t n, void *out, void *stream) {
  if (n < 0 || row_elems < 0) return esr::fail(ESR_ERR_ARG, "esr_segreduce: negative size");
  if (n == 0 || row_elems == 0) return ESR_OK;
  if (!rowptr || !out) return esr::fail(ESR_ERR_ARG, "esr_segreduce: null pointer");
  cudaStream_t st = esr::as_stream(stream);
  switch (dtype) {
    case ESR_F32: return launch_segreduce<float>(op, t, row_elems, rowptr, perm, n, out, st);
    case ESR_F64: return launch_segreduce<double>(op, t, row_elems, rowptr, perm, n, out, st);
    case ESR_I32: return launch_segreduce<int32_t>(op, t, row_elems, rowptr, perm, n, out, st);
    case ESR_I64: return launch_segreduce<int64_t>(op, t, row_elems, rowptr, perm, n, out, st);
    default: return esr::fail(ESR_ERR_UNSUPPORTED, "esr_segreduce: dtype");
  }
}

extern "C" int esr_linsys_apply(int dtype, const void *x, const void *ae, const void *av, const int32_t *col,
                                const int32_t *rowptr, const int32_t *perm, int64_t n, void *y, void *stream) {
  if (n < 0) return esr::fail(ESR_ERR_ARG, "esr_linsys_apply: negative size");
  if (n == 0) return ESR_OK;
  if (!x || !av || !rowptr || !y) return esr::fail(ESR_ERR_ARG, "esr_linsys_apply: null pointer");
  cudaStream_t st = esr::as_stream(stream);
  switch (dtype) {
    case ESR_F32: return launch_linsys<float>(x, ae, av, col, rowptr, perm, n, y, st);
    case ESR_F64: return launch_linsys<double>(x, ae, av, col, rowptr, perm, n, y, st);
    default: return esr::fail(ESR_ERR_UNSUPPORTED, "esr_linsys_apply: dtype");
  }
}

extern "C" int64_t esr_aggregate_workspace_bytes(int64_t n, int64_t cols) {
  if (n < 0 || cols < 0) return -1;
  const int64_t limit = agg_limit_bytes(n, cols), need = agg_blocks(n, cols) * (cols < 1 ? 1 : cols) * 8;
  return need > limit ? need : limit;
}

extern "C" int esr_aggregate(int dtype, int agg, const void *t, int64_t n, int64_t cols, void *out,
                             void *workspace, void *stream) {
  if (n < 0 || cols < 0) return esr::fail(ESR_ERR_ARG, "esr_aggregate: negative size");
  if (cols == 0) return ESR_OK;
  if (!out || !workspace || (n && !t)) return esr::fail(ESR_ERR_ARG, "esr_aggregate: null pointer");
  if (cols > 65535) return esr::fail(ESR_ERR_UNSUPPORTED, "esr_aggregate: too many columns");
  cudaStream_t st = esr::as_stream(stream);
  switch (dtype) {
    case ESR_F32: return launch_agg<float>(agg, t, n, cols, out, workspace, st);
    case ESR_F64: return launch_agg<double>(agg, t, n, cols, out, workspace, st);
    case ESR_I32:
      if (agg == ESR_AGG_NORM) return esr::fail(ESR_ERR_UNSUPPORTED, "norm of an integer tensor");
      return launch_agg<int32_t>(agg, t, n, cols, out, workspace, st);
    case ESR_I64:
      if (agg == ESR_AGG_NORM) return esr::fail(ESR_ERR_UNSUPPORTED, "norm of an integer tensor");
      return launch_agg<int64_t>(agg, t, n, cols, out, workspace, st);
    default: return esr::fail(ESR_ERR_UNSUPPORTED, "esr_aggregate: dtype");
  }
}

extern "C" int64_t esr_dot_workspace_bytes(int64_t n) {
  if (n < 0) return -1;
  return (int64_t)kDotMaxBlocks * sizeof(double) + 64;
}

extern "C" int esr_dot(int dtype, const void *a, const void *b, int64_t n, double *out_f64, void *workspace,
                       void *stream) {
  if (n < 0) return esr::fail(ESR_ERR_ARG, "esr_dot: negative size");
  if (!out_f64 || !workspace || (n && (!a || !b))) return esr::fail(ESR_ERR_ARG, "esr_dot: null pointer");
  cudaStream_t st = esr::as_stream(stream);
  double *partial = (double *)workspace;
  unsigned int *counter = (unsigned int *)((char *)workspace + kDotMaxBlocks * sizeof(double));
  const int g = dot_blocks(n);
  switch (dtype) {
    case ESR_F32:
      dot_kernel<float><<<g, kThreads, 0, st>>>((const float *)a, (const float *)b, n, partial, counter, out_f64);
      break;
    case ESR_F64:
      dot_kernel<double><<<g, kThreads, 0, st>>>((const double *)a, (const double *)b, n, partial, counter, out_f64);
      break;
    default: return esr::fail(ESR_ERR_UNSUPPORTED, "esr_dot: dtype");
  }
  ESR_LAUNCH_CHECK("esr_dot");
  return ESR_OK;
}

// ------------------------------------------------------ allocation-free --
// esr_aggregate_noalloc runs the same two launches as esr_aggregate, but its
// block partials live in the file-scope device array below instead of a
// workspace the caller allocates.  It exists for callers that cannot call
// cudaMalloc at the point where they need an aggregate: cudaMalloc/cudaFree
// synchronise the whole device (stalling every other stream of a time-step
// loop or solver), they can fail with out-of-memory in the middle of a run,
// and some host applications hand all device memory to their own pool and
// forbid libraries from allocating.  The array is a fixed 1 MiB per device
// that loaded this library, held until the process exits.
static __device__ __align__(256) unsigned char g_agg_noalloc_scratch[ESR_AGG_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kNoAllocMaxDevices = 64;
// The array's device address belongs to one CUDA context: the primary
// context of a device, recreated with a new address after cudaDeviceReset,
// or a context the caller created with the driver API.  It is cached per
// device together with the unique ID (cuCtxGetId) of the context it was
// looked up in, and looked up again whenever the current context's ID
// differs.
std::mutex g_noalloc_mu;
struct NoAllocAddr {
  unsigned long long ctx_id;
  void *addr;
};
NoAllocAddr g_noalloc_addr[kNoAllocMaxDevices];

using CtxGetCurrentFn = int (*)(void **);
using CtxGetIdFn = int (*)(void *, unsigned long long *);
CtxGetCurrentFn g_ctx_get_current;
CtxGetIdFn g_ctx_get_id;

// Driver entry points through the runtime (no link against libcuda).
cudaError_t noalloc_driver_fns() {
  if (g_ctx_get_current && g_ctx_get_id) return cudaSuccess;
  void *a = nullptr, *b = nullptr;
  cudaDriverEntryPointQueryResult qa, qb;
  cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &a, 12000, cudaEnableDefault, &qa);
  if (e != cudaSuccess) return e;
  e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &b, 12000, cudaEnableDefault, &qb);
  if (e != cudaSuccess) return e;
  if (qa != cudaDriverEntryPointSuccess || qb != cudaDriverEntryPointSuccess || !a || !b)
    return cudaErrorSymbolNotFound;
  g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(a);
  g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(b);
  return cudaSuccess;
}

// ID of the context current on this thread; 0 when there is none yet.
cudaError_t noalloc_ctx_id(unsigned long long *id) {
  *id = 0;
  void *ctx = nullptr;
  if (g_ctx_get_current(&ctx) != 0) return cudaErrorDeviceUninitialized;
  if (!ctx) return cudaSuccess;
  if (g_ctx_get_id(ctx, id) != 0) return cudaErrorDeviceUninitialized;
  return cudaSuccess;
}
}  // namespace

extern "C" int esr_aggregate_noalloc(int dtype, int agg, const void *t, int64_t n, int64_t cols, void *out,
                                     void *stream) {
  if (n < 0 || cols < 0) return esr::fail(ESR_ERR_ARG, "esr_aggregate_noalloc: negative size");
  if (cols == 0) return ESR_OK;
  if (!out || (n && !t)) return esr::fail(ESR_ERR_ARG, "esr_aggregate_noalloc: null pointer");
  const int64_t need = agg_limit_bytes(n, cols);
  if (need > (int64_t)ESR_AGG_NOALLOC_SCRATCH_BYTES)
    return esr::fail(ESR_ERR_ARG, "esr_aggregate_noalloc: n=" + std::to_string(n) + ", cols=" +
                                      std::to_string(cols) + " needs " + std::to_string(need) +
                                      " bytes of scratch, more than the " +
                                      std::to_string((long long)ESR_AGG_NOALLOC_SCRATCH_BYTES) +
                                      " bytes of the static array (any cols <= " +
                                      std::to_string(ESR_AGG_NOALLOC_MAX_COLS) +
                                      " fits); use esr_aggregate with a workspace");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate_noalloc/cudaGetDevice");
  if (dev < 0 || dev >= kNoAllocMaxDevices) return esr::fail(ESR_ERR_UNSUPPORTED, "esr_aggregate_noalloc: device ordinal");
  void *ws = nullptr;
  {
    // Set-up, on the first call in a context: look up the array's device
    // address (this may load the module, so it must not be the first call
    // inside a stream capture).
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    e = noalloc_driver_fns();
    if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate_noalloc/driver entry points");
    unsigned long long id = 0;
    e = noalloc_ctx_id(&id);
    if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate_noalloc/current context");
    NoAllocAddr &slot = g_noalloc_addr[dev];
    if (id == 0 || slot.addr == nullptr || slot.ctx_id != id) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, g_agg_noalloc_scratch);
      if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate_noalloc/cudaGetSymbolAddress");
      if (id == 0) {  // the lookup made the device's primary context current
        e = noalloc_ctx_id(&id);
        if (e != cudaSuccess) return esr::cuda_check(e, "esr_aggregate_noalloc/current context");
      }
      slot.ctx_id = id;
      slot.addr = p;
    }
    ws = slot.addr;
  }
  // Every partial slot the second launch reads is written by the first one,
  // so nothing needs clearing between calls.
  cudaStream_t st = esr::as_stream(stream);
  switch (dtype) {
    case ESR_F32: return launch_agg<float>(agg, t, n, cols, out, ws, st);
    case ESR_F64: return launch_agg<double>(agg, t, n, cols, out, ws, st);
    case ESR_I32:
      if (agg == ESR_AGG_NORM) return esr::fail(ESR_ERR_UNSUPPORTED, "norm of an integer tensor");
      return launch_agg<int32_t>(agg, t, n, cols, out, ws, st);
    case ESR_I64:
      if (agg == ESR_AGG_NORM) return esr::fail(ESR_ERR_UNSUPPORTED, "norm of an integer tensor");
      return launch_agg<int64_t>(agg, t, n, cols, out, ws, st);
    default: return esr::fail(ESR_ERR_UNSUPPORTED, "esr_aggregate_noalloc: dtype");
  }
}
