// Fused restarted GMRES on a SELL-32 Linsys, easier/numeric/solver/gmres.py.
//
// Restart cycles (gmres.py:235-261) on the device, in one cooperative launch
// (gm_cycle_kernel below) or, for systems that do not fit it, as a fixed
// sequence of launches (the host captures it in a CUDA graph):
//   initv       V_0 = r / ||r||
//   for j < restart:
//     matvec(j) V_j = w_prev / H[j][j-1] (j >= 1, written for own rows and
//               formed on the fly for gathered columns), w = A M V_j,
//               H[0][j] = V_0 . w
//     mgs(i, j) for i = 0..j: w -= H[i][j] V_i, then H[i+1][j] = V_{i+1} . w
//               (i < j) or H[j+1][j] = ||w|| (i == j): modified Gram-Schmidt
//               in the reference's order, each dot fused into the preceding
//               axpy's pass
//   lsq         y = argmin || ||r|| e_1 - H y || by Givens rotations (one
//               thread; the reference takes the SVD pseudo-inverse with
//               singular values clamped at 1e-8: the same y for a full-rank H)
//   updatex     x += M (V[:, :k] y)
//   residual    r = b - A x, ||r|| for the host's stopping test
// A breakdown (H[j+1][j] < 1e-15) ends the Arnoldi loop: the remaining
// matvec/mgs launches of the cycle see the flag and return.  Dots
// accumulate in FP64 per thread and are combined by the grid's last block
// in block order (deterministic).  V is column-contiguous: V_c = V + c*n.
#include <cmath>
#include <cstdint>

#include "esr_internal.h"
#include "grid_exchange.cuh"
#include "reduce_util.cuh"
#include "soft64.cuh"

namespace {

constexpr int kGmThreads = 256;
constexpr int kGmMaxBlocks = 1216;
constexpr int kGmMaxRestart = 64;

struct GmState {
  double rnorm, bnorm, tol, pad0;
  int32_t jend;    // Arnoldi columns of the current cycle
  int32_t broken;  // breakdown in the current cycle
  int32_t cycles;
  int32_t timed_out;  // a wait between CTAs gave up (any of them) since the init
  // (the host reads the fields above)
  double H[(kGmMaxRestart + 1) * kGmMaxRestart];  // [i][j] at i * kGmMaxRestart + j
  double y[kGmMaxRestart];
};

// many sums at once: sum i is added by CTA i % grid and posted back to all
constexpr int kGmMaxSums = kGmMaxRestart + 1;
struct GmComm {
  GridComm one;
  ulonglong2 part[kGmMaxSums][kSoloMaxCtas];   // [sum][from]
  ulonglong2 total[kSoloMaxCtas][kGmMaxSums];  // [to][sum]
};

struct GmWork {
  GmState s;
  unsigned int counter[4];
  double partial[kGmMaxBlocks];
  GmComm comm;
};

inline int grid_for(int64_t n) {
  int64_t g = (n + kGmThreads - 1) / kGmThreads;
  return (int)(g < 1 ? 1 : (g > kGmMaxBlocks ? kGmMaxBlocks : g));
}

// sum over the row's SELL slots of val * f(col), in slot order
template <typename T, class F>
__device__ __forceinline__ double gm_row(int64_t i, int64_t n, const int64_t *__restrict__ slice_ptr,
                                         const int32_t *__restrict__ col, const T *__restrict__ val, F f) {
  const int64_t s = i >> 5;
  const int lane = (int)(i & 31);
  const int64_t b = __ldg(slice_ptr + s);
  const int w = (int)((__ldg(slice_ptr + s + 1) - b) >> 5);
  double acc = 0.0;
  for (int k = 0; k < w; ++k) {
    const int64_t e = b + 32 * k + lane;
    const int32_t c = __ldg(col + e);
    if (c >= 0 && (int64_t)c < n) acc = fma((double)__ldg(val + e), f(c), acc);
  }
  return acc;
}

// block partial -> last block writes the grid total through `store`
template <class S>
__device__ __forceinline__ void gm_finish(double v, GmWork *w, S store) {
  __shared__ double s_red[kGmThreads / 32];
  const double bs = esr::block_sum_fixed<kGmThreads>(v, s_red);
  if (esr::last_block_done(bs, w->partial, &w->counter[0])) {
    double acc = 0.0;
    for (int q = threadIdx.x; q < (int)gridDim.x; q += kGmThreads) acc += __ldcg(w->partial + q);
    const double tot = esr::block_sum_fixed<kGmThreads>(acc, s_red);
    if (threadIdx.x == 0) {
      store(tot);
      w->counter[0] = 0u;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kGmThreads) gm_norm_kernel(int64_t n, const T *__restrict__ b, double rtol,
                                                             double atol, int has_atol, GmWork *w) {
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kGmThreads) {
    const double v = (double)b[i];
    acc = fma(v, v, acc);
  }
  gm_finish(acc, w, [&](double tot) {
    GmState &s = w->s;
    s.bnorm = sqrt(tot);
    double tol = rtol * s.bnorm;
    if (has_atol && atol > tol) tol = atol;
    s.tol = tol;
    s.cycles = 0;
  });
}

// r = b - A x; ||r||
template <typename T>
__global__ void __launch_bounds__(kGmThreads)
gm_resid_kernel(esr_sell A, const T *__restrict__ b, const T *__restrict__ x, T *__restrict__ r, GmWork *w) {
  const T *val = (const T *)A.val, *diag = (const T *)A.diag;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; i < A.n;
       i += (int64_t)gridDim.x * kGmThreads) {
    const double ax = fma((double)diag[i], (double)x[i],
                          gm_row<T>(i, A.n, A.slice_ptr, A.col, val, [&](int32_t c) { return (double)x[c]; }));
    const T ri = (T)((double)b[i] - ax);
    r[i] = ri;
    acc = fma((double)ri, (double)ri, acc);
  }
  gm_finish(acc, w, [&](double tot) {
    w->s.rnorm = sqrt(tot);
    w->s.broken = 0;
    w->s.jend = 0;
  });
}

template <typename T>
__global__ void __launch_bounds__(kGmThreads) gm_initv_kernel(int64_t n, const T *__restrict__ r, T *__restrict__ v0,
                                                              const GmWork *w) {
  const double rn = w->s.rnorm;
  const double inv = rn > 0.0 ? 1.0 / rn : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kGmThreads)
    v0[i] = (T)((double)r[i] * inv);
}

// V_j (j >= 1: from w_prev), w = A M V_j, H[0][j] = V_0 . w
template <typename T>
__global__ void __launch_bounds__(kGmThreads)
gm_matvec_kernel(esr_sell A, const T *__restrict__ invdiag, T *__restrict__ V, const T *__restrict__ w_prev,
                 T *__restrict__ w_out, int j, GmWork *w) {
  if (w->s.broken) return;
  const int64_t n = A.n;
  const T *val = (const T *)A.val, *diag = (const T *)A.diag;
  T *vj = V + (int64_t)j * n;
  const T *v0 = V;
  const double inv_h = j >= 1 ? 1.0 / w->s.H[j * kGmMaxRestart + (j - 1)] : 1.0;
  auto vcol = [&](int64_t c) -> double {  // V_j[c] without reading V_j
    return j >= 1 ? (double)(T)((double)w_prev[c] * inv_h) : (double)vj[c];
  };
  auto zcol = [&](int64_t c) -> double {  // (M V_j)[c]
    const double v = vcol(c);
    return invdiag ? (double)(T)(v * (double)invdiag[c]) : v;
  };
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kGmThreads) {
    if (j >= 1) vj[i] = (T)((double)w_prev[i] * inv_h);
    const double wi =
        fma((double)diag[i], zcol(i), gm_row<T>(i, n, A.slice_ptr, A.col, val, [&](int32_t c) { return zcol(c); }));
    const T wt = (T)wi;
    w_out[i] = wt;
    acc = fma((double)v0[i], (double)wt, acc);
  }
  gm_finish(acc, w, [&](double tot) { w->s.H[0 * kGmMaxRestart + j] = tot; });
}

// w -= H[i][j] V_i; then H[i+1][j] = V_{i+1} . w (i < j) or ||w|| (i == j)
template <typename T>
__global__ void __launch_bounds__(kGmThreads)
gm_mgs_kernel(int64_t n, const T *__restrict__ V, T *__restrict__ wv, int i, int j, int restart, GmWork *w) {
  if (w->s.broken) return;
  const double h = w->s.H[i * kGmMaxRestart + j];
  const T *vi = V + (int64_t)i * n;
  const T *vn = (i < j) ? V + (int64_t)(i + 1) * n : nullptr;
  double acc = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kGmThreads) {
    const T nw = (T)((double)wv[r] - h * (double)vi[r]);
    wv[r] = nw;
    acc = vn ? fma((double)vn[r], (double)nw, acc) : fma((double)nw, (double)nw, acc);
  }
  gm_finish(acc, w, [&](double tot) {
    GmState &s = w->s;
    if (i < j) {
      s.H[(i + 1) * kGmMaxRestart + j] = tot;
    } else {
      const double hn = sqrt(tot);
      s.H[(j + 1) * kGmMaxRestart + j] = hn;
      s.jend = j + 1;
      if (!(hn >= 1e-15)) s.broken = 1;
    }
  });
  (void)restart;
}

// y = argmin || rnorm e_1 - H[:k+1, :k] y ||, k = jend (one thread)
__global__ void gm_lsq_kernel(GmWork *w) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  GmState &s = w->s;
  const int k = s.jend;
  double R[(kGmMaxRestart + 1) * kGmMaxRestart];  // local copy, column j of row i at i*k + j
  double g[kGmMaxRestart + 1];
  for (int i = 0; i <= k; ++i) {
    g[i] = i == 0 ? s.rnorm : 0.0;
    for (int j = 0; j < k; ++j) R[i * kGmMaxRestart + j] = s.H[i * kGmMaxRestart + j];
  }
  for (int j = 0; j < k; ++j) {  // rotate rows j, j+1 to zero R[j+1][j]
    const double a = R[j * kGmMaxRestart + j], b = R[(j + 1) * kGmMaxRestart + j];
    const double rr = hypot(a, b);
    const double c = rr > 0.0 ? a / rr : 1.0, sn = rr > 0.0 ? b / rr : 0.0;
    for (int q = j; q < k; ++q) {
      const double u = R[j * kGmMaxRestart + q], v = R[(j + 1) * kGmMaxRestart + q];
      R[j * kGmMaxRestart + q] = c * u + sn * v;
      R[(j + 1) * kGmMaxRestart + q] = -sn * u + c * v;
    }
    const double u = g[j], v = g[j + 1];
    g[j] = c * u + sn * v;
    g[j + 1] = -sn * u + c * v;
  }
  for (int j = k - 1; j >= 0; --j) {  // back substitution; a zero pivot keeps y_j = 0
    double t = g[j];
    for (int q = j + 1; q < k; ++q) t -= R[j * kGmMaxRestart + q] * s.y[q];
    const double d = R[j * kGmMaxRestart + j];
    s.y[j] = fabs(d) > 1e-300 ? t / d : 0.0;
  }
  s.cycles += 1;
}

// x += M (sum_{c < k} y_c V_c)
template <typename T>
__global__ void __launch_bounds__(kGmThreads)
gm_updatex_kernel(int64_t n, const T *__restrict__ V, const T *__restrict__ invdiag, T *__restrict__ x,
                  const GmWork *w) {
  __shared__ double sy[kGmMaxRestart];
  const int k = w->s.jend;
  for (int c = threadIdx.x; c < k; c += kGmThreads) sy[c] = w->s.y[c];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * kGmThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kGmThreads) {
    double dx = 0.0;
    for (int c = 0; c < k; ++c) dx = fma((double)V[(int64_t)c * n + i], sy[c], dx);
    const T d = (T)dx;
    x[i] = (T)((double)x[i] + (invdiag ? (double)(T)((double)d * (double)invdiag[i]) : (double)d));
  }
}

// ---- restart cycles in one cooperative launch
//
// The launches above cost 5.7 us each at 40,000 rows (234 a cycle of 20) and
// read every basis vector four times.  Here a CTA per multiprocessor keeps its
// rows of w in shared memory and a step takes three exchanges
// (grid_exchange.cuh) whatever its number of basis vectors, by classical
// Gram-Schmidt applied twice (Giraud, Langou, Rozloznik, van den Eshof 2005:
// orthogonal to working precision, which modified Gram-Schmidt is not):
//   w = A M v_j; h = V^T w               -> exchange of j + 1 sums
//   w -= V h;    h' = V^T w, w.w         -> exchange of j + 2 sums
//   w -= V h';   w is published          -> barrier
// with ||w||^2 = w.w - h'.h' (the second pass removes little; where it does
// not, the norm is summed).  V is only read by the CTA that owns the rows, so
// it stays in shared memory too where it fits.
// An extra warp of every CTA reduces the Hessenberg columns by Givens rotations
// as they arrive, beside the next steps, and solves for y at the end; all CTAs
// hold the same sums, so none has to tell another.  Then x += M V y, which is
// published, and the next residual and its norm.
// 39,601 rows, GMRES(20): 1,340 -> 426 us a cycle.  Of a step's 38,000 cycles
// half are the two exchanges of many sums (two hops each: a CTA adds, then
// tells), a quarter the FP64 instructions of the two passes over V.
constexpr int kGmThreads2 = kSoloThreads + 32;
constexpr int kGmSmem = 200 * 1024;
constexpr int kGmSpins = 1 << 26;

struct GmShared : ExchangeShared {
  double h[kGmMaxSums];  // this exchange's sums
  double cs[kGmMaxRestart], sn[kGmMaxRestart], g[kGmMaxRestart + 1], inv[kGmMaxRestart], y[kGmMaxRestart];
  double scale, rnorm;
  int broken, again;
  // compute threads -> extra warp: cycles begun (-1: no more), columns posted, their final number; back: y is there
  volatile int cycle, ready, finished, solved;
};

// V^T w over the grid for columns 0 .. columns (and w.w if `square`): into
// sh.h, past a barrier.  V: the CTA's rows, columns `stride` apart.
template <typename T, int POLLS>
__device__ __forceinline__ bool many_dots(GmShared &sh, const T *V, int64_t stride, int rows, const double *ws,
                                          int columns, bool square, GmComm *comm, uint32_t epoch) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, grid = (int)gridDim.x, me = (int)blockIdx.x;
  constexpr int kWarps = kSoloThreads / 32;
  const int count = columns + (square ? 1 : 0);
  if (square && warp == kWarps - 1) {
    double a = 0.0;
    for (int l = lane; l < rows; l += 32) a = fma(ws[l], ws[l], a);
    a = warp_sum(a);
    if (lane == 0) post(&comm->part[columns][me], a, epoch);
  }
  const int pairs = columns > kWarps ? 2 : 1;  // sums a warp forms together
  for (int i = warp * pairs; i < columns; i += kWarps * pairs) {
    const bool two = pairs == 2 && i + 1 < columns;
    const T *v0 = V + i * stride, *v1 = v0 + (two ? stride : 0);
    double a0 = 0.0, a1 = 0.0;
    if (two) {
#pragma unroll 4
      for (int l = lane; l < rows; l += 32) {
        const double w = ws[l];
        a0 = fma((double)v0[l], w, a0);
        a1 = fma((double)v1[l], w, a1);
      }
      // lanes 0 .. 15 go on with sum i, the others with i + 1
      const double keep = lane < 16 ? a0 : a1, give = lane < 16 ? a1 : a0;
      a0 = keep + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    } else {
#pragma unroll 4
      for (int l = lane; l < rows; l += 32) a0 = fma((double)v0[l], ws[l], a0);
      a0 = warp_sum(a0);
    }
    if (lane == 0) post(&comm->part[i][me], a0, epoch);
    if (two && lane == 16) post(&comm->part[i + 1][me], a0, epoch);
  }
  // the sums this CTA adds: one a warp, from the last warp down
  for (int i = me + (kWarps - 1 - warp) * grid; i < count; i += kWarps * grid) {
    double v[kSoloMaxCtas / 32], b = 0.0;
    bool got = false;
    for (int tries = 0; tries < POLLS && !got; ++tries) {
      got = true;
#pragma unroll
      for (int q = 0; q < kSoloMaxCtas / 32; ++q) {
        v[q] = 0.0;
        if (lane + 32 * q < grid) {
          uint64_t x0, x1;
          asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x0), "=l"(x1)
                       : "l"(&comm->part[i][lane + 32 * q]) : "memory");
          got = got && (uint32_t)(x0 >> 32) == epoch && (uint32_t)(x1 >> 32) == epoch;
          v[q] = __longlong_as_double((long long)((x0 << 32) | (uint32_t)x1));
        }
      }
      got = __all_sync(0xffffffffu, got);
    }
    if (!got) sh.failed = 1;
#pragma unroll
    for (int q = 0; q < kSoloMaxCtas / 32; ++q)
      if (q * 32 < grid) b += v[q];
    b = __shfl_sync(0xffffffffu, warp_sum(b), 0);
    for (int to = lane; to < grid; to += 32) post(&comm->total[to][i], b, epoch);
  }
  if (t < count) {
    double h;
    if (!poll<POLLS>(&comm->total[me][t], true, false, epoch, h)) sh.failed = 1;
    sh.h[t] = h;
  }
  sync_part(0, kSoloThreads);
  return sh.failed == 0;
}

// w - sum_c h[c] V_c[i]
template <typename T>
__device__ __forceinline__ double minus_basis(double w, const T *V, int64_t n, int i, const double *h, int count) {
  const T *v = V + i;
  int c = 0;
  for (; c + 4 <= count; c += 4) {
    const double a = (double)v[(int64_t)c * n], b = (double)v[(int64_t)(c + 1) * n];
    const double d = (double)v[(int64_t)(c + 2) * n], e = (double)v[(int64_t)(c + 3) * n];
    w = fma(-h[c], a, w);
    w = fma(-h[c + 1], b, w);
    w = fma(-h[c + 2], d, w);
    w = fma(-h[c + 3], e, w);
  }
  for (; c < count; ++c) w = fma(-h[c], (double)v[(int64_t)c * n], w);
  return w;
}

// The extra warp, one cycle: columns R (column j at R + j * (restart + 1),
// entries 0 .. j + 1) are rotated in place as they arrive; then y.
__device__ __forceinline__ void least_squares(GmShared &sh, double *R, int restart) {
  const int lane = threadIdx.x & 31;
  int j = 0;
  while (j <= restart) {
    int there = 0;
    if (lane == 0) {
      for (int spin = 0; spin < kGmSpins; ++spin) {
        const int fin = sh.finished;  // (read before `ready`: its columns are posted)
        if (sh.ready > j) {
          there = 1;
          break;
        }
        if (fin == j) break;
        __nanosleep(50);
      }
      __threadfence_block();
    }
    there = __shfl_sync(0xffffffffu, there, 0);
    if (!there) break;
    if (lane == 0) {
      double *c = R + j * (restart + 1);
      double a = c[0];
#pragma unroll 4
      for (int i = 0; i < j; ++i) {  // earlier rotations
        const double b = c[i + 1], cs = sh.cs[i], sn = sh.sn[i];
        c[i] = fma(cs, a, sn * b);
        a = fma(-sn, a, cs * b);
      }
      const double b = c[j + 1], most = fmax(fabs(a), fabs(b));
      const double rho = most > 1e-140 && most < 1e140 ? sqrt(fma(a, a, b * b)) : hypot(a, b);
      const soft64::Divisor by_rho(rho);
      const double cs = rho > 0.0 ? soft64::quotient(a, by_rho) : 1.0;
      const double sn = rho > 0.0 ? soft64::quotient(b, by_rho) : 0.0;
      sh.cs[j] = cs;
      sh.sn[j] = sn;
      const double g = sh.g[j];
      sh.g[j] = cs * g;
      sh.g[j + 1] = -sn * g;
      sh.inv[j] = rho > 1e-300 ? soft64::quotient(1.0, by_rho) : 0.0;  // a zero pivot keeps y_j = 0
    }
    ++j;
  }
  __syncwarp();
  // back substitution, entries i and i + 32 in lane i
  double g0 = sh.g[lane], g1 = lane + 32 < kGmMaxRestart ? sh.g[lane + 32] : 0.0;
  for (int q = j - 1; q >= 0; --q) {
    const double y = __shfl_sync(0xffffffffu, q < 32 ? g0 : g1, q & 31) * sh.inv[q];
    const double *c = R + q * (restart + 1);
    if (lane < q) g0 = fma(-c[lane], y, g0);
    if (lane + 32 < q) g1 = fma(-c[lane + 32], y, g1);
    if (lane == 0) sh.y[q] = y;
  }
  __threadfence_block();
  __syncwarp();
  if (lane == 0) sh.solved = 1;
}

template <typename T, int POLLS>
__global__ void __launch_bounds__(kGmThreads2, 1)
gm_cycle_kernel(esr_sell A, const T *__restrict__ invdiag, const T *__restrict__ b, T *x, T *r, T *Vg, T *zs,
                int32_t restart, int32_t cap, int32_t on_chip, int32_t cycles, GmWork *work) {
  extern __shared__ double smem[];
  __shared__ GmShared sh;
  double *const ws = smem, *const R = smem + cap;
  const int64_t n = A.n, slices = (n + 31) >> 5;
  const int64_t s0 = slices * blockIdx.x / gridDim.x, s1 = slices * (blockIdx.x + 1) / gridDim.x;
  const int64_t row0 = s0 * 32;
  const int nsl = (int)(s1 - s0), rows = (int)((s1 * 32 < n ? s1 * 32 : n) - row0);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  // the basis: this CTA's rows of it, columns `stride` apart
  T *const V = on_chip ? reinterpret_cast<T *>(R + restart * (restart + 1)) : Vg + row0;
  const int64_t stride = on_chip ? cap : n;
  const T *val = (const T *)A.val, *diag = (const T *)A.diag;
  GmState &st = work->s;
  GmComm *comm = &work->comm;
  uint32_t epoch = comm->one.epoch;
  const double tol = st.tol;
  if (t == 0) {
    sh.failed = 0;
    sh.rnorm = st.rnorm;
    sh.cycle = 0;
  }
  __syncthreads();
  if (t >= kSoloThreads) {
    for (int c = 0; c < cycles; ++c) {
      int now = 0;
      for (int spin = 0; spin < kGmSpins && now >= 0 && now <= c; ++spin) {
        now = sh.cycle;
        if (now <= c) __nanosleep(50);
      }
      __threadfence_block();
      __syncwarp();
      if (now <= c) break;
      least_squares(sh, R, restart);
    }
    return;
  }
  int columns = 0, done = 0;
  bool ok = true;
  for (int cyc = 0; cyc < cycles; ++cyc) {
    if (t == 0) {
      const double rn = sh.rnorm;
      sh.broken = 0;
      sh.ready = 0;
      sh.finished = -1;
      sh.solved = 0;
      sh.g[0] = rn;
      sh.scale = rn > 0.0 ? soft64::quotient(1.0, soft64::Divisor(rn)) : 0.0;
      __threadfence_block();
      sh.cycle = cyc + 1;
    }
    sync_part(0, kSoloThreads);
    double scale = sh.scale;  // 1 / norm of the vector that v_j is formed from
    for (int j = 0; j < restart; ++j) {
      // v_j of the own rows; w = A M v_j.  FP64: zs holds M w of the step
      // before, v_j's scale is applied to the row's sum.  FP32: zs holds w, and
      // v_j and M v_j are rounded as stored.
      auto mv = [&](int32_t c) -> double {
        if constexpr (sizeof(T) == 8) {
          if (j > 0) return __ldcg(zs + c);
          const double v = __ldcg(r + c);
          return invdiag ? v * __ldg(invdiag + c) : v;
        } else {
          const T v = (T)((double)__ldcg((j > 0 ? zs : r) + c) * scale);
          return invdiag ? (double)(T)((double)v * (double)__ldg(invdiag + c)) : (double)v;
        }
      };
      for (int s = warp; s < nsl; s += kSoloThreads / 32) {
        const int l = s * 32 + lane;
        const int64_t i = row0 + l;
        const double sum = row_sum(s0 + s, lane, n, A.slice_ptr, A.col, val, mv);
        if (i < n) {
          const double own = j > 0 ? ws[l] : (double)__ldcg(r + i);
          V[j * stride + l] = (T)(own * scale);
          const double w = fma((double)__ldg(diag + i), mv((int32_t)i), sum);
          ws[l] = sizeof(T) == 8 ? w * scale : w;
        }
      }
      sync_part(0, kSoloThreads);
      if (!(ok = many_dots<T, POLLS>(sh, V, stride, rows, ws, j + 1, false, comm, ++epoch))) break;
      const double h1 = t <= j ? sh.h[t] : 0.0;
      for (int l = t; l < rows; l += kSoloThreads) ws[l] = minus_basis<T>(ws[l], V, stride, l, sh.h, j + 1);
      sync_part(0, kSoloThreads);
      if (!(ok = many_dots<T, POLLS>(sh, V, stride, rows, ws, j + 1, true, comm, ++epoch))) break;
      if (t <= j) R[j * (restart + 1) + t] = h1 + sh.h[t];
      if (warp == kSoloThreads / 32 - 1) {  // the norm, beside the other warps' rows
        double hh = lane <= j ? sh.h[lane] * sh.h[lane] : 0.0;
        if (lane + 32 <= j) hh = fma(sh.h[lane + 32], sh.h[lane + 32], hh);
        hh = warp_sum(hh);
        if (lane == 0) {
          const double ww = sh.h[j + 1], h2 = ww - hh;
          sh.again = h2 > 0.25 * ww ? 0 : 1;  // (also for NaN)
          const double hn = sqrt(h2);
          R[j * (restart + 1) + j + 1] = hn;
          sh.broken = hn >= 1e-15 ? 0 : 1;
          sh.scale = soft64::quotient(1.0, soft64::Divisor(hn));
        }
      }
      double v[1] = {0.0};
      for (int l = t; l < rows; l += kSoloThreads) {
        const double w = (double)(T)minus_basis<T>(ws[l], V, stride, l, sh.h, j + 1);
        ws[l] = w;
        v[0] = fma(w, w, v[0]);
        if (j + 1 < restart)
          __stcg(zs + row0 + l, sizeof(T) == 8 && invdiag ? (T)(w * (double)__ldg(invdiag + row0 + l)) : (T)w);
      }
      if (!(ok = publish<POLLS>(sh, &comm->one, ++epoch))) break;
      if (sh.again) {
        if (!(ok = exchange<1, false, POLLS>(sh, v, &comm->one, 0, ++epoch))) break;
        if (t == 0) {
          const double hn = sqrt(grid_sum(sh, 0));
          R[j * (restart + 1) + j + 1] = hn;
          sh.broken = hn >= 1e-15 ? 0 : 1;
          sh.scale = soft64::quotient(1.0, soft64::Divisor(hn));
        }
        sync_part(0, kSoloThreads);
      }
      if (t == 0) {
        __threadfence_block();
        sh.ready = j + 1;
      }
      scale = sh.scale;
      columns = j + 1;
      if (sh.broken) break;
    }
    if (t == 0) {
      sh.finished = ok ? columns : sh.ready;
      int solved = 0;
      for (int spin = 0; spin < kGmSpins && !solved; ++spin) solved = sh.solved;
      __threadfence_block();
      if (!solved) sh.failed = 1;
    }
    sync_part(0, kSoloThreads);
    ok = sh.failed == 0;
    if (!ok) break;
    for (int l = t; l < rows; l += kSoloThreads) {
      const int64_t i = row0 + l;
      const T d = (T)-minus_basis<T>(0.0, V, stride, l, sh.y, columns);
      x[i] = (T)((double)x[i] + (invdiag ? (double)(T)((double)d * (double)__ldg(invdiag + i)) : (double)d));
    }
    if (!(ok = publish<POLLS>(sh, &comm->one, ++epoch))) break;
    double rr[1] = {0.0};
    for (int s = warp; s < nsl; s += kSoloThreads / 32) {
      const int64_t i = row0 + s * 32 + lane;
      const double sum =
          row_sum(s0 + s, lane, n, A.slice_ptr, A.col, val, [&](int32_t c) { return (double)__ldcg(x + c); });
      if (i < n) {
        const T ri = (T)((double)__ldg(b + i) - fma((double)__ldg(diag + i), (double)__ldcg(x + i), sum));
        __stcg(r + i, ri);
        rr[0] = fma((double)ri, (double)ri, rr[0]);
      }
    }
    if (!(ok = exchange<1, true, POLLS>(sh, rr, &comm->one, 2, ++epoch))) break;
    if (t == 0) sh.rnorm = sqrt(grid_sum(sh, 0));
    ++done;
    sync_part(0, kSoloThreads);
    if (sh.rnorm <= tol) break;
  }
  if (t == 0) {
    sh.cycle = -1;
    if (!ok) {
      esr::raise_status(ESR_DEV_WAIT_TIMEOUT);
      atomicExch(&st.timed_out, 1);
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    st.rnorm = ok ? sh.rnorm : nan("");
    st.jend = columns;
    st.broken = sh.broken;
    st.cycles += done;
    comm->one.epoch = epoch;
  }
}

// CTAs of the one-launch cycle on the current device (0: it does not fit)
int cycle_ctas(int64_t n, int32_t restart, int *cap_out) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  if (n >= ((int64_t)1 << 31)) return 0;
  const int64_t slices = (n + 31) >> 5;
  int64_t g = (slices + 7) / 8;
  if (g > sms) g = sms;
  if (g > kSoloMaxCtas) g = kSoloMaxCtas;
  const int64_t cap = (slices + g - 1) / g * 32;
  if ((cap + (int64_t)restart * (restart + 1)) * 8 > kGmSmem) return 0;
  *cap_out = (int)cap;
  return (int)g;
}

template <typename T, int POLLS>
int run_coop(const esr_sell *A, const T *invdiag, const T *b, T *x, T *r, T *V, T *w2, int32_t restart, GmWork *w,
             int ctas, int cap, int32_t cycles, cudaStream_t s) {
  int smem = (cap + restart * (restart + 1)) * (int)sizeof(double);
  int32_t on_chip = smem + (int64_t)cap * restart * (int)sizeof(T) <= kGmSmem ? 1 : 0;
  if (on_chip) smem += cap * restart * (int)sizeof(T);
  const void *fn = (const void *)gm_cycle_kernel<T, POLLS>;
  // (the limit belongs to the function, not to this launch: always the largest,
  // or another thread's smaller system could lower it before this launch)
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGmSmem);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_gmres_cycle/smem attribute");
  esr_sell a = *A;
  void *args[] = {&a, &invdiag, &b, &x, &r, &V, &w2, &restart, &cap, &on_chip, &cycles, &w};
  e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)ctas), dim3(kGmThreads2), args, (size_t)smem, s);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_gmres_cycle");
  return ESR_OK;
}

int check(const esr_sell *A, int32_t restart) {
  if (!A || A->n <= 0) return esr::fail(ESR_ERR_ARG, "empty Linsys");
  if (A->dtype != ESR_F32 && A->dtype != ESR_F64) return esr::fail(ESR_ERR_UNSUPPORTED, "GMRES needs F32 or F64");
  if (restart < 1 || restart > kGmMaxRestart) return esr::fail(ESR_ERR_ARG, "restart must be in [1, 64]");
  if (!A->slice_ptr || !A->col || !A->val || !A->diag) return esr::fail(ESR_ERR_ARG, "null SELL array");
  return ESR_OK;
}

template <typename T, int POLLS>
int run_cycle(const esr_sell *A, const T *invdiag, const T *b, T *x, T *r, T *V, T *w2, int32_t restart,
              int32_t cycles, GmWork *w, cudaStream_t s) {
  const int64_t n = A->n;
  int cap = 0;
  if (const int ctas = cycle_ctas(n, restart, &cap))
    return run_coop<T, POLLS>(A, invdiag, b, x, r, V, w2, restart, w, ctas, cap, cycles, s);
  if (cycles != 1) return esr::fail(ESR_ERR_UNSUPPORTED, "several GMRES cycles a call need the one-launch cycle");
  const int g = grid_for(n);
  gm_initv_kernel<T><<<g, kGmThreads, 0, s>>>(n, r, V, w);
  for (int j = 0; j < restart; ++j) {
    T *wout = w2 + (int64_t)(j & 1) * n;
    const T *wprev = w2 + (int64_t)((j + 1) & 1) * n;
    gm_matvec_kernel<T><<<g, kGmThreads, 0, s>>>(*A, invdiag, V, wprev, wout, j, w);
    for (int i = 0; i <= j; ++i) gm_mgs_kernel<T><<<g, kGmThreads, 0, s>>>(n, V, wout, i, j, restart, w);
  }
  gm_lsq_kernel<<<1, 32, 0, s>>>(w);
  gm_updatex_kernel<T><<<g, kGmThreads, 0, s>>>(n, V, invdiag, x, w);
  gm_resid_kernel<T><<<g, kGmThreads, 0, s>>>(*A, b, x, r, w);
  ESR_LAUNCH_CHECK("esr_gmres_cycle");
  return ESR_OK;
}

template <int POLLS>
int run_cycles(const esr_sell *A, const void *invdiag, const void *b, void *x, void *r, void *V, void *w2,
               int32_t restart, int32_t cycles, void *workspace, void *stream) {
  int st = check(A, restart);
  if (st) return st;
  if (!b || !x || !r || !V || !w2 || !workspace) return esr::fail(ESR_ERR_ARG, "null vector");
  if (cycles < 1) return esr::fail(ESR_ERR_ARG, "cycles must be positive");
  cudaStream_t s = esr::as_stream(stream);
  GmWork *w = (GmWork *)workspace;
  if (A->dtype == ESR_F64)
    return run_cycle<double, POLLS>(A, (const double *)invdiag, (const double *)b, (double *)x, (double *)r, (double *)V,
                                    (double *)w2, restart, cycles, w, s);
  return run_cycle<float, POLLS>(A, (const float *)invdiag, (const float *)b, (float *)x, (float *)r, (float *)V,
                                 (float *)w2, restart, cycles, w, s);
}

}  // namespace

ESR_DEFINE_STATUS_READER(esr_status_gmres)

extern "C" int esr_gmres_one_launch(const esr_sell *A, int32_t restart) {
  int cap = 0;
  return check(A, restart) == ESR_OK && cycle_ctas(A->n, restart, &cap) > 0 ? 1 : 0;
}

extern "C" int64_t esr_gmres_workspace_bytes(int64_t n, int32_t restart) {
  if (n <= 0 || restart < 1 || restart > kGmMaxRestart) return -1;
  return (int64_t)sizeof(GmWork);
}

extern "C" int esr_gmres_init(const esr_sell *A, const void *b, double rtol, double atol, void *workspace,
                              void *stream) {
  int st = check(A, 1);
  if (st) return st;
  if (!b || !workspace) return esr::fail(ESR_ERR_ARG, "null vector");
  cudaStream_t s = esr::as_stream(stream);
  cudaError_t e = cudaMemsetAsync(workspace, 0, sizeof(GmWork), s);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_gmres_init/memset");
  GmWork *w = (GmWork *)workspace;
  const int g = grid_for(A->n);
  if (A->dtype == ESR_F64)
    gm_norm_kernel<double><<<g, kGmThreads, 0, s>>>(A->n, (const double *)b, rtol, atol, atol > 0.0, w);
  else
    gm_norm_kernel<float><<<g, kGmThreads, 0, s>>>(A->n, (const float *)b, rtol, atol, atol > 0.0, w);
  ESR_LAUNCH_CHECK("esr_gmres_init");
  return ESR_OK;
}

extern "C" int esr_gmres_residual(const esr_sell *A, const void *b, const void *x, void *r, void *workspace,
                                  void *stream) {
  int st = check(A, 1);
  if (st) return st;
  if (!b || !x || !r || !workspace) return esr::fail(ESR_ERR_ARG, "null vector");
  cudaStream_t s = esr::as_stream(stream);
  GmWork *w = (GmWork *)workspace;
  const int g = grid_for(A->n);
  if (A->dtype == ESR_F64)
    gm_resid_kernel<double><<<g, kGmThreads, 0, s>>>(*A, (const double *)b, (const double *)x, (double *)r, w);
  else
    gm_resid_kernel<float><<<g, kGmThreads, 0, s>>>(*A, (const float *)b, (const float *)x, (float *)r, w);
  ESR_LAUNCH_CHECK("esr_gmres_residual");
  return ESR_OK;
}

extern "C" int esr_gmres_cycles(const esr_sell *A, const void *invdiag, const void *b, void *x, void *r, void *V,
                                void *w2, int32_t restart, int32_t cycles, void *workspace, void *stream) {
  return run_cycles<kSoloPolls>(A, invdiag, b, x, r, V, w2, restart, cycles, workspace, stream);
}

extern "C" int esr_gmres_cycles_timeout(const esr_sell *A, const void *invdiag, const void *b, void *x, void *r,
                                        void *V, void *w2, int32_t restart, int32_t cycles, void *workspace,
                                        void *stream) {
  return run_cycles<0>(A, invdiag, b, x, r, V, w2, restart, cycles, workspace, stream);
}

extern "C" int esr_gmres_cycle(const esr_sell *A, const void *invdiag, const void *b, void *x, void *r, void *V,
                               void *w2, int32_t restart, void *workspace, void *stream) {
  return esr_gmres_cycles(A, invdiag, b, x, r, V, w2, restart, 1, workspace, stream);
}

extern "C" int esr_gmres_read(const void *workspace, esr_gmres_scalars *out, void *stream) {
  if (!workspace || !out) return esr::fail(ESR_ERR_ARG, "null argument");
  cudaStream_t s = esr::as_stream(stream);
  const GmWork *w = (const GmWork *)workspace;
  struct {
    double rnorm, bnorm, tol, pad0;
    int32_t jend, broken, cycles, timed_out;
  } h;  // the head of GmState
  cudaError_t e = cudaMemcpyAsync(&h, &w->s, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_gmres_read");
  out->rnorm = h.rnorm;
  out->bnorm = h.bnorm;
  out->tol = h.tol;
  out->jend = h.jend;
  out->broken = h.timed_out ? 2 : h.broken;
  out->cycles = h.cycles;
  out->pad_ = 0;
  return ESR_OK;
}
