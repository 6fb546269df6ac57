// (P)CG of one FP64 system with its vectors on the chip: one cooperative
// launch runs many iterations (the batched engine's state, scalars and
// stopping test, bcg.cu; Jacobi or no preconditioner).
//
// Bound of the three-launch iteration it replaces: at 40,000 rows launch and
// grid-tail latency (20 us an iteration for 0.8 us of FP64 work a
// multiprocessor), at 1 M rows the FP64 pipe, a third of it spent on block
// sums (45 adds a 256-thread block) and on predicated-off multiply-adds of
// narrow rows.  Here every multiprocessor keeps x, r, p and q of its rows in
// shared memory (32 bytes a row, up to 7,000 rows) for the whole launch, the
// matrix streams from L2, and only z goes through memory.  An iteration has
// two grid exchanges instead of three launches:
//   p = z + beta p, q = A z + beta q   (A p_new = A z + beta A p_old, as
//                                       bcg_pq_kernel); p.q   -> exchange
//   x += alpha p, r -= alpha q, z = M r; r.r, r.z             -> exchange
// The second exchange also publishes z.
// Measured: FV Poisson, 40,000 rows, 682 iterations 14.1 -> 5.8 ms; P1 grid,
// 998,001 rows, 2,720 iterations 153 -> 84 ms (31 us an iteration, 23 of them
// the two sweeps' FP64 instructions; z = M r takes its product to the integer
// pipes, soft64.cuh).  Between the two the sweeps' and the exchanges' shares
// trade places; below them only latency is left: about 1,500 cycles from a
// post to its poll, 700 for the sums of a CTA, 800 for a scalar division.
//
// Exchange: a CTA posts its block sum to every CTA's mailbox, as two 64-bit
// words that each hold 32 bits of the double and the exchange's number; every
// CTA polls its own mailbox and adds the sums itself in the same order, so all
// take the same decisions and no second barrier distributes the result.  That
// its z is stored a CTA tells with a word of its own, posted by other warps
// behind a fence while the sums are added.  (One set of words
// that all CTAs poll: 9,000 cycles a poll, 23,000 sector reads a round on
// twenty lines.)
// Slots of the two exchanges alternate: a CTA posts its next sum of one kind
// only after all others have posted the other kind, so none still reads the
// old word.  Polls are bounded: a CTA that gives up raises
// ESR_DEV_WAIT_TIMEOUT and leaves, and so, in turn, do the others.
#include "bcg_common.cuh"
#include "soft64.cuh"

namespace {

constexpr int kSoloThreads = 512;
constexpr int kSoloMaxCtas = 256;
constexpr int kSoloPolls = 1 << 24;  // (about ten seconds)
constexpr int kSoloSmem = 226 * 1024 - 12 * 1024;  // dynamic: the vectors; static: the sums

struct SoloComm {
  uint32_t epoch;  // exchanges done by earlier launches
  uint32_t pad[63];
  ulonglong2 mail[3][kSoloMaxCtas][kSoloMaxCtas];  // p.q, r.r, r.z: [to][from]
  uint32_t ready[kSoloMaxCtas][kSoloMaxCtas];      // number of the last exchange whose z is stored: [to][from]
};

__device__ __forceinline__ void post(ulonglong2 *w, double v, uint32_t epoch) {
  const uint64_t u = (uint64_t)__double_as_longlong(v), tag = (uint64_t)epoch << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(tag | (u >> 32)), "l"(tag | (uint32_t)u)
               : "memory");
}

// Polls the words at w (if a) and w + 128 (if b) together; their sum in v.
__device__ __forceinline__ bool poll(const ulonglong2 *w, bool a, bool b, uint32_t epoch, double &v) {
  uint64_t x0 = 0, x1 = 0, y0 = 0, y1 = 0;
  for (int tries = 0; tries < kSoloPolls; ++tries) {
    if (a) asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x0), "=l"(x1) : "l"(w) : "memory");
    if (b) asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(y0), "=l"(y1) : "l"(w + 128) : "memory");
    const bool got_a = !a || ((uint32_t)(x0 >> 32) == epoch && (uint32_t)(x1 >> 32) == epoch);
    const bool got_b = !b || ((uint32_t)(y0 >> 32) == epoch && (uint32_t)(y1 >> 32) == epoch);
    if (got_a && got_b) {
      v = a ? __longlong_as_double((long long)((x0 << 32) | (uint32_t)x1)) : 0.0;
      if (b) v += __longlong_as_double((long long)((y0 << 32) | (uint32_t)y1));
      return true;
    }
  }
  v = 0.0;
  return false;
}

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void sync_part(int barrier, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(threads) : "memory");
}

struct SoloShared {
  double part[2][kSoloThreads];  // per-thread sums
  double warp[2][4];
  double cta[2][4];              // the grid's sums, four parts each
  double alpha, beta;
  int stop, failed;
};

// Sums v[0..K) over the grid.  Warps 4 k .. 4 k + 3 add the CTA's values of
// sum k (one warp a scheduler: FP64 adds issue every 64 cycles each), post
// them and poll the other CTAs' (a warp 64 of them); 32-CTA sums are left in
// sh.cta, past a barrier (grid_sum() adds them).  PUBLISH: every thread's
// earlier global stores are visible to all CTAs afterwards (warps 8 .. 15).
// False: a poll gave up.
template <int K, bool PUBLISH>
__device__ __forceinline__ bool exchange(SoloShared &sh, const double (&v)[K], SoloComm *comm, int first,
                                         uint32_t epoch) {
  const int t = threadIdx.x, g = t >> 7, u = t & 127, lane = t & 31, grid = (int)gridDim.x;
#pragma unroll
  for (int k = 0; k < K; ++k) sh.part[k][t] = v[k];
  __syncthreads();
  if (g < K) {
    const double *s = sh.part[g];
    const double w = warp_sum((s[u] + s[u + 128]) + (s[u + 256] + s[u + 384]));
    if (lane == 0) sh.warp[g][u >> 5] = w;
    sync_part(1 + g, 128);
    const double b = (sh.warp[g][0] + sh.warp[g][1]) + (sh.warp[g][2] + sh.warp[g][3]);
    for (int to = u; to < grid; to += 128) post(&comm->mail[first + g][to][blockIdx.x], b, epoch);
    double two;
    if (!poll(&comm->mail[first + g][blockIdx.x][u], u < grid, u + 128 < grid, epoch, two)) sh.failed = 1;
    const double m = warp_sum(two);
    if (lane == 0) sh.cta[g][u >> 5] = m;
  } else if (PUBLISH && t >= 256) {
    fence_gpu();
    for (int to = t - 256; to < grid; to += 256)
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&comm->ready[to][blockIdx.x]), "r"(epoch) : "memory");
    for (int i = t - 256; i < grid; i += 256) {
      uint32_t e = epoch - 1;
      for (int tries = 0; tries < kSoloPolls && e != epoch; ++tries)
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(&comm->ready[blockIdx.x][i]) : "memory");
      if (e != epoch) sh.failed = 1;
    }
    fence_gpu();
  }
  __syncthreads();
  return sh.failed == 0;
}

__device__ __forceinline__ double grid_sum(const SoloShared &sh, int k) {
  const double *c = sh.cta[k];
  return (c[0] + c[1]) + (c[2] + c[3]);
}

// sum over a row's W slots of val * z(col), all loads in flight (W = the
// slice's width, uniform in the warp: predicated-off FP64 instructions would
// still take their pipe)
template <int W>
__device__ __forceinline__ double row_of(const int32_t *__restrict__ cp, const double *__restrict__ vp, int64_t n,
                                         const double *z) {
  int32_t c[W];
  double v[W], zc[W];
#pragma unroll
  for (int k = 0; k < W; ++k) c[k] = __ldg(cp + 32 * k);
#pragma unroll
  for (int k = 0; k < W; ++k) {
    v[k] = __ldg(vp + 32 * k);
    zc[k] = (uint32_t)c[k] < (uint32_t)n ? __ldcg(z + c[k]) : 0.0;  // -1 = padding
  }
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((uint32_t)c[k] < (uint32_t)n) acc = fma(v[k], zc[k], acc);
  return acc;
}

__device__ __forceinline__ double row_sum(int64_t slice, int lane, int64_t n, const int64_t *__restrict__ slice_ptr,
                                          const int32_t *__restrict__ col, const double *__restrict__ val,
                                          const double *z) {
  const int64_t b = __ldg(slice_ptr + slice);
  const int w = (int)((__ldg(slice_ptr + slice + 1) - b) >> 5);
  const int32_t *cp = col + b + lane;
  const double *vp = val + b + lane;
  switch (w) {
    case 0: return 0.0;
    case 1: return row_of<1>(cp, vp, n, z);
    case 2: return row_of<2>(cp, vp, n, z);
    case 3: return row_of<3>(cp, vp, n, z);
    case 4: return row_of<4>(cp, vp, n, z);
    case 5: return row_of<5>(cp, vp, n, z);
    case 6: return row_of<6>(cp, vp, n, z);
    case 7: return row_of<7>(cp, vp, n, z);
    default: break;
  }
  double acc = 0.0;
  for (int k = 0; k < w; ++k) {
    const int32_t c = __ldg(cp + 32 * k);
    if ((uint32_t)c < (uint32_t)n) acc = fma(__ldg(vp + 32 * k), __ldcg(z + c), acc);
  }
  return acc;
}

// One row's matrix entries, diagonal and its inverse.
struct HeldRow {
  double diag, inv;
  int32_t w, c[8];
  double v[8];
  __device__ __forceinline__ void load(int64_t slice, int lane, const BArgs &a, const double *val, const double *dg,
                                       const double *iv) {
    const int64_t b = a.slice_ptr[slice], i = slice * 32 + lane;
    w = (int)((a.slice_ptr[slice + 1] - b) >> 5);
    diag = dg[i];
    inv = iv ? iv[i] : 1.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = k < w && (uint32_t)a.col[b + 32 * k + lane] < (uint32_t)a.n;  // -1 = padding
      c[k] = in ? a.col[b + 32 * k + lane] : -1;
      v[k] = in ? val[b + 32 * k + lane] : 0.0;
    }
  }
  __device__ __forceinline__ double sum(const double *z) const {
    double zc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < w) zc[k] = c[k] >= 0 ? __ldcg(z + c[k]) : 0.0;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k >= w) break;  // (uniform in the warp)
      if (c[k] >= 0) acc = fma(v[k], zc[k], acc);
    }
    return acc;
  }
};

// SMALL: at most one slice a warp, of at most eight slots: its matrix stays in
// registers.
template <bool JACOBI, bool SMALL>
__global__ void __launch_bounds__(kSoloThreads, 1)
pcg_solo_kernel(BArgs a, const double *__restrict__ val, const double *__restrict__ diag,
                const double *__restrict__ invdiag, double *__restrict__ x, double *__restrict__ r, double *z,
                double *__restrict__ p, double *__restrict__ q, int32_t iters, int32_t cap, BcgLayout L,
                SoloComm *comm) {
  extern __shared__ double smem[];
  __shared__ SoloShared sh;
  double *const sx = smem, *const sr = sx + cap, *const sp = sr + cap, *const sq = sp + cap;
  esr_bcg_inst &inst = L.inst[0];
  if (inst.done) return;
  const int64_t slices = a.n >> 5;
  const int64_t s0 = slices * blockIdx.x / gridDim.x, s1 = slices * (blockIdx.x + 1) / gridDim.x;
  const int64_t row0 = s0 * 32;
  const int rows = (int)((s1 - s0) * 32), nsl = (int)(s1 - s0);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  uint32_t epoch = comm->epoch;
  double rz = inst.rz, rr = inst.rr, pq = inst.pq;
  const double tol = inst.tol, tol2 = tol * tol;
  int count = inst.iters, done = 0;
  const int maxiter = inst.maxiter;
  bool first = inst.refresh != 0;
  if (t == 0) {
    sh.beta = inst.beta;
    sh.failed = 0;
    sh.stop = 0;
  }
  for (int j = t; j < rows; j += kSoloThreads) {
    sx[j] = x[row0 + j];
    sr[j] = r[row0 + j];
    sp[j] = p[row0 + j];
    sq[j] = first ? 0.0 : q[row0 + j];
  }
  __syncthreads();
  double beta = sh.beta, alpha = 0.0;
  HeldRow own;
  if constexpr (SMALL) {
    if (warp < nsl) own.load(s0 + warp, lane, a, val, diag, JACOBI ? invdiag : nullptr);
  }
  // squares that tell ||r|| <= tol without a square root
  const bool far = tol2 > 1e-280 && tol2 < 1e280;
  const double tol2_lo = tol2 * (1 - 1e-12), tol2_hi = tol2 * (1 + 1e-12);
  for (int it = 0; it < iters; ++it) {
    double v1[1] = {0.0};
#pragma unroll 2
    for (int s = warp; s < nsl; s += kSoloThreads / 32) {
      const int64_t i = (s0 + s) * 32 + lane;
      const int j = s * 32 + lane;
      const double zi = __ldcg(z + i);
      double w;
      if constexpr (SMALL) w = fma(own.diag, zi, own.sum(z));
      else w = fma(__ldg(diag + i), zi, row_sum(s0 + s, lane, a.n, a.slice_ptr, a.col, val, z));
      const double pi = first ? zi : fma(beta, sp[j], zi);
      const double qi = first ? w : fma(beta, sq[j], w);
      sp[j] = pi;
      sq[j] = qi;
      v1[0] = fma(pi, qi, v1[0]);
    }
    if (!exchange<1, false>(sh, v1, comm, 0, ++epoch)) break;
    if (t == 0) {
      pq = grid_sum(sh, 0);
      sh.stop = (!(pq != 0.0) || !isfinite(pq)) ? 3 : 0;
      sh.alpha = sh.stop ? 0.0 : soft64::quotient(rz, soft64::Divisor(pq));
    }
    __syncthreads();
    if (sh.stop) {  // breakdown
      done = 3;
      break;
    }
    alpha = sh.alpha;
    first = false;
    double v2[2] = {0.0, 0.0};
#pragma unroll 2
    for (int s = warp; s < nsl; s += kSoloThreads / 32) {
      const int64_t i = (s0 + s) * 32 + lane;
      const int j = s * 32 + lane;
      sx[j] = fma(alpha, sp[j], sx[j]);
      const double ri = fma(-alpha, sq[j], sr[j]);
      sr[j] = ri;
      double zi = ri;
      if constexpr (JACOBI && SMALL) zi = ri * own.inv;
      else if constexpr (JACOBI) zi = soft64::product(ri, __ldg(invdiag + i));  // (beside the busy FP64 pipe)
      __stcg(z + i, zi);
      v2[0] = fma(ri, ri, v2[0]);
      if (JACOBI) v2[1] = fma(ri, zi, v2[1]);
    }
    const soft64::Divisor by_rz(rz);  // (thread 0's)
    bool ok;
    if (JACOBI) {
      ok = exchange<2, true>(sh, v2, comm, 1, ++epoch);
    } else {  // z = r: one sum
      const double v[1] = {v2[0]};
      ok = exchange<1, true>(sh, v, comm, 1, ++epoch);
    }
    if (!ok) break;
    ++count;
    if (t == 0) {
      rr = grid_sum(sh, 0);
      const double rz_new = JACOBI ? grid_sum(sh, 1) : rr;
      const bool met = far && !(rr > tol2_lo && rr < tol2_hi) ? rr <= tol2 : sqrt(rr) <= tol;
      int stop = 0;
      if (met) stop = 1;  // (false for NaN)
      else if (maxiter >= 0 && count - 1 >= maxiter) stop = 2;
      else if (!isfinite(rr) || !isfinite(rz_new) || rz == 0.0) stop = 3;
      else {
        sh.beta = soft64::quotient(rz_new, by_rz);
        rz = rz_new;
      }
      sh.stop = stop;
    }
    __syncthreads();
    if (sh.stop) {
      done = sh.stop;
      break;
    }
    beta = sh.beta;
  }
  const bool failed = sh.failed != 0;
  for (int j = t; j < rows; j += kSoloThreads) {
    x[row0 + j] = sx[j];
    r[row0 + j] = sr[j];
    p[row0 + j] = sp[j];
    q[row0 + j] = sq[j];
  }
  if (t == 0 && failed) esr::raise_status(ESR_DEV_WAIT_TIMEOUT);
  if (blockIdx.x == 0 && t == 0) {
    inst.rz = rz;
    inst.rz_jac = rz;
    inst.rr = rr;
    inst.pq = pq;
    inst.iters = count;
    inst.refresh = first ? inst.refresh : 0;
    set_alpha(inst, alpha);
    set_beta(inst, sh.beta);
    comm->epoch = epoch;
    if (failed) done = 3;
    if (done) {
      inst.done = done;
      retire(L);
    }
  }
}

// CTAs of a system of n rows on `sms` multiprocessors, 0 if its vectors do not
// fit: eight slices (one row a lane for half the warps) pay for a CTA.
int solo_ctas(int64_t n, int sms) {
  const int64_t slices = n >> 5;
  int64_t g = (slices + 7) / 8;
  if (g > sms) g = sms;
  if (g > kSoloMaxCtas) g = kSoloMaxCtas;
  if (g < 1) return 0;
  const int64_t cap = (slices + g - 1) / g * 32;
  return cap * 4 * (int64_t)sizeof(double) <= kSoloSmem ? (int)g : 0;
}

int device_sms(int *sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
  return e == cudaSuccess ? ESR_OK : esr::cuda_check(e, "esr_pcg_solo");
}

}  // namespace

ESR_DEFINE_STATUS_READER(esr_status_pcg_solo)

extern "C" int esr_pcg_solo_ctas(const esr_batch *B) {
  if (check_batch(B) || B->ninst != 1 || B->df64 || B->gnn || B->poly_degree || B->n >= ((int64_t)1 << 31)) return 0;
  int sms = 0;
  if (device_sms(&sms)) return 0;
  return solo_ctas(B->n, sms);
}

extern "C" int64_t esr_pcg_solo_comm_bytes(void) { return (int64_t)sizeof(SoloComm); }

extern "C" int esr_pcg_solo_iterate(const esr_batch *B, int32_t max_width, void *x, void *r, void *z, void *p, void *q,
                                    int32_t k, void *workspace, void *comm, void *stream) {
  int st = check_batch(B);
  if (st) return st;
  if (!x || !r || !z || !p || !q || !workspace || !comm) return esr::fail(ESR_ERR_ARG, "null vector");
  if (k < 0) return esr::fail(ESR_ERR_ARG, "negative iteration count");
  const int ctas = esr_pcg_solo_ctas(B);
  if (!ctas) return esr::fail(ESR_ERR_UNSUPPORTED, "esr_pcg_solo_iterate: one FP64 system that fits the chip's shared memory");
  if (k == 0) return ESR_OK;
  BcgLayout L = layout_of(workspace, B->ninst, B->nchunks);
  BArgs a = bargs(B);
  const int64_t slices = B->n >> 5;
  int32_t cap = (int32_t)((slices + ctas - 1) / ctas * 32);
  const int smem = cap * 4 * (int)sizeof(double);
  const bool small = cap <= kSoloThreads && max_width <= 8;
  const void *fn = B->invdiag ? (small ? (const void *)pcg_solo_kernel<true, true> : (const void *)pcg_solo_kernel<true, false>)
                              : (small ? (const void *)pcg_solo_kernel<false, true> : (const void *)pcg_solo_kernel<false, false>);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_pcg_solo_iterate/smem attribute");
  const double *val = (const double *)B->val, *diag = (const double *)B->diag, *inv = (const double *)B->invdiag;
  SoloComm *cm = (SoloComm *)comm;
  void *args[] = {&a, &val, &diag, &inv, &x, &r, &z, &p, &q, &k, &cap, &L, &cm};
  e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)ctas), dim3(kSoloThreads), args, (size_t)smem, esr::as_stream(stream));
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_pcg_solo_iterate");
  return ESR_OK;
}
