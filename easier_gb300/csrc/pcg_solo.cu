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
// matrix streams from L2, and only p goes through memory.  An iteration has
// three grid exchanges instead of three launches:
//   q = A p; p.q                                      -> exchange
//   x += alpha p, r -= alpha q, z = M r; r.r, r.z     -> exchange
//   p = z + beta p, published                         -> barrier
// Each is of another kind than the one before, so no CTA posts a word that
// another may still read; a CTA whose poll gave up raises ESR_DEV_WAIT_TIMEOUT
// and stops the instance.
// (The form p = z + beta p, q = A z + beta q needs one exchange fewer, z being
// published with r.r: 5.8 ms in place of 6.6 in the first case below, the same
// time in the second.  But its q drifts from A p: two to four times the launch
// sequence's distance from CG in extended precision, where this form has 0.9
// to 1.15 times.)
// Measured: FV Poisson, 40,000 rows, 682 iterations 14.4 -> 6.6 ms; P1 grid,
// 998,001 rows, 2,720 iterations 156 -> 88 ms (32 us an iteration, most of them
// the sweeps' FP64 instructions; z = M r takes its product to the integer
// pipes, soft64.cuh).  Below them only latency is left: about 1,500 cycles from
// a post to its poll, 700 for the sums of a CTA, 800 for a scalar division.

#include "bcg_common.cuh"
#include "grid_exchange.cuh"
#include "soft64.cuh"

namespace {

constexpr int kSoloSmem = 226 * 1024 - 12 * 1024;  // dynamic: the vectors; static: the sums

struct SoloShared : ExchangeShared {
  double alpha, beta;
  int stop;
};

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
  __device__ __forceinline__ double sum(const double *p) const {
    double pc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < w) pc[k] = c[k] >= 0 ? __ldcg(p + c[k]) : 0.0;
    double acc = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k >= w) break;  // (uniform in the warp)
      if (c[k] >= 0) acc = fma(v[k], pc[k], acc);
    }
    return acc;
  }
};

// SMALL: at most one slice a warp, of at most eight slots: its matrix stays in
// registers.
template <bool JACOBI, bool SMALL, int POLLS>
__global__ void __launch_bounds__(kSoloThreads, 1)
pcg_solo_kernel(BArgs a, const double *__restrict__ val, const double *__restrict__ diag,
                const double *__restrict__ invdiag, double *__restrict__ x, double *__restrict__ r, double *p,
                int32_t iters, int32_t cap, BcgLayout L, GridComm *comm) {
  extern __shared__ double smem[];
  __shared__ SoloShared sh;
  // (q = A p until the update, z = M r after it)
  double *const sx = smem, *const sr = sx + cap, *const sp = sr + cap, *const sqz = sp + cap;
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
  const int maxiter = inst.maxiter, count0 = count;
  if (t == 0) {
    sh.beta = inst.beta;
    sh.failed = 0;
    sh.stop = 0;
  }
  for (int j = t; j < rows; j += kSoloThreads) {
    sx[j] = x[row0 + j];
    sr[j] = r[row0 + j];
    sp[j] = p[row0 + j];
  }
  __syncthreads();
  double alpha = 0.0;
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
      const double pi = sp[j];
      double qi;
      if constexpr (SMALL) qi = fma(own.diag, pi, own.sum(p));
      else qi = fma(__ldg(diag + i), pi, row_sum(s0 + s, lane, a.n, a.slice_ptr, a.col, val, [&](int32_t c) { return __ldcg(p + c); }));
      sqz[j] = qi;
      v1[0] = fma(pi, qi, v1[0]);
    }
    if (!exchange<1, false, POLLS>(sh, v1, comm, 0, ++epoch)) break;
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
    double v2[2] = {0.0, 0.0};
#pragma unroll 2
    for (int s = warp; s < nsl; s += kSoloThreads / 32) {
      const int64_t i = (s0 + s) * 32 + lane;
      const int j = s * 32 + lane;
      sx[j] = fma(alpha, sp[j], sx[j]);
      const double ri = fma(-alpha, sqz[j], sr[j]);
      sr[j] = ri;
      double zi = ri;
      if constexpr (JACOBI && SMALL) zi = ri * own.inv;
      else if constexpr (JACOBI) zi = soft64::product(ri, __ldg(invdiag + i));  // (beside the busy FP64 pipe)
      sqz[j] = zi;
      v2[0] = fma(ri, ri, v2[0]);
      if (JACOBI) v2[1] = fma(ri, zi, v2[1]);
    }
    const soft64::Divisor by_rz(rz);  // (thread 0's)
    bool ok;
    if (JACOBI) {
      ok = exchange<2, false, POLLS>(sh, v2, comm, 1, ++epoch);
    } else {  // z = r: one sum
      const double v[1] = {v2[0]};
      ok = exchange<1, false, POLLS>(sh, v, comm, 1, ++epoch);
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
    const double beta = sh.beta;
#pragma unroll 2
    for (int s = warp; s < nsl; s += kSoloThreads / 32) {
      const int j = s * 32 + lane;
      const double pi = fma(beta, sp[j], sqz[j]);
      sp[j] = pi;
      __stcg(p + row0 + j, pi);
    }
    if (!publish<POLLS>(sh, comm, ++epoch)) break;
  }
  const bool failed = sh.failed != 0;
  for (int j = t; j < rows; j += kSoloThreads) {
    x[row0 + j] = sx[j];
    r[row0 + j] = sr[j];
  }
  if (t == 0 && failed) {  // (any CTA: the others may have got their sums and left)
    esr::raise_status(ESR_DEV_WAIT_TIMEOUT);
    give_up(L, 0);
  }
  if (blockIdx.x == 0 && t == 0) {
    inst.rz = rz;
    inst.rz_jac = rz;
    inst.rr = rr;
    inst.pq = pq;
    inst.iters = count;
    if (count > count0) inst.refresh = 0;
    set_alpha(inst, alpha);
    set_beta(inst, sh.beta);
    comm->epoch = epoch;
    if (done && atomicCAS(&inst.done, 0, done) == 0) retire(L);
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

template <int POLLS>
int run_solo(const esr_batch *B, int32_t max_width, void *x, void *r, void *z, void *p, void *q, int32_t k,
             void *workspace, void *comm, void *stream) {
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
  const void *fn =
      B->invdiag ? (small ? (const void *)pcg_solo_kernel<true, true, POLLS> : (const void *)pcg_solo_kernel<true, false, POLLS>)
                 : (small ? (const void *)pcg_solo_kernel<false, true, POLLS> : (const void *)pcg_solo_kernel<false, false, POLLS>);
  // (the limit belongs to the function, not to this launch: always the largest,
  // or another thread's smaller system could lower it before this launch)
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSoloSmem);
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_pcg_solo_iterate/smem attribute");
  const double *val = (const double *)B->val, *diag = (const double *)B->diag, *inv = (const double *)B->invdiag;
  GridComm *cm = (GridComm *)comm;
  void *args[] = {&a, &val, &diag, &inv, &x, &r, &p, &k, &cap, &L, &cm};
  e = cudaLaunchCooperativeKernel(fn, dim3((unsigned)ctas), dim3(kSoloThreads), args, (size_t)smem, esr::as_stream(stream));
  if (e != cudaSuccess) return esr::cuda_check(e, "esr_pcg_solo_iterate");
  return ESR_OK;
}

}  // namespace

ESR_DEFINE_STATUS_READER(esr_status_pcg_solo)

extern "C" int esr_pcg_solo_ctas(const esr_batch *B) {
  if (check_batch(B) || B->ninst != 1 || B->df64 || B->gnn || B->poly_degree || B->n >= ((int64_t)1 << 31)) return 0;
  int sms = 0;
  if (device_sms(&sms)) return 0;
  return solo_ctas(B->n, sms);
}

extern "C" int64_t esr_pcg_solo_comm_bytes(void) { return (int64_t)sizeof(GridComm); }

extern "C" int esr_pcg_solo_iterate(const esr_batch *B, int32_t max_width, void *x, void *r, void *z, void *p, void *q,
                                    int32_t k, void *workspace, void *comm, void *stream) {
  return run_solo<kSoloPolls>(B, max_width, x, r, z, p, q, k, workspace, comm, stream);
}

extern "C" int esr_pcg_solo_iterate_timeout(const esr_batch *B, int32_t max_width, void *x, void *r, void *z, void *p,
                                            void *q, int32_t k, void *workspace, void *comm, void *stream) {
  return run_solo<0>(B, max_width, x, r, z, p, q, k, workspace, comm, stream);
}
