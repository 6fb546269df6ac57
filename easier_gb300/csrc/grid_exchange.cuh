// Exchange of block sums between the CTAs of a cooperative launch.
//
// A CTA posts its sum to every CTA's mailbox, as two 64-bit words that each
// hold 32 bits of the double and the exchange's number; every CTA polls its
// own mailbox and adds the sums itself in the same order, so all take the same
// decisions and no second barrier distributes the result.  That its global
// stores are done a CTA tells with a word of its own, posted behind a fence: by
// other warps while the sums are added, or in a barrier of its own (publish).  A word is posted again only after
// an exchange that everybody's reading of the last one precedes.  (One set of
// words that all CTAs poll: 9,000 cycles a poll, 23,000 sector reads a round
// on twenty lines; mailboxes: 1,500.)  Polls are bounded: a CTA that gives up
// leaves, and so, in turn, do the others.
#pragma once

#include <cstdint>

#include "esr_internal.h"

namespace {

constexpr int kSoloThreads = 512;  // threads that take part
constexpr int kSoloMaxCtas = 256;
constexpr int kSoloPolls = 1 << 24;  // (about ten seconds; POLLS below: 0 in tests of the giving up)

struct GridComm {
  uint32_t epoch;  // exchanges done by earlier launches
  uint32_t pad[63];
  ulonglong2 mail[3][kSoloMaxCtas][kSoloMaxCtas];  // three kinds of sums: [to][from]
  uint32_t ready[kSoloMaxCtas][kSoloMaxCtas];      // the last exchange before which stores are done: [to][from]
};

__device__ __forceinline__ void post(ulonglong2 *w, double v, uint32_t epoch) {
  const uint64_t u = (uint64_t)__double_as_longlong(v), tag = (uint64_t)epoch << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(tag | (u >> 32)), "l"(tag | (uint32_t)u)
               : "memory");
}

// Polls the words at w (if a) and w + 128 (if b) together; their sum in v.
template <int POLLS>
__device__ __forceinline__ bool poll(const ulonglong2 *w, bool a, bool b, uint32_t epoch, double &v) {
  uint64_t x0 = 0, x1 = 0, y0 = 0, y1 = 0;
  for (int tries = 0; tries < POLLS; ++tries) {
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

struct ExchangeShared {
  double part[2][kSoloThreads];  // per-thread sums
  double warp[2][4];
  double cta[2][4];              // the grid's sums, four parts each
  int failed;
};

// Threads first .. of `threads` of a CTA whose stores are done (past a barrier)
// tell all CTAs so and wait for the same from them.
template <int POLLS>
__device__ __forceinline__ void tell_and_wait(ExchangeShared &sh, GridComm *comm, uint32_t epoch, int first,
                                              int threads) {
  const int grid = (int)gridDim.x;
  if ((first & ~31) >= grid) return;  // (whole warps without a CTA to tell)
  fence_gpu();
  for (int to = first; to < grid; to += threads)
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&comm->ready[to][blockIdx.x]), "r"(epoch) : "memory");
  for (int i = first; i < grid; i += threads) {
    uint32_t e = epoch - 1;  // (a CTA ahead may already have told of a later exchange)
    for (int tries = 0; tries < POLLS && (int32_t)(e - epoch) < 0; ++tries)
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(&comm->ready[blockIdx.x][i]) : "memory");
    if ((int32_t)(e - epoch) < 0) sh.failed = 1;
  }
  fence_gpu();
}

// Barrier of the grid: every thread's earlier global stores are visible to all
// CTAs afterwards.
template <int POLLS>
__device__ __forceinline__ bool publish(ExchangeShared &sh, GridComm *comm, uint32_t epoch) {
  sync_part(0, kSoloThreads);
  tell_and_wait<POLLS>(sh, comm, epoch, (int)threadIdx.x, kSoloThreads);
  sync_part(0, kSoloThreads);
  return sh.failed == 0;
}

// Sums v[0..K) over the grid.  Warps 4 k .. 4 k + 3 add the CTA's values of
// sum k (one warp a scheduler: FP64 adds issue every 64 cycles each), post
// them and poll the other CTAs' (a warp 64 of them); 32-CTA sums are left in
// sh.cta, past a barrier (grid_sum() adds them).  PUBLISH: every thread's
// earlier global stores are visible to all CTAs afterwards (warps 8 .. 15).
// False: a poll gave up.
template <int K, bool PUBLISH, int POLLS>
__device__ __forceinline__ bool exchange(ExchangeShared &sh, const double (&v)[K], GridComm *comm, int first,
                                         uint32_t epoch) {
  const int t = threadIdx.x, g = t >> 7, u = t & 127, lane = t & 31, grid = (int)gridDim.x;
#pragma unroll
  for (int k = 0; k < K; ++k) sh.part[k][t] = v[k];
  sync_part(0, kSoloThreads);
  if (g < K) {
    const double *s = sh.part[g];
    const double w = warp_sum((s[u] + s[u + 128]) + (s[u + 256] + s[u + 384]));
    if (lane == 0) sh.warp[g][u >> 5] = w;
    sync_part(1 + g, 128);
    const double b = (sh.warp[g][0] + sh.warp[g][1]) + (sh.warp[g][2] + sh.warp[g][3]);
    for (int to = u; to < grid; to += 128) post(&comm->mail[first + g][to][blockIdx.x], b, epoch);
    double two;
    if (!poll<POLLS>(&comm->mail[first + g][blockIdx.x][u], u < grid, u + 128 < grid, epoch, two)) sh.failed = 1;
    const double m = warp_sum(two);
    if (lane == 0) sh.cta[g][u >> 5] = m;
  } else if (PUBLISH && t >= 256) {
    tell_and_wait<POLLS>(sh, comm, epoch, t - 256, 256);
  }
  sync_part(0, kSoloThreads);
  return sh.failed == 0;
}

__device__ __forceinline__ double grid_sum(const ExchangeShared &sh, int k) {
  const double *c = sh.cta[k];
  return (c[0] + c[1]) + (c[2] + c[3]);
}

// sum over a row's W slots of val * x(col), all loads in flight (W = the
// slice's width, uniform in the warp: predicated-off FP64 instructions would
// still take their pipe)
template <int W, typename T, class X>
__device__ __forceinline__ double row_of(const int32_t *__restrict__ cp, const T *__restrict__ vp, int64_t n,
                                         const X &x) {
  int32_t c[W];
  double v[W], xc[W];
#pragma unroll
  for (int k = 0; k < W; ++k) c[k] = __ldg(cp + 32 * k);
#pragma unroll
  for (int k = 0; k < W; ++k) {
    v[k] = (double)__ldg(vp + 32 * k);
    xc[k] = (uint32_t)c[k] < (uint32_t)n ? x(c[k]) : 0.0;  // -1 = padding
  }
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < W; ++k)
    if ((uint32_t)c[k] < (uint32_t)n) acc = fma(v[k], xc[k], acc);
  return acc;
}

template <typename T, class X>
__device__ __forceinline__ double row_sum(int64_t slice, int lane, int64_t n, const int64_t *__restrict__ slice_ptr,
                                          const int32_t *__restrict__ col, const T *__restrict__ val, const X &x) {
  const int64_t b = __ldg(slice_ptr + slice);
  const int w = (int)((__ldg(slice_ptr + slice + 1) - b) >> 5);
  const int32_t *cp = col + b + lane;
  const T *vp = val + b + lane;
  switch (w) {
    case 0: return 0.0;
    case 1: return row_of<1>(cp, vp, n, x);
    case 2: return row_of<2>(cp, vp, n, x);
    case 3: return row_of<3>(cp, vp, n, x);
    case 4: return row_of<4>(cp, vp, n, x);
    case 5: return row_of<5>(cp, vp, n, x);
    case 6: return row_of<6>(cp, vp, n, x);
    case 7: return row_of<7>(cp, vp, n, x);
    default: break;
  }
  double acc = 0.0;
  for (int k = 0; k < w; ++k) {
    const int32_t c = __ldg(cp + 32 * k);
    if ((uint32_t)c < (uint32_t)n) acc = fma((double)__ldg(vp + 32 * k), x(c), acc);
  }
  return acc;
}

}  // namespace
