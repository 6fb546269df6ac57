// The streaming loop of the batched PCG's sweeps (bcg.cu).
//
// The sweeps are bound by memory, and a thread that loads a row, computes and
// stores it keeps too few bytes in flight: 64 registers a thread allow 32
// warps a SM, each waiting for its own slice pointer, then its columns, then
// its gathers, and at the end of each chunk for a fence and a ticket in L2.
// Here a CTA has three kinds of warps, which meet at mbarriers only:
//   * one fetches: it walks the CTA's chunks and copies each tile's rows into
//     a ring of stages (bulk asynchronous copies, issued by one lane an
//     array), with a header that says which tile it is;
//   * eight compute, a row a thread, out of the stages;
//   * one finishes: it adds a chunk's eight partial sums, publishes them and
//     takes the instance's ticket while the others stream the next chunk.
// The fetching and the finishing warp read the headers of 32 chunks at once,
// one a lane, so that their chains of dependent loads run side by side.
//
// Measured on 48 P1 meshes of 32 to 384 cells a side (2.35 M rows, 1,480
// iterations, double-float): 118.9 -> 85.7 ms, an iteration of all of them
// 78 us where the copy rate allows 56.  What bounds it now: in the direction
// sweep the arithmetic's latency (2,400 of 3,500 cycles a tile, the gathers of
// z with it) at the 24 computing warps that the rings leave room for, in the
// update sweep the copies' latency at either end (13,000 of 40,000 cycles).
// Slower, against 91.0 ms with the rings of that time, were: gathers loaded a
// tile ahead, which takes deeper rings and so 16 warps a SM (108 ms); copies issued by the computing warps, an array each
// (117 ms: a copy takes its warp 200 cycles to issue); no rings but the next
// tile's columns in registers (199 ms: spills); the next sweep launched early
// (91.3: no gain inside a captured graph).
//
// Every wait is bounded.  A warp that gives up raises ESR_DEV_WAIT_TIMEOUT
// and leaves; so, in turn, do the others, and the finishing warp stops the
// instances of the chunks it did not get (done = kTimedOut).
#pragma once

#include "bcg_common.cuh"

namespace {

constexpr int kBWarps = kBThreads / 32;         // warps that compute
constexpr int kStreamThreads = kBThreads + 64;  // and those that fetch and finish
constexpr int kStreamPolls = 1 << 22;           // polls of a wait before it gives up (POLLS below: 0 in tests of that)
constexpr int kTileBytes = kBThreads * 8;       // a tile's rows of one vector

__device__ __forceinline__ uint32_t shared_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t *bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(shared_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_arrive_expect(uint64_t *bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_addr(bar)), "r"(bytes) : "memory");
}
template <int POLLS>
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity) {
  for (int tries = 0; tries < POLLS; ++tries) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(shared_addr(bar)), "r"(parity)
                 : "memory");
    if (done) return true;
  }
  esr::raise_status(ESR_DEV_WAIT_TIMEOUT);
  return false;
}
// (both ends on 16 bytes, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, int bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   shared_addr(dst)),
               "l"(src), "r"(bytes), "r"(shared_addr(bar))
               : "memory");
}

enum : int { kLastTile = 1, kFlag = 2, kStop = 4 };

struct StageHead {
  unsigned long long coefficient;
  int tile, bits;
};

template <class P, int S, int K>
struct StreamShared {
  uint64_t full[S], empty[S];
  uint64_t parts_full[2], parts_empty[2];  // sets of parts
  __align__(16) StageHead head[S];
  int2 slice[S][kBWarps];                // (where in the stage, how wide) the tile's slices are
  typename P::V parts[2][K][kBThreads];  // the threads' sums of a chunk
};

// Copies `bytes` (a multiple of 128) for the whole warp where the source may
// lie on any 4 bytes.
__device__ __forceinline__ void plain_copy(void *dst, const void *src, int bytes, int lane) {
  for (int o = lane; o < bytes / 4; o += 32) ((uint32_t *)dst)[o] = ((const uint32_t *)src)[o];
}

// The chunks [base, base + 32 grid) of this CTA's stride, one a lane.
template <class OP>
struct ChunkHeads {
  int chunk = 0, inst = 0, t0 = 0, t1 = 0, flag = 0;
  unsigned long long coefficient = 0;
  unsigned mask;  // the lanes with a chunk of a running instance
  // (`done` cannot change under a chunk that runs: only the instance's last
  // chunk to arrive sets it, after all have read it here; a finishing warp
  // that gives up sets it too, and then the sweep's result is void)
  __device__ __forceinline__ ChunkHeads(const BArgs &a, const BcgLayout &L, int64_t base, int count) {
    const int64_t u = base + (threadIdx.x & 31) * (int64_t)gridDim.x;
    int4 e = make_int4(0, 0, 0, 0);
    if (u < a.nchunks) e = L.heads[u];  // (beside the count)
    if (u < count) {
      chunk = e.x;
      inst = e.y;
      const esr_bcg_inst &s = L.inst[inst];
      const typename OP::V v = OP::coefficient(s);
      memcpy(&coefficient, &v, 8);
      flag = OP::flag(s) ? kFlag : 0;
      if (!s.done) {
        t0 = e.z;
        t1 = e.w;
      }
    }
    mask = __ballot_sync(0xffffffffu, t0 < t1);
  }
};

// ---- the sum of 256 threads' parts, by one warp (valid in lane 0, fixed order)
__device__ __forceinline__ double thread_part(const DotAccD &a) { return a.v; }
__device__ __forceinline__ df64::df thread_part(const DotAccDF &a) { return df64::quick_two_sum(a.hi, a.lo); }
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double parts_sum(const double *v) {
  double t[kBWarps / 2];
#pragma unroll
  for (int k = 0; k < kBWarps / 2; ++k) t[k] = v[64 * k] + v[64 * k + 32];
  return warp_total((t[0] + t[1]) + (t[2] + t[3]));
}
__device__ __forceinline__ double parts_sum(const df64::df *v) {
  df64::df t[kBWarps / 2];
#pragma unroll
  for (int k = 0; k < kBWarps / 2; ++k) t[k] = df64::add(v[64 * k], v[64 * k + 32]);
  const df64::df s = warp_sum_df(df64::add(df64::add(t[0], t[1]), df64::add(t[2], t[3])));
  return (double)s.hi + (double)s.lo;
}

// ---- A chunk's sum in the instance's mail: two words, each with 32 bits of
// the double and the sweep's tag.  The words say themselves that they have
// arrived, so a chunk's ticket needs no fence, which waits until the stores of
// the whole SM have drained (95.2 -> 93.8 ms); whoever takes the last ticket reads the
// instance's mail, and again what is not there yet: posted, all of it, by
// warps that have their tickets already.
constexpr int kMailAhead = 4;

__device__ __forceinline__ void post_sum(ulonglong2 *w, double v, uint32_t tag) {
  const uint64_t u = (uint64_t)__double_as_longlong(v), t = (uint64_t)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(t | (u >> 32)), "l"(t | (uint32_t)u)
               : "memory");
}

// Adds to v, in order, the sums at w, w + 32, ... (`count` of them, at most kMailAhead)
template <int POLLS>
__device__ __forceinline__ bool read_sums(const ulonglong2 *w, int count, uint32_t tag, double &v) {
  for (int tries = 0; tries < POLLS; ++tries) {
    uint64_t x[kMailAhead], y[kMailAhead];
    bool there = true;
#pragma unroll
    for (int k = 0; k < kMailAhead; ++k) {
      if (k >= count) continue;
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x[k]), "=l"(y[k]) : "l"(w + 32 * k) : "memory");
    }
#pragma unroll
    for (int k = 0; k < kMailAhead; ++k)
      there = there && (k >= count || ((uint32_t)(x[k] >> 32) == tag && (uint32_t)(y[k] >> 32) == tag));
    if (!there) continue;
#pragma unroll
    for (int k = 0; k < kMailAhead; ++k)
      if (k < count) v += __longlong_as_double((long long)((x[k] << 32) | (uint32_t)y[k]));
    return true;
  }
  esr::raise_status(ESR_DEV_WAIT_TIMEOUT);
  return false;
}

// Runs this CTA's chunks of the running instances.  OP has
//   S, kStageBytes, K          ring depth, bytes a stage, sums
//   kSweep                     1 or 2: which sweep of an iteration
//   coefficient(inst), flag(inst)   what compute needs of an instance
//   meta(tile, lane)           what the fetching warp must know of a tile
//   fetch(tile, meta, stage, slice, bar, lane)   starts its copies
//   compute(tile, stage, slice, coefficient, flag)   this thread's row
//   acc[K]                     the sums so far
//   finish(inst, tot)          the instance's sums are complete
template <int POLLS, class OP>
__device__ __forceinline__ void stream_chunks(const BArgs &a, const BcgLayout &L, char *ring,
                                              StreamShared<typename OP::P, OP::S, OP::K> &sh, OP &op) {
  using V = typename OP::V;
  constexpr int S = OP::S, K = OP::K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      bar_init(&sh.full[s], 1);
      bar_init(&sh.empty[s], kBWarps);
    }
    for (int s = 0; s < 2; ++s) {
      bar_init(&sh.parts_full[s], kBWarps);
      bar_init(&sh.parts_empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int count = L.head->acount;
  if (warp < kBWarps) {
    int stage = 0, number = 0;
    uint32_t phase = 0;
    while (true) {
      if (!bar_wait<POLLS>(&sh.full[stage], phase)) return;
      const StageHead h = sh.head[stage];
      if (h.bits & kStop) return;
      V coefficient;
      memcpy(&coefficient, &h.coefficient, 8);
      op.compute(h.tile, ring + stage * OP::kStageBytes, sh.slice[stage][warp], coefficient, h.bits & kFlag);
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.empty[stage]);
      if (++stage == S) {
        stage = 0;
        phase ^= 1;
      }
      if (h.bits & kLastTile) {
        const int set = number & 1;
        if (!bar_wait<POLLS>(&sh.parts_empty[set], ((number >> 1) & 1) ^ 1)) return;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          sh.parts[set][k][threadIdx.x] = thread_part(op.acc[k]);
          op.acc[k] = {};
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&sh.parts_full[set]);
        ++number;
      }
    }
  }
  if (warp == kBWarps) {  // fetch
    int stage = 0, tiles = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int64_t base = blockIdx.x; ok && base < count; base += 32 * (int64_t)gridDim.x) {
      const ChunkHeads<OP> own(a, L, base, count);
      unsigned left = own.mask;
      if (!left) continue;
      int k = __ffs((int)left) - 1;
      int t = __shfl_sync(0xffffffffu, own.t0, k), t1 = __shfl_sync(0xffffffffu, own.t1, k);
      typename OP::Meta next = op.meta(t, lane);
      while (ok && left) {
        const typename OP::Meta m = next;
        const int flag = __shfl_sync(0xffffffffu, own.flag, k);
        const unsigned long long coefficient = __shfl_sync(0xffffffffu, own.coefficient, k);
        StageHead h{coefficient, t, flag | (t + 1 == t1 ? kLastTile : 0)};
        if (++t == t1) {  // the tile after this one, whose meta is loaded meanwhile
          left &= left - 1;
          k = left ? __ffs((int)left) - 1 : 0;
          t = __shfl_sync(0xffffffffu, own.t0, k);
          t1 = __shfl_sync(0xffffffffu, own.t1, k);
        }
        if (left) next = op.meta(t, lane);
        ok = bar_wait<POLLS>(&sh.empty[stage], phase ^ 1);
        if (!ok) break;
        if (lane == 0) sh.head[stage] = h;
        op.fetch(h.tile, m, ring + stage * OP::kStageBytes, sh.slice[stage], &sh.full[stage], lane);
        if (++stage == S) {
          stage = 0;
          phase ^= 1;
        }
        ++tiles;
      }
    }
    // no copy may land after the CTA has left, whoever gave up (before the stop,
    // which completes another phase)
    for (int t = max(tiles - S, 0); t < tiles; ++t) bar_wait<kStreamPolls>(&sh.full[t % S], (t / S) & 1);
    if (ok) ok = bar_wait<POLLS>(&sh.empty[stage], phase ^ 1);
    if (ok && lane == 0) {
      sh.head[stage].bits = kStop;
      bar_arrive(&sh.full[stage]);
    }
    return;
  }
  int number = 0;  // finish
  bool ok = true;
  for (int64_t base = blockIdx.x; base < count; base += 32 * (int64_t)gridDim.x) {
    const ChunkHeads<OP> own(a, L, base, count);
    int first = 0, end = 0, iters = 0;
    if (own.t0 < own.t1) {
      first = a.inst_chunk0[own.inst];
      end = a.inst_chunk0[own.inst + 1];
      iters = L.inst[own.inst].iters;
    }
    for (unsigned left = own.mask; left; left &= left - 1, ++number) {
      const int k = __ffs((int)left) - 1, set = number & 1;
      const int chunk = __shfl_sync(0xffffffffu, own.chunk, k), inst = __shfl_sync(0xffffffffu, own.inst, k);
      const int c0 = __shfl_sync(0xffffffffu, first, k), c1 = __shfl_sync(0xffffffffu, end, k);
      // (the instance's count of iterations, and which sweep: no two sweeps
      // of a solve share a tag)
      const uint32_t tag = 2u * (uint32_t)__shfl_sync(0xffffffffu, iters, k) + OP::kSweep;
      if (ok) ok = bar_wait<POLLS>(&sh.parts_full[set], (number >> 1) & 1);
      bool there = ok;
      if (ok) {
        double sum[K];
#pragma unroll
        for (int j = 0; j < K; ++j) sum[j] = parts_sum(&sh.parts[set][j][lane]);
        __syncwarp();
        unsigned int ticket = 0;
        if (lane == 0) {
          bar_arrive(&sh.parts_empty[set]);
#pragma unroll
          for (int j = 0; j < K; ++j) post_sum(L.mail + j * (int64_t)a.nchunks + chunk, sum[j], tag);
          asm volatile("atom.relaxed.gpu.global.add.u32 %0, [%1], 1;"
                       : "=r"(ticket)
                       : "l"(L.counter + inst * (int64_t)kCounterStride)
                       : "memory");
        }
        if (__shfl_sync(0xffffffffu, ticket, 0) != (unsigned int)(c1 - c0 - 1)) continue;
        double tot[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
          double v = 0.0;
          for (int q = c0 + lane; q < c1; q += 32 * kMailAhead)
            there = read_sums<POLLS>(L.mail + j * (int64_t)a.nchunks + q, (c1 - q + 31) / 32, tag, v) && there;
          tot[j] = warp_total(v);
        }
        there = __all_sync(0xffffffffu, there);
        if (there && lane == 0) {
          L.counter[inst * (int64_t)kCounterStride] = 0u;
          op.finish(L.inst[inst], tot);
        }
      }
      if (!there && lane == 0) give_up(L, inst);
    }
  }
}

}  // namespace
