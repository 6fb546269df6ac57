// IEEE double division and multiplication on the integer and FP32 pipes.
//
// GB300's FP64 pipe runs 1/59 of its FP32 rate: one FP64 instruction of a
// warp holds a scheduler's share of the pipe for 64 cycles, and a division
// issues eight or nine of them.  The same quotient, correctly rounded, takes
// about 45 integer instructions, which the other pipes run in a sixth of that
// time; a product about 45 too, no faster than the machine's, but beside it:
// a kernel bound by the FP64 pipe runs part of its products here.
//
// Division: long division with a 32-bit reciprocal (Knuth, TAOCP vol. 2, 4.3.1:
// a digit estimated from below and corrected by its remainder).  With
// mantissas ma, mb in [2^52, 2^53), ma doubled if below mb, the quotient
// ma / mb lies in [1, 2):
//   R     <= 2^84 / mb, short by less than 4 (FP32 reciprocal approximation,
//            one Newton step in FP32, biased downwards)
//   q1     = floor(floor(ma / 2^22) R / 2^32)      at most 6 below 2^30 ma/mb
//   r1     = 2^30 ma - q1 mb                       in [0, 6 mb): 56 bits
//   q2     = floor(floor(r1 / 2^24) R / 2^37)      at most 1.2 below 2^23 r1/mb
//   r2     = 2^23 r1 - q2 mb                       in [0, 2.2 mb)
//   q      = 2^23 q1 + q2 + (r2 >= mb) = floor(2^53 ma / mb)
// and q + 1 >> 1 is the quotient rounded to nearest: 2^53 ma / mb is never an
// odd integer (mb would have to hold a factor 2^53), so there are no ties.
// Remainders are formed modulo 2^64, which holds them.  Operands or results
// outside the normal range take the machine's division.
//
// Compiled for the host too (the device intrinsics restated), so the
// arithmetic can be checked against the host's own division.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define ESR_HD __host__ __device__ __forceinline__
#else
#define ESR_HD inline
#endif

namespace soft64 {

ESR_HD uint64_t bits(double v) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t u;
  std::memcpy(&u, &v, 8);
  return u;
#endif
}
ESR_HD double value(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double v;
  std::memcpy(&v, &u, 8);
  return v;
#endif
}
ESR_HD uint32_t fbits(float v) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(v);
#else
  uint32_t u;
  std::memcpy(&u, &v, 4);
  return u;
#endif
}
ESR_HD float fvalue(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float v;
  std::memcpy(&v, &u, 4);
  return v;
#endif
}
ESR_HD uint32_t mul_hi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
ESR_HD float fma_f(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}
// 1 / x within 2^-23, x in [1, 2)
ESR_HD float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}

// R of a mantissa (52 fraction bits in hi:lo; exponent and sign bits of hi are
// ignored) from an approximation r0 within 2^-22.  r0 in [1/2, 1) is 2^-24
// times the integer of its mantissa bits; the Newton correction r0 (1 - b r0),
// at most 2^-22, goes to units of 2^-32 through the 1.5 * 2^23 addend; minus 1
// keeps R at or below the exact value (the correction is good to 2^-44).
ESR_HD uint32_t reciprocal(uint32_t hi, uint32_t lo, float r0) {
  const float bh = fvalue((((hi << 3) | (lo >> 29)) & 0x7fffffu) | 0x3f800000u);
  r0 = r0 < 0x1.fffffep-1f ? (r0 > 0.5f ? r0 : 0.5f) : 0x1.fffffep-1f;
  const float bl = fvalue(((lo >> 6) & 0x7fffffu) | 0x3f800000u) - 1.0f;  // times 2^-23
  float e = fma_f(-bh, r0, 1.0f);
  e = fma_f(bl * -0x1p-23f, r0, e);
  const float c = fma_f(r0 * e, 0x1p32f, 12582912.0f);
  return ((fbits(r0) << 8) | 0x80000000u) + (fbits(c) - 0x4b400000u) - 1u;
}

// A divisor prepared for several quotients.
struct Divisor {
  double b;
  uint32_t hi, lo;  // mantissa with its leading bit
  uint32_t r;
  ESR_HD explicit Divisor(double v) : b(v) {
    const uint64_t u = bits(v);
    lo = (uint32_t)u;
    const uint32_t h = (uint32_t)(u >> 32);
    r = reciprocal(h, lo, rcp_approx(fvalue((((h << 3) | (lo >> 29)) & 0x7fffffu) | 0x3f800000u)));
    hi = (h & 0xfffffu) | 0x100000u;
  }
};

ESR_HD double quotient(double a, const Divisor &d) {
  const uint64_t ua = bits(a), ub = bits(d.b);
  const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
  const int32_t ea = (int32_t)((ha >> 20) & 0x7ffu), eb = (int32_t)((hb >> 20) & 0x7ffu);
  const uint64_t mb = ((uint64_t)d.hi << 32) | d.lo;
  uint64_t ma = ((uint64_t)((ha & 0xfffffu) | 0x100000u) << 32) | (uint32_t)ua;
  const bool below = ma < mb;
  ma <<= below ? 1 : 0;
  const uint32_t q1 = mul_hi((uint32_t)(ma >> 22), d.r);
  const uint64_t r1 = (ma << 30) - (uint64_t)q1 * mb;
  const uint32_t q2 = mul_hi((uint32_t)(r1 >> 24), d.r) >> 5;
  const uint64_t r2 = (r1 << 23) - (uint64_t)q2 * mb;
  const uint64_t q = ((uint64_t)q1 << 23) + q2 + (r2 >= mb ? 1u : 0u);
  const int32_t e = ea - eb + 1023 - (below ? 1 : 0);
  const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
  // the leading bit of (q + 1) >> 1 adds one to the exponent field
  const uint64_t out = (((q + 1) >> 1) + ((uint64_t)(uint32_t)(e - 1) << 52)) | sign;
  // normal operands and a result away from the range's ends
  const bool plain = (uint32_t)(ea - 1) < 2046u && (uint32_t)(eb - 1) < 2046u && (uint32_t)(e - 1) < 2045u;
  if (plain) return value(out);
  const bool zero = (ua << 1) == 0 && (uint32_t)(eb - 1) < 2046u;  // 0 / normal
  return zero ? value(sign) : a / d.b;
}

// a * b, rounded to nearest even.  A = 2^11 ma times mb has its 53 result bits
// in the product's upper 64 (one fewer if ma mb < 2^105: all three words move
// up by s) and the fraction to round by in the lower 64.
ESR_HD uint32_t shift_left(uint32_t lo, uint32_t hi, uint32_t s) {  // upper word of hi:lo << s
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)((((uint64_t)hi << 32 | lo) << s) >> 32);
#endif
}

// The machine's product for rare paths, kept out of line: inlined, the
// compiler predicates the one instruction, which then takes the FP64 pipe of
// warps that do not need it.
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
inline
#endif
double machine_product(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

// (mh:ml:t) + r, with e added to the upper word
ESR_HD void round_up(uint32_t &mh, uint32_t &ml, uint32_t t, uint32_t r, uint32_t e) {
#ifdef __CUDA_ARCH__
  asm("{\n.reg .u32 d;\nadd.cc.u32 d, %2, %3;\naddc.cc.u32 %1, %1, 0;\naddc.u32 %0, %0, %4;\n}\n"
      : "+r"(mh), "+r"(ml)
      : "r"(t), "r"(r), "r"(e));
#else
  const uint32_t c = (uint32_t)(((uint64_t)t + r) >> 32);
  const uint64_t m = ((uint64_t)mh << 32 | ml) + c;
  mh = (uint32_t)(m >> 32) + e;
  ml = (uint32_t)m;
#endif
}

ESR_HD double product(double a, double b) {
  const uint64_t ua = bits(a), ub = bits(b);
  const uint32_t ha = (uint32_t)(ua >> 32), la = (uint32_t)ua, hb = (uint32_t)(ub >> 32), lb = (uint32_t)ub;
  // both exponent fields in 512 .. 1534 (factors in [2^-511, 2^512)): the
  // result's, with the carry of the mantissas' product or of the rounding (never
  // both), in 1 .. 2046, always a normal number.  One more on top and 2^512 *
  // 2^512 would run into the infinity pattern and the sign bit.
  if ((ha << 1) - (512u << 21) < (1023u << 21) && (hb << 1) - (512u << 21) < (1023u << 21)) {
    const uint32_t ah = shift_left(la, ha, 11) | 0x80000000u, al = la << 11;
    const uint32_t bh = (hb & 0xfffffu) | 0x100000u;
    const uint64_t p00 = (uint64_t)al * lb;
    const uint64_t p01 = (uint64_t)al * bh + (p00 >> 32);
    const uint64_t p10 = (uint64_t)ah * lb + (uint32_t)p01;
    const uint64_t p11 = (uint64_t)ah * bh + (p01 >> 32) + (p10 >> 32);
    uint32_t mh = (uint32_t)(p11 >> 32), ml = (uint32_t)p11, f1 = (uint32_t)p10, f0 = (uint32_t)p00;
    const uint32_t s = ((mh >> 20) & 1u) ^ 1u;
    mh = shift_left(ml, mh, s);
    ml = shift_left(f1, ml, s);
    f1 = shift_left(f0, f1, s);
    f0 <<= s;
    const uint32_t t = f1 | (f0 != 0 ? 1u : 0u);
    // the leading bit of the mantissa adds one to the exponent field
    const uint32_t e = (ha & 0x7ff00000u) + (hb & 0x7ff00000u) - (1023u << 20) + s * 0xfff00000u;
    round_up(mh, ml, t, 0x7fffffffu + (ml & 1u), e);
    return value((uint64_t)(mh | ((ha ^ hb) & 0x80000000u)) << 32 | ml);
  }
  const bool za = (ua << 1) == 0, zb = (ub << 1) == 0;
  const bool fa = (ha & 0x7ff00000u) != 0x7ff00000u, fb = (hb & 0x7ff00000u) != 0x7ff00000u;
  if ((za && fb) || (zb && fa)) return value((ua ^ ub) & 0x8000000000000000ull);
  return machine_product(a, b);
}

// a / 2: one less in the exponent field (subnormal results: the machine's)
ESR_HD double half(double a) {
  const uint64_t u = bits(a);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
  if (e - 2u < 2045u) return value(u - 0x0010000000000000ull);
  return machine_product(a, 0.5);
}

// -a without the FP64 add the compiler makes of it
ESR_HD double negated(double a) { return value(bits(a) ^ 0x8000000000000000ull); }

// 0 + a: a, with -0 turned into +0
ESR_HD double from_zero(double a) {
  const uint64_t u = bits(a);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const uint32_t kept = ((hi << 1) | lo) == 0 ? 0u : hi;
  return value((uint64_t)kept << 32 | lo);
}

}  // namespace soft64
