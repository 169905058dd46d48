// mf_ieee64.cuh - FP64 division, square root, comparisons and scalings by
// powers of two on the integer pipes, bit for bit the results of the FP64
// instructions.
//
// GB300 executes 2 FP64 lanes per SM and clock: one FP64 instruction of a warp
// holds the pipe for as long as the other pipes need for some 40 to 80 integer
// instructions.  The library's division takes 7 and its square root 7.3 such
// slots (measured: 576 and 601 clocks per warp and scheduler against 82 for an
// add, a multiply, a fused multiply-add or a comparison in the same loop;
// 77 with the pipe saturated).  div() and root()
// below take 117 and 115 clocks of integer issue when nothing else runs and
// nothing at all beside FP64 arithmetic (four fused multiply-adds and a div()
// take the 320 clocks of the four alone), so a kernel bound by the FP64 pipe
// gets its divisions and roots for free.
//
// div: schoolbook division of the 53-bit significands in two digits (Knuth,
// The Art of Computer Programming vol. 2, 4.3.1) with a 32-bit reciprocal from
// the FP32 approximation and one Newton step, kept below the true value so
// that every partial remainder is >= 0; the last remainder decides the 54th
// bit exactly, and since a quotient of two 53-bit significands is never half
// way between two 53-bit numbers, adding one to the 54-bit floor and dropping
// its last bit rounds to nearest even.  root: the same with the digits of the
// square root.  Operands or results outside the normal range (zero
// denominators, subnormals, infinities, NaN) take the FP64 instruction; a zero
// numerator or radicand is handled here (they are common: vanishing fields).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mf {
namespace ieee64 {

__device__ __forceinline__ uint32_t hi_of(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t lo_of(double x) { return (uint32_t)__double2loint(x); }
__device__ __forceinline__ double pack(uint32_t hi, uint32_t lo) {
  return __hiloint2double((int)hi, (int)lo);
}
__device__ __forceinline__ uint64_t join(uint32_t hi, uint32_t lo) {
  return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ uint32_t rcp_bits(uint32_t b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(b)));
  return __float_as_uint(y);
}
__device__ __forceinline__ uint32_t rsqrt_bits(uint32_t b) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(b)));
  return __float_as_uint(y);
}
__device__ __forceinline__ uint64_t mul32x64(uint32_t a, uint32_t bh, uint32_t bl) {
  return (uint64_t)a * bl + ((uint64_t)(a * bh) << 32);  // mod 2^64
}

// 2^32 / b, low by a relative error below 2^-29.4, for the significand
// (mbh, mbl) = b 2^52, 1 <= b < 2.  The seed (at most 2 units of 2^-24 high,
// from the truncated b, and 1 of the instruction's own error) is lowered by 5
// units, so that 1 - b r0 lies in (0, 2^-20.1) and its leading bits are the
// complement of the product's.
__device__ __forceinline__ uint32_t recip32(uint32_t mbh, uint32_t mbl) {
  const uint32_t b32 = __funnelshift_r(mbl, mbh, 21);
  const uint32_t r0 = (rcp_bits((b32 >> 8) + 0x3f000000u) - 0x3e800005u) << 8;
  const uint64_t p = (uint64_t)r0 * b32;
  const uint32_t e = ~__funnelshift_r((uint32_t)p, (uint32_t)(p >> 32), 12);
  return r0 + (__umulhi(r0, e) >> 19) - 2u;
}

__device__ __forceinline__ double div(double a, double b) {
  const uint32_t ha = hi_of(a), hb = hi_of(b), mal = lo_of(a), mbl = lo_of(b);
  const uint32_t ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u;
  const bool za = ((ha << 1) | mal) == 0u;
  const bool in = (ea - 0x00100000u < 0x7fe00000u) & (ea - eb + 0x3fd00000u < 0x7fb00000u);
  if (!((eb - 0x00100000u < 0x7fe00000u) & (za | in))) return a / b;
  const uint32_t mah = (ha & 0xfffffu) | 0x100000u, mbh = (hb & 0xfffffu) | 0x100000u;
  const uint64_t mb = join(mbh, mbl);
  uint64_t ma = join(mah, mal);
  const uint32_t R = recip32(mbh, mbl);
  const bool lt = ma < mb;
  ma = lt ? ma << 1 : ma;  // 1 <= ma / mb < 2
  // 30 fraction bits of the quotient (at most 6 units low), then 23 more (at
  // most one unit low)
  const uint32_t q1 = __umulhi(__funnelshift_r((uint32_t)ma, (uint32_t)(ma >> 32), 22), R);
  const uint64_t r1 = (ma << 30) - mul32x64(q1, mbh, mbl);
  uint32_t q2 = __umulhi((uint32_t)(r1 >> 24), R) >> 5;
  const uint64_t rem = (r1 << 23) - mul32x64(q2, mbh, mbl);
  q2 += (rem >= mb) ? 2u : 1u;  // the floor, plus one to round
  const uint64_t q = (((uint64_t)q1 << 23) + q2) >> 1;
  const uint32_t sg = (ha ^ hb) & 0x80000000u;
  const uint32_t ex = ea - eb + (lt ? 0x3fd00000u : 0x3fe00000u);
  return za ? pack(sg, 0u) : pack(((uint32_t)(q >> 32) + ex) | sg, (uint32_t)q);
}

__device__ __forceinline__ double root(double x) {
  const uint32_t h = hi_of(x), l = lo_of(x);
  const bool zero = ((h << 1) | l) == 0u;
  if (!((h - 0x00100000u < 0x7fe00000u) | zero)) return ::sqrt(x);
  const bool odd = !(h & 0x00100000u);  // the unbiased exponent
  uint64_t m = join((h & 0xfffffu) | 0x100000u, l);
  const uint32_t frac = __funnelshift_r(l, h, 29) & 0x7fffffu;
  const uint32_t y0 = (rsqrt_bits((odd ? 0x40000000u : 0x3f800000u) | frac) - 0x3e800004u) << 8;
  m = odd ? m << 1 : m;  // v 2^52, 1 <= v < 4
  const uint32_t m32 = __funnelshift_r((uint32_t)m, (uint32_t)(m >> 32), 22);
  // 2^32 / sqrt(v), low by a relative error below 2^-28
  const uint64_t p = (uint64_t)__umulhi(y0, y0) * m32;
  const uint32_t e = ~__funnelshift_r((uint32_t)p, (uint32_t)(p >> 32), 11);
  const uint32_t Y = y0 + (__umulhi(y0, e) >> 20) - 4u;
  // 30 fraction bits of the root, then 23 more (at most one unit low)
  const uint32_t s1 = __umulhi(m32, Y);
  const uint64_t r1 = (m << 8) - (uint64_t)s1 * s1;
  uint32_t s2 = __umulhi((uint32_t)(r1 >> 4), Y) >> 4;
  const uint64_t T = ((uint64_t)s1 << 24) + s2;
  const uint64_t rem = (r1 << 46) - mul32x64(s2, (uint32_t)(T >> 32), (uint32_t)T);
  s2 += (rem > T + s2) ? 2u : 1u;
  const uint64_t s = (((uint64_t)s1 << 23) + s2) >> 1;
  const uint32_t ex = ((((h >> 20) + 1023u) >> 1) - 1u) << 20;
  return zero ? x : pack((uint32_t)(s >> 32) + ex, (uint32_t)s);
}

// a b rounded to nearest even: the 106-bit product of the significands in four
// 32-bit products, its top 64 bits shifted by one where the product of two
// numbers in [1, 2) stays below 2.  About 40 integer instructions; a zero
// factor is handled here, operands or results outside the normal range take the
// FP64 instruction.  Worth it beside FP64 arithmetic only: alone it takes as
// long as the instruction (73 clocks against 77 per warp and scheduler).
__device__ __forceinline__ double mul(double a, double b) {
  const uint32_t ha = hi_of(a), hb = hi_of(b), la = lo_of(a), lb = lo_of(b);
  const uint32_t ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u;
  const bool zero = (((ha << 1) | la) == 0u) | (((hb << 1) | lb) == 0u);
  const bool na = ea - 0x00100000u < 0x7fe00000u, nb = eb - 0x00100000u < 0x7fe00000u;
  // exponent fields' sum in [1024, 3067]: a normal result either way of the shift
  const bool in = na & nb & (((ea >> 1) + (eb >> 1)) - 0x20000000u < 0x3fe00000u);
  if (!(in | (zero & (ea != 0x7ff00000u) & (eb != 0x7ff00000u)))) return a * b;
  const uint32_t Ah = __funnelshift_l(la, ha, 11) | 0x80000000u, Al = la << 11;
  const uint32_t Bh = (hb & 0xfffffu) | 0x100000u;
  const uint64_t t0 = (uint64_t)Al * lb;
  const uint64_t t1 = (uint64_t)Ah * lb + (uint32_t)(t0 >> 32);
  const uint64_t t2 = (uint64_t)Al * Bh + (uint32_t)t1;
  const uint64_t H = (uint64_t)Ah * Bh + (uint32_t)(t1 >> 32) + (uint32_t)(t2 >> 32);
  const uint32_t up = (uint32_t)(H >> 52);  // 1: the product is >= 2
  const uint32_t hh = __funnelshift_l((uint32_t)H, (uint32_t)(H >> 32), 1 - up);
  const uint32_t hl = __funnelshift_l((uint32_t)t2, (uint32_t)H, 1 - up);
  const uint32_t rest = __funnelshift_l((uint32_t)t0, (uint32_t)t2, 1 - up);
  // round up above half, and at half where the last bit is odd
  const uint32_t sticky = (((uint32_t)t0 << (1 - up)) != 0u) | (hl & 1u);
  const uint64_t q = join(hh, hl) + ((rest | sticky) > 0x80000000u ? 1u : 0u);
  const uint32_t ex = ea + eb - 0x40000000u + (up << 20);
  const uint32_t sg = (ha ^ hb) & 0x80000000u;
  return zero ? pack(sg, 0u) : pack(((uint32_t)(q >> 32) + ex) | sg, (uint32_t)q);
}

// Sign-magnitude bits as an ordered integer (-0 and +0 equal): the NaN lie
// outside [-kInf, kInf], so the same 64-bit comparisons keep all of them out,
// those with their payload in the low word too.
constexpr int64_t kInf = 0x7ff0000000000000ll;
__device__ __forceinline__ int64_t key(double x) {
  const int64_t s = (int64_t)((int32_t)hi_of(x) >> 31);
  return ((int64_t)join(hi_of(x) & 0x7fffffffu, lo_of(x)) ^ s) - s;
}
__device__ __forceinline__ bool lt(double a, double b) {
  const int64_t ka = key(a), kb = key(b);
  return (ka < kb) & (ka >= -kInf) & (kb <= kInf);
}
__device__ __forceinline__ bool le(double a, double b) {
  const int64_t ka = key(a), kb = key(b);
  return (ka <= kb) & (ka >= -kInf) & (kb <= kInf);
}
__device__ __forceinline__ double absval(double x) { return pack(hi_of(x) & 0x7fffffffu, lo_of(x)); }
// x with its sign changed where the top bit of s is set
__device__ __forceinline__ double flip(double x, uint32_t s) {
  return pack(hi_of(x) ^ (s & 0x80000000u), lo_of(x));
}
// fmax: the other operand where one is NaN
__device__ __forceinline__ double maxnum(double a, double b) {
  const int64_t ka = key(a), kb = key(b);
  return ((ka < kb) & (kb <= kInf)) | (ka > kInf) ? b : a;
}
__device__ __forceinline__ double minnum(double a, double b) {
  const int64_t ka = key(a), kb = key(b);
  return ((kb < ka) & (kb >= -kInf)) | (ka < -kInf) ? b : a;
}

// x 2^K (|K| <= 8): the exponent moved, where x and the result are normal or
// x is zero; else the multiplication.
template <int K>
__device__ __forceinline__ double scale(double x) {
  const uint32_t h = hi_of(x), e = h & 0x7ff00000u;
  const uint32_t first = (K < 0) ? (uint32_t)(1 - K) << 20 : 1u << 20;
  const uint32_t count = (uint32_t)(2046 - (K < 0 ? -K : K)) << 20;
  if (e - first < count) return pack(h + ((uint32_t)K << 20), lo_of(x));
  if (((h << 1) | lo_of(x)) == 0u) return x;
  return x * (K < 0 ? 1.0 / (1 << (K < 0 ? -K : 0)) : (double)(1 << (K < 0 ? 0 : K)));
}
__device__ __forceinline__ double half(double x) { return scale<-1>(x); }

// minmod of two differences (reconstructionF.ChF:5-13): the one of smaller
// magnitude where the signs agree, else a zero of a's sign.  As in the FP64
// form, sign(a) max(0, min(|a|, sign(a) b)), a NaN gives way to the other
// difference: a where b alone is NaN, b or zero by the signs where a alone is,
// a zero where both are.  (A NaN has the larger magnitude; differences are
// quiet NaN, whose high word tells.)
__device__ __forceinline__ double minmod(double a, double b) {
  const uint32_t ha = hi_of(a), hb = hi_of(b);
  const uint64_t ua = join(ha & 0x7fffffffu, lo_of(a)), ub = join(hb & 0x7fffffffu, lo_of(b));
  const bool first = ua <= ub;
  const uint32_t h = first ? ha : hb, l = first ? lo_of(a) : lo_of(b);
  const bool take = ((int32_t)(ha ^ hb) >= 0) | ((hb & 0x7fffffffu) > 0x7ff00000u);
  const bool keep = take & ((h & 0x7fffffffu) <= 0x7ff00000u);
  return pack(keep ? h : ha & 0x80000000u, keep ? l : 0u);
}

}  // namespace ieee64
}  // namespace mf
