// FP64 products by a constant on the integer pipe, rounded as __dmul_rn rounds.
//
// This part issues an FP64 warp instruction every 19 cycles an SM, so a trellis
// of many warps is bound by the number of its FP64 instructions, while its
// integer pipes are two thirds idle.  A product's exact 106 bits are four
// 32 x 32-bit products; the rounding to nearest even is one carry.  An addition
// costs about 70 integer instructions (operands to align, sums to normalise), so
// only products are moved: about 26 instructions, 45 cycles of the integer
// pipes, for the 76 FP64 cycles of a DMUL with every scheduler at work.
#pragma once
#include "sdm_internal.h"

#include <cstring>

namespace dsdgpu {

// The range of int_mul's operand: exponents 200 .. 1800 of 0 .. 2046, with
// coefficients between 2^-100 and 2^100, so that every product is normal.
// range_word grows past kRangeSpan outside it (zero, subnormal, infinite, NaN).
constexpr unsigned kRangeLo = 200u << 21, kRangeSpan = (1800u - 200u) << 21;
__device__ __forceinline__ unsigned range_word(double s) {
  return 2u * (unsigned)__double2hiint(s) - kRangeLo;
}

// round(c * s) for s in that range.  With c = C 2^-63 2^(ec - 1023) (C its
// mantissa << 11) and s = S 2^(es - 1075), C S lies in [2^115, 2^117): its upper
// 64 bits hold 52 or 53 bits of the result's mantissa.
__device__ __forceinline__ double int_mul(const IntCoef& c, double s) {
  const unsigned sh = (unsigned)__double2hiint(s), sl = (unsigned)__double2loint(s);
  const unsigned mh = (sh & 0x000fffffu) | 0x00100000u;
  const unsigned long long p0 = (unsigned long long)c.cl * sl;
  const unsigned long long p1 = (unsigned long long)c.ch * sl + (p0 >> 32);
  const unsigned long long p2 = (unsigned long long)c.cl * mh + (unsigned)p1;
  const unsigned long long p3 = (unsigned long long)c.ch * mh + ((p1 >> 32) + (p2 >> 32));
  const unsigned h1 = (unsigned)(p3 >> 32), h0 = (unsigned)p3;
  const unsigned l1 = (unsigned)p2, l0 = (unsigned)p0;
  const unsigned n = h1 & 0x00100000u;        // 53 bits already
  const unsigned k = n ? 0u : 1u;             // else one bit further
  const unsigned r1 = __funnelshift_l(h0, h1, k);
  const unsigned r0 = __funnelshift_l(l1, h0, k);
  const unsigned t = __funnelshift_l(l0, l1, k);
  // what is below: t : l0 (l0's bits only count as "not zero"); up if it is
  // above one half, or one half and r0 odd
  const unsigned half = (l0 | (r0 & 1u)) ? 0x80000000u : 0x7fffffffu;
  unsigned o0, o1;
  asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, 0;\n\t}"
      : "=r"(o0), "=r"(o1)
      : "r"(t), "r"(half), "r"(r0), "r"(r1));
  // the implicit bit of o1 counts one exponent, as does a carry out of the rounding
  const unsigned hi = o1 + n + (sh & 0x7ff00000u) + c.kc;
  return __hiloint2double((int)(hi | ((sh ^ c.sign) & 0x80000000u)), (int)o0);
}

// The same with zeros in the operand's range.
__device__ __forceinline__ bool is_zero(double s) {
  return (2u * (unsigned)__double2hiint(s) | (unsigned)__double2loint(s)) == 0u;
}
__device__ __forceinline__ unsigned range_word0(double s) { return is_zero(s) ? 0u : range_word(s); }
__device__ __forceinline__ double int_mul0(const IntCoef& c, double s) {
  const double r = int_mul(c, s);
  const double z = __hiloint2double((int)(((unsigned)__double2hiint(s) ^ c.sign) & 0x80000000u), 0);
  return is_zero(s) ? z : r;
}

// Whether v may be a coefficient of int_mul, and its form.
inline bool int_coef(double v, IntCoef* c) {
  unsigned long long b;
  memcpy(&b, &v, 8);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  const unsigned long long m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 11;
  c->ch = (unsigned)(m >> 32);
  c->cl = (unsigned)m;
  c->kc = (e - 1024u) << 20;
  c->sign = (unsigned)(b >> 32) & 0x80000000u;
  return e >= 1023 - 100 && e <= 1023 + 100;
}

}  // namespace dsdgpu
