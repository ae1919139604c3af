// White noise rounded to FP32, on the FP32 pipes.
//
// The generator (mf_noise.h) is defined by a fixed sequence of FP64
// operations.  An FP32 grid stores its draws rounded to the nearest float, and
// for that the draw is needed only well enough to know which float is nearest.
// normal_pair_f32 evaluates the same draws (the same Philox block, ln, square
// root, sine and cosine) in float pairs (hi, lo), ~2^-41 relative, and accepts
// a result when the whole interval of +-2^-36 around it rounds to one float;
// the FP64 sequence itself is within 2^-49 of the mathematical value, so the
// accepted float is the one that it rounds to.  Otherwise (about 2^-12 of the
// draws) it returns false and the caller evaluates the FP64 sequence.
//
// Why: the sequence takes ~61 FP64 operations per pair at 1.68 per clock and
// SM; the float pairs take ~300 FP32 operations at ~120.  A noise field and its
// potential on a 384^3 grid: 4.60 ms with the FP64 sequence (3.64 ms of it the
// noise), 1.37 ms with the pairs (1.13 ms with the transform passes of today).
#pragma once

#include "mf_noise.h"

namespace mf {
namespace noise {

struct FF {
  float h, l;
};

__device__ __forceinline__ FF ff_quick(float a, float b) {  // a + b exactly, |a| >= |b|
  const float s = __fadd_rn(a, b);
  return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_two(float a, float b) {  // a + b exactly
  const float s = __fadd_rn(a, b), v = __fsub_rn(s, a);
  return FF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v))};
}
__device__ __forceinline__ FF ff_mulp(FF a, FF b) {  // product, not renormalised
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  return FF{p, e};
}
__device__ __forceinline__ FF ff_mulff(FF a, FF b) {
  const FF p = ff_mulp(a, b);
  return ff_quick(p.h, p.l);
}
// c + w x for a term w x no larger than c
__device__ __forceinline__ FF ff_horner(FF c, FF w, FF x) {
  const FF p = ff_mulp(w, x);
  const FF s = ff_quick(c.h, p.h);
  return ff_quick(s.h, __fadd_rn(s.l, __fadd_rn(c.l, p.l)));
}
// signed integer |x| < 2^62 times 2^-sh as a float pair, ~2^-48 relative
__device__ __forceinline__ FF ff_from_int(long long x, int sh) {
  const int a = (int)(x >> 40);                    // 22 bits and the sign
  const int b = (int)((x >> 20) & 0xfffff), c = (int)(x & 0xfffff);
  const FF ab = ff_two((float)a * 1099511627776.0f, (float)b * 1048576.0f);
  const FF s = ff_two(ab.h, __fadd_rn(ab.l, (float)c));
  const float sc = __int_as_float((127 - sh) << 23);
  return FF{s.h * sc, s.l * sc};
}
__device__ __forceinline__ float ff_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ff_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// the float nearest to the pair, if everything within 2^-36 of it agrees
__device__ __forceinline__ bool ff_round(FF z, float* out) {
  const float e = fabsf(z.h) * 0x1p-36f;
  const float lo = __fadd_rn(z.h, __fsub_rn(z.l, e)), hi = __fadd_rn(z.h, __fadd_rn(z.l, e));
  *out = lo;
  return lo == hi;
}

__device__ __forceinline__ bool normal_pair_f32(uint64_t p, uint64_t seed, float* z0, float* z1) {
  uint32_t c[4] = {(uint32_t)(p & 0xFFFFFFFFu), (uint32_t)(p >> 32), 0u, 0u};
  philox4x32_10(c, (uint32_t)(seed & 0xFFFFFFFFu), (uint32_t)(seed >> 32));
  const uint64_t b1 = ((((uint64_t)c[1]) << 32) | c[0]) >> 11;
  const uint64_t b2 = ((((uint64_t)c[3]) << 32) | c[2]) >> 11;
  // u in units of 2^-54: b1 + 1/2 rounded to 53 bits (ties to even from 2^52 on)
  const uint64_t u = (b1 >> 52) ? 2 * (b1 + (b1 & 1)) : 2 * b1 + 1;
  bool ok = (u >> 54) == 0;  // u = 1: the sequence gives a signed zero
  // u = m 2^e, m in [sqrt(1/2), sqrt(2)]; d = m - 1 in units of 2^-62, exact
  const int lz = __clzll((long long)u);
  const uint64_t mi = u << lz;  // m 2^63 in [2^63, 2^64)
  int e = 9 - lz;
  long long di;
  if ((uint32_t)(mi >> 32) > 0xB504F333u) {
    e += 1;
    di = (long long)(mi >> 2) - (1ll << 62);
  } else {
    di = (long long)((mi - (1ull << 63)) >> 1);
  }
  const FF d = ff_from_int(di, 62);
  // s = d / (2 + d); ln m = 2 atanh s = s (2 + 2/3 z + 2/5 z^2 + ...), z = s^2 <= 0.0295
  const FF D0 = ff_quick(2.0f, d.h);
  const FF D = FF{D0.h, __fadd_rn(D0.l, d.l)};
  const float rD = ff_rcp(D.h);
  const float q0 = __fmul_rn(d.h, rD);
  const float rem = __fadd_rn(__fmaf_rn(-q0, D.h, d.h), __fmaf_rn(-q0, D.l, d.l));
  const FF s = ff_quick(q0, __fmul_rn(rem, rD));
  const FF z = ff_mulff(s, s);
  float t = 2.0f / 17.0f;  // terms z^3.. in FP32: z^3 2/7 is 2^-17 of the sum
  t = __fmaf_rn(t, z.h, 2.0f / 15.0f);
  t = __fmaf_rn(t, z.h, 2.0f / 13.0f);
  t = __fmaf_rn(t, z.h, 2.0f / 11.0f);
  t = __fmaf_rn(t, z.h, 2.0f / 9.0f);
  t = __fmaf_rn(t, z.h, 2.0f / 7.0f);
  // coefficients as (float, double - float)
  FF P = ff_horner(FF{0.4f, (float)(0.4 - (double)0.4f)}, z, FF{t, 0.0f});
  P = ff_horner(FF{2.0f / 3.0f, (float)(2.0 / 3.0 - (double)(2.0f / 3.0f))}, z, P);
  P = ff_horner(FF{2.0f, 0.0f}, z, P);
  const FF lm = ff_mulp(s, P);
  constexpr double kLn2 = 0x1.62e42fefa39efp-1;
  constexpr float kLn2h = (float)kLn2, kLn2l = (float)(kLn2 - (double)kLn2h);
  const float ef = (float)e;
  const float ph = __fmul_rn(ef, kLn2h);
  const float pl = __fmaf_rn(ef, kLn2l, __fmaf_rn(ef, kLn2h, -ph));
  const FF L0 = ff_two(ph, lm.h);
  const FF L = ff_quick(L0.h, __fadd_rn(L0.l, __fadd_rn(pl, lm.l)));
  // r = sqrt(-2 ln u)
  const FF x = FF{-2.0f * L.h, -2.0f * L.l};
  const float y = ff_rsqrt(x.h);
  const float r0 = __fmul_rn(x.h, y);
  const float rr = __fadd_rn(__fmaf_rn(-r0, r0, x.h), x.l);
  const FF r = ff_quick(r0, __fmul_rn(rr, __fmul_rn(0.5f, y)));
  // angle: quarter-turn index q and remainder f in [-1/2, 1/2] (sincos_turn53)
  const uint64_t q = (b2 + (1ull << 50)) >> 51;
  const int64_t num = (int64_t)(2 * b2 + 1) - (int64_t)(q << 52);
  const FF f = ff_from_int(num, 52);
  const FF w = ff_mulff(f, f);
  // the Taylor series of sincos_turn53, the terms from w^4 on in FP32 (below 2^-18 of the sums)
#define MF_FFC(v) FF { (float)(v), (float)((v) - (double)(float)(v)) }
  float ts = (float)-0x1.6fadb9f155744p-31;
  ts = __fmaf_rn(ts, w.h, (float)0x1.e8f434d018d63p-25);
  ts = __fmaf_rn(ts, w.h, (float)-0x1.e3074fde8871fp-19);
  ts = __fmaf_rn(ts, w.h, (float)0x1.50783487ee782p-13);
  FF ps = ff_horner(MF_FFC(-0x1.32d2cce62bd86p-8), w, FF{ts, 0.0f});
  ps = ff_horner(MF_FFC(0x1.466bc6775aae2p-4), w, ps);
  ps = ff_horner(MF_FFC(-0x1.4abbce625be53p-1), w, ps);
  ps = ff_horner(MF_FFC(0x1.921fb54442d18p+0), w, ps);
  const FF sn = ff_mulff(f, ps);
  float tc = (float)-0x1.b6e24f44b128fp-28;
  tc = __fmaf_rn(tc, w.h, (float)0x1.f9d38a3763cc3p-22);
  tc = __fmaf_rn(tc, w.h, (float)-0x1.a6d1f2a204a8cp-16);
  tc = __fmaf_rn(tc, w.h, (float)0x1.e1f506891babbp-11);
  FF pc = ff_horner(MF_FFC(-0x1.55d3c7e3cbffap-6), w, FF{tc, 0.0f});
  pc = ff_horner(MF_FFC(0x1.03c1f081b5ac4p-2), w, pc);
  pc = ff_horner(MF_FFC(-0x1.3bd3cc9be45dep+0), w, pc);
  const FF cs = ff_horner(FF{1.0f, 0.0f}, w, pc);
#undef MF_FFC
  // quadrant: (sin, cos) = (s, c), (c, -s), (-s, -c), (-c, s)
  FF a = ff_mulp(r, cs), b = ff_mulp(r, sn);  // the draws for q = 0: r cos, r sin
  const int qq = (int)(q & 3);
  if (qq & 1) {
    const FF sw = a;
    a = b;
    b = sw;
  }
  const float sa = (qq == 1 || qq == 2) ? -1.0f : 1.0f;  // sign of the cosine draw
  const float sb = (qq >= 2) ? -1.0f : 1.0f;             // sign of the sine draw
  a = ff_quick(a.h * sa, a.l * sa);
  b = ff_quick(b.h * sb, b.l * sb);
  ok = ff_round(a, z0) && ok;
  ok = ff_round(b, z1) && ok;
  return ok;
}

// The draws in FP64: the operations of normal_pair (mf_noise.h) that round, in
// its order, with those that are exact done on integers -- the conversions of
// the 53-bit integers, the halving and the powers of two, nine of ~66
// operations on the FP64 pipe, which bounds it.
__device__ __forceinline__ double exact_double(long long x, int sh) {  // x 2^-sh, |x| < 2^53
  const long long s = x >> 63;
  const unsigned long long a = (unsigned long long)((x ^ s) - s);
  const int lz = __clzll((long long)a);
  const long long b = (long long)((a << (lz & 63)) >> 11) + ((long long)(1085 - lz - sh) << 52);
  return __longlong_as_double(a ? (b | (s & (long long)0x8000000000000000ull)) : 0ll);
}
__device__ __forceinline__ void normal_pair_f64(uint64_t p, uint64_t seed, double* z0, double* z1) {
  uint32_t c[4] = {(uint32_t)(p & 0xFFFFFFFFu), (uint32_t)(p >> 32), 0u, 0u};
  philox4x32_10(c, (uint32_t)(seed & 0xFFFFFFFFu), (uint32_t)(seed >> 32));
  const uint64_t b1 = ((((uint64_t)c[1]) << 32) | c[0]) >> 11;
  const uint64_t b2 = ((((uint64_t)c[3]) << 32) | c[2]) >> 11;
  const uint64_t u = (b1 >> 52) ? 2 * (b1 + (b1 & 1)) : 2 * b1 + 1;  // as in normal_pair_f32
  if (u >> 54) {
    normal_pair(p, seed, z0, z1);
    return;
  }
  // log_pos: u = m 2^e
  const int lz = __clzll((long long)u);
  const uint64_t mant = ((u << lz) >> 11) & 0x000FFFFFFFFFFFFFull;
  int e = 9 - lz;
  const bool half = mant > 0x6a09e667f3bcdull;  // m > sqrt(2)
  e += half;
  const double m = from_bits(mant | ((half ? 0x3FEull : 0x3FFull) << 52));
  const double s = div_(sub(m, 1.0), add(m, 1.0));
  const double z = mul(s, s);
  double q = 0x1.642c8590b2164p-4;
  q = fma_(q, z, 0x1.8618618618618p-4);
  q = fma_(q, z, 0x1.af286bca1af28p-4);
  q = fma_(q, z, 0x1.e1e1e1e1e1e1ep-4);
  q = fma_(q, z, 0x1.1111111111111p-3);
  q = fma_(q, z, 0x1.3b13b13b13b14p-3);
  q = fma_(q, z, 0x1.745d1745d1746p-3);
  q = fma_(q, z, 0x1.c71c71c71c71cp-3);
  q = fma_(q, z, 0x1.2492492492492p-2);
  q = fma_(q, z, 0x1.999999999999ap-2);
  q = fma_(q, z, 0x1.5555555555555p-1);
  q = fma_(q, z, 2.0);
  const double ln = fma_(exact_double(e, 0), 0x1.62e42fefa39efp-1, mul(s, q));
  // -2 ln: exact (ln is negative and normal for u < 1)
  const double r = sqrt_(from_bits((bits(ln) ^ 0x8000000000000000ull) + (1ull << 52)));
  // sincos_turn53 with its exact argument
  const uint64_t t = (b2 + (1ull << 50)) >> 51;
  const double f = exact_double((long long)(2 * b2 + 1) - (long long)(t << 52), 52);
  const double w = mul(f, f);
  double ps = -0x1.8a404211f9547p-45;
  ps = fma_(ps, w, 0x1.aaec32af93359p-38);
  ps = fma_(ps, w, -0x1.6fadb9f155744p-31);
  ps = fma_(ps, w, 0x1.e8f434d018d63p-25);
  ps = fma_(ps, w, -0x1.e3074fde8871fp-19);
  ps = fma_(ps, w, 0x1.50783487ee782p-13);
  ps = fma_(ps, w, -0x1.32d2cce62bd86p-8);
  ps = fma_(ps, w, 0x1.466bc6775aae2p-4);
  ps = fma_(ps, w, -0x1.4abbce625be53p-1);
  ps = fma_(ps, w, 0x1.921fb54442d18p+0);
  double pc = -0x1.2a0c591af8314p-41;
  pc = fma_(pc, w, 0x1.20c62c2f2d7f5p-34);
  pc = fma_(pc, w, -0x1.b6e24f44b128fp-28);
  pc = fma_(pc, w, 0x1.f9d38a3763cc3p-22);
  pc = fma_(pc, w, -0x1.a6d1f2a204a8cp-16);
  pc = fma_(pc, w, 0x1.e1f506891babbp-11);
  pc = fma_(pc, w, -0x1.55d3c7e3cbffap-6);
  pc = fma_(pc, w, 0x1.03c1f081b5ac4p-2);
  pc = fma_(pc, w, -0x1.3bd3cc9be45dep+0);
  pc = fma_(pc, w, 1.0);
  const double sn = mul(f, ps);
  const int k = (int)(t & 3);
  const double a = mul(r, (k & 1) ? sn : pc), b = mul(r, (k & 1) ? pc : sn);
  // quadrants: (sin, cos) = (s, c), (c, -s), (-s, -c), (-c, s); signs are exact
  *z0 = (k == 1 || k == 2) ? -a : a;
  *z1 = (k >= 2) ? -b : b;
}

}  // namespace noise
}  // namespace mf
