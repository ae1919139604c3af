// FP64 line transforms in 64-bit fixed point.
//
// The device issues 1.68 FP64 operations per clock and SM but ~42 64-bit
// integer additions and ~53 32x32+64 multiply-adds (measured), so a line FFT
// of FP64 values runs on the integer pipes: the line is converted to
// q = round(x 2^xs), transformed with exact additions and twiddle products of
// 62-bit twiddles, and converted back.
//
// Scale.  Every value inside an unnormalised DFT is a sum of inputs times
// phases, so its modulus is at most the line's L1 norm.  xs places an upper
// bound of that norm (moduli as max + 0.4142 min of the components, at most 8 %
// too large) at 1.3125 2^62, less the growth of a pre- or post-processing step:
// the sums of two components inside radix 8 stay below 2^63 then, so nothing
// overflows and no stage needs a shift.  xs is lower where a single value would
// pass 2^62.
//
// Error.  In units of 2^-xs a conversion is off by at most 1/2, a twiddle
// product by 0.55 r.m.s. and at most 2.3 (the rounding and two products of low
// words that are left out), a product with sqrt(3)/2 by at most 1.12.  The
// largest terms are the conversions of a long line: a unit is 2^-62 to 2^-61 of
// the L1 norm, which for L white values is 1.25 L of one's r.m.s.; the one or two
// bits of growth of the real transforms make it two or four times as large.
// Measured, relative L2 of a product with a field of one mode, the largest of
// eight amplitudes, and what FP64 butterflies left: N=64 1.3e-16 / 3.2e-16, 128
// 3.8 / 5.1, 256 1.3 / 3.5, 384 2.2 / 3.9, 512 (L = 768) 5.4 / 5.9.  With the norm
// from |re| + |im| at 2^62 it was 7.1e-16 at N=512, more than the butterflies.
//
// Forward transforms of white values against extended precision: 0.9e-16 at
// N=256, 1.0e-16 at 384, 1.4e-16 at 512, where FP64 butterflies are 3.6e-16, 2.8e-16
// and 3.3e-16 off.
//
// Time (N=256, FP64): z c2r of a padded operand 1734 -> 386 us, y c2r 1000
// -> 262 us per operand, a 3LPT run 114.0 -> 35.0 ms (32.0 with the cheaper
// operand factors and sources since).  What bounds it now is instruction
// issue: ~100 instructions per element in the butterflies, ~100 in conversions.
//
// Lines holding an infinity or a NaN come out NaN.  The norm of a line outside
// the float range that it is summed in is summed again relative to its largest
// exponent, and extreme results are scaled by FP64 products: like FP64
// arithmetic, the transform commutes with powers of two.
#pragma once

#include <cmath>
#include <type_traits>

#include "mf_fft.cuh"

namespace mf {

template <> struct cplx_of<long long> { using type = longlong2; };

namespace fx {

constexpr int kNan = 1 << 20;  // scale of a line that holds no finite result

// twiddle component w, |w| <= 1, as q = round(w 2^62) split into a signed low
// word and the matching high word (the form cmul reads)
__host__ inline long long split_q62(long double w) {
  long long q = llroundl(w * 4611686018427387904.0L);
  int lo = (int)(unsigned)(q & 0xffffffffll);
  if (lo == (int)0x80000000) { ++q; ++lo; }  // so that -lo exists
  const long long hi = (q - (long long)lo) >> 32;
  return (long long)(((unsigned long long)hi << 32) | (unsigned)lo);
}

__device__ __forceinline__ int lo32(long long a) { return (int)(unsigned)(unsigned long long)a; }
__device__ __forceinline__ int hi32(long long a) { return (int)(a >> 32); }
__device__ __forceinline__ long long wide(int a, int b) {
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ long long mad(int a, int b, long long c) {  // a b + c
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
// a split into a signed low word and the matching high word
__device__ __forceinline__ void split(long long a, int& h, int& l) {
  l = lo32(a);
  h = hi32(a) + (int)((unsigned)l >> 31);
}
// (h 2^64 + m 2^32) / 2^62 for |h 2^2| < 2^63
__device__ __forceinline__ long long join(long long h, long long m) {
  const long long u = mad(hi32(m), 1, h);  // h 2^32 + m, its upper 64 bits
  const unsigned lo = __funnelshift_l((unsigned)lo32(m), (unsigned)lo32(u), 2);
  const unsigned hi = __funnelshift_l((unsigned)lo32(u), (unsigned)hi32(u), 2);
  return (long long)(((unsigned long long)hi << 32) | lo);
}
// a c / 2^62 rounded, for a constant c in Q62, |a| < 2^63 (the product of the
// low words, up to 0.62 units at sqrt(3)/2, is left out: both are signed)
__device__ __forceinline__ long long mulc(long long a, int ch, int cl) {
  int ah, al;
  split(a, ah, al);
  return join(wide(ah, ch), mad(ah, cl, mad(al, ch, 1ll << 29)));
}

// upper bound of |x| 2^(896-off) as a float: the exponent rebased and the
// mantissa rounded up; 0 below the float range, infinity or NaN above it
__device__ __forceinline__ float mag(int hi_abs, int off = 896) {
  int h = hi_abs - off * 0x100000;
  h = max(h, 0);
  h = min(h, 0x0ff00000);
  return __int_as_float((h << 3) + 8);
}
__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }

// bound of the modulus from the components' high words, a >= b
__device__ __forceinline__ float modulus(int a, int b, int off = 896) {
  return fmaf(mag(b, off), 0.41421357f, mag(a, off));  // sqrt(2) - 1, rounded up
}
// bound of a line: sum of the moduli times 2^-base, largest high word
struct Norm {
  float l1 = 0.f;
  int mx = 0;
  int base = 0;
  __device__ __forceinline__ void add(double2 v) {
    const int a = hi_abs(v.x), b = hi_abs(v.y), m = max(a, b);
    l1 += modulus(m, min(a, b));
    mx = max(mx, m);
  }
  // term of the sum relative to the largest exponent (of this, the line's norm)
  __device__ __forceinline__ float rebased(double2 v) const {
    const int a = hi_abs(v.x), b = hi_abs(v.y);
    return modulus(max(a, b), min(a, b), (mx >> 20) - 127);
  }
  __device__ __forceinline__ void add(const Norm& o) {
    l1 += o.l1;
    mx = max(mx, o.mx);
  }
  __device__ __forceinline__ Norm shfl_xor(int o) const {
    Norm r;
    r.l1 = __shfl_xor_sync(0xffffffffu, l1, o);
    r.mx = __shfl_xor_sync(0xffffffffu, mx, o);
    return r;
  }
  __device__ __forceinline__ bool in_range() const { return l1 > 0x1p-100f && l1 < 0x1p120f; }
  // whether the moduli are to be summed again relative to the largest
  // exponent; of a part of a line: if no part's are, the whole is in range
  __device__ __forceinline__ bool sum_again() const { return mx != 0 && !(l1 > 0x1p-100f && l1 < 0x1p110f); }
  // the result of that; lines of subnormal or with non-finite values keep theirs
  __device__ __forceinline__ void set_rebased(float sum) {
    const int e = mx >> 20;
    if (in_range() || e == 0 || e == 0x7ff) return;
    l1 = sum;
    base = e - 1023;
  }
};

// scale of a line from its norm; grow: bits of growth of the processing around
// the transform
__device__ __forceinline__ int scale(const Norm& n, int len_bits, int grow) {
  if (n.in_range()) {
    // l1 (1 + 2^-6) covers the rounding of the float sum; at most 1.3125 2^62,
    // and 2^62 for the largest value (from_double)
    const int X = (__float_as_int(n.l1 * (1.015625f / 1.3125f)) >> 23) - 126;
    return min(62 - grow - X - n.base, 1084 - max(n.mx >> 20, 1));
  }
  // every value below 2^(e-1022), subnormal ones among them
  int e = n.mx >> 20;
  if (e == 0x7ff) return kNan;
  if (e == 0) e = max(12 - __clz(n.mx), -(grow + len_bits));  // (xs <= 1083: from_double)
  return 62 - grow - (e - 1022 + 1 + len_bits);
}

// round(x 2^xs) for |x| 2^xs < 2^62, xs <= 1083
__device__ __forceinline__ long long from_double(double x, int xs) {
  const int hi = __double2hiint(x), h = hi & 0x7fffffff;
  const unsigned lo = (unsigned)__double2loint(x);
  // |x| = m 2^(e-1084) for the 53-bit mantissa m at bits 10..62 (normal or, e = 0,
  // subnormal), shifted right to twice the value (a count of 64 or more leaves 0)
  const int e = max((h >> 20) - 1, 0);
  const unsigned mh = __funnelshift_l(lo, (unsigned)(h - (e << 20)), 10);
  const unsigned long long m = ((unsigned long long)mh << 32) | (lo << 10);
  const unsigned r = (unsigned)(1083 - xs - e);
  unsigned long long q;
  asm("shr.u64 %0, %1, %2;" : "=l"(q) : "l"(m), "r"(r));
  const long long s = (long long)(hi >> 31);
  // (q + 1) / 2 for a positive value, floor(-q / 2) for a negative one: halves away from zero
  return (((long long)q ^ s) + 1) >> 1;
}

// q 2^-xs, rounded to the nearest double, for any scale and |q| < 2^63
static __device__ __noinline__ double to_double_any(long long q, int xs) {
  if (xs >= kNan) return __longlong_as_double(0x7ff8000000000000ll);
  double d = (double)q;
  int k = -xs;
  while (k > 1000) { d *= 0x1p1000; k -= 1000; }
  while (k < -1000) { d *= 0x1p-1000; k += 1000; }
  return d * __hiloint2double((1023 + k) << 20, 0);
}
__device__ __forceinline__ double to_double(long long q, int xs) {
  const int s = hi32(q) >> 31;
  const unsigned long long a = (unsigned long long)((q ^ (long long)s) - (long long)s);
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
  // |q| < 2^32 (zeros among them) and unusual scales
  if (ah == 0u || (unsigned)(xs + 900) > 1800u) return q == 0 && xs < kNan ? 0.0 : to_double_any(q, xs);
  const int lz = __clz((int)ah);  // 1..31
  // bit 62 set, rounded to 53 bits (or 2^53)
  const unsigned nh = __funnelshift_l(al, ah, lz - 1), nl = al << (lz - 1);
  const unsigned long long m = ((((unsigned long long)nh << 32) | nl) + 0x200) >> 10;
  const unsigned hi = (unsigned)(m >> 32) + ((unsigned)(1085 - xs) << 20) - ((unsigned)lz << 20);
  return __hiloint2double((int)(hi | ((unsigned)s & 0x80000000u)), (int)(unsigned)m);
}

__device__ __forceinline__ longlong2 from_c(double2 v, int xs) {
  return make_longlong2(from_double(v.x, xs), from_double(v.y, xs));
}
__device__ __forceinline__ double2 to_c(longlong2 v, int xs) {
  return make_double2(to_double(v.x, xs), to_double(v.y, xs));
}

__host__ __device__ constexpr int ceil_log2(int n) {
  int b = 0;
  while ((1 << b) < n) ++b;
  return b;
}

}  // namespace fx

// complex products of a fixed-point value with a split Q62 twiddle: four
// 32x32 products per component are summed in 64 bits before one rounding
// shift, two more carry the high words
__device__ __forceinline__ longlong2 fx_cmul(longlong2 a, int wxh, int wxl, int wyh, int wyl) {
  int axh, axl, ayh, ayl;
  fx::split(a.x, axh, axl);
  fx::split(a.y, ayh, ayl);
  const int nyh = -wyh, nyl = -wyl;
  const long long half = 1ll << 29;
  const long long mr = fx::mad(axh, wxl, fx::mad(axl, wxh, fx::mad(ayh, nyl, fx::mad(ayl, nyh, half))));
  const long long hr = fx::mad(axh, wxh, fx::wide(ayh, nyh));
  const long long mi = fx::mad(axh, wyl, fx::mad(axl, wyh, fx::mad(ayh, wxl, fx::mad(ayl, wxh, half))));
  const long long hi = fx::mad(axh, wyh, fx::wide(ayh, wxh));
  return make_longlong2(fx::join(hr, mr), fx::join(hi, mi));
}
template <>
__device__ __forceinline__ longlong2 cmul<longlong2>(longlong2 a, longlong2 w) {
  return fx_cmul(a, fx::hi32(w.x), fx::lo32(w.x), fx::hi32(w.y), fx::lo32(w.y));
}
// a * conj(w)
template <>
__device__ __forceinline__ longlong2 cmulc<longlong2>(longlong2 a, longlong2 w) {
  return fx_cmul(a, fx::hi32(w.x), fx::lo32(w.x), -fx::hi32(w.y), -fx::lo32(w.y));
}

// radix-3 and radix-8 butterflies: constants in Q62, halving by a shift that
// rounds ties to even (a plain shift would leave the same quarter unit in
// every output)
namespace fx {
constexpr int kS32h = 0x376cf5d1, kS32l = -1332128537;  // sqrt(3)/2
constexpr int kS12h = 0x2d413ccd, kS12l = -25716447;    // 1/sqrt(2)
__device__ __forceinline__ long long half_even(long long s) { return (s + ((lo32(s) >> 1) & 1)) >> 1; }
template <bool INV>
__device__ __forceinline__ void dft3(longlong2* a) {
  const longlong2 s = cadd(a[1], a[2]), d = csub(a[1], a[2]);
  const longlong2 m = make_longlong2(a[0].x - half_even(s.x), a[0].y - half_even(s.y));
  a[0] = cadd(a[0], s);
  longlong2 r = cmul_mi<INV>(d);
  r.x = mulc(r.x, kS32h, kS32l);
  r.y = mulc(r.y, kS32h, kS32l);
  a[1] = cadd(m, r);
  a[2] = csub(m, r);
}
template <bool INV>
__device__ __forceinline__ void dft8(longlong2* a) {
  longlong2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
  longlong2 o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
  dft4v<long long, INV>(e0, e1, e2, e3);
  dft4v<long long, INV>(o0, o1, o2, o3);
  longlong2 w1, w2, w3;
  if (!INV) {
    w1 = make_longlong2(mulc(o1.x + o1.y, kS12h, kS12l), mulc(o1.y - o1.x, kS12h, kS12l));
    w2 = make_longlong2(o2.y, -o2.x);
    w3 = make_longlong2(mulc(o3.y - o3.x, kS12h, kS12l), mulc(-(o3.x + o3.y), kS12h, kS12l));
  } else {
    w1 = make_longlong2(mulc(o1.x - o1.y, kS12h, kS12l), mulc(o1.x + o1.y, kS12h, kS12l));
    w2 = make_longlong2(-o2.y, o2.x);
    w3 = make_longlong2(mulc(-(o3.x + o3.y), kS12h, kS12l), mulc(o3.x - o3.y, kS12h, kS12l));
  }
  a[0] = cadd(e0, o0); a[4] = csub(e0, o0);
  a[1] = cadd(e1, w1); a[5] = csub(e1, w1);
  a[2] = cadd(e2, w2); a[6] = csub(e2, w2);
  a[3] = cadd(e3, w3); a[7] = csub(e3, w3);
}
}  // namespace fx
template <> __device__ __forceinline__ void dft3<long long, false>(longlong2* a) { fx::dft3<false>(a); }
template <> __device__ __forceinline__ void dft3<long long, true>(longlong2* a) { fx::dft3<true>(a); }
template <> __device__ __forceinline__ void dft8<long long, false>(longlong2* a) { fx::dft8<false>(a); }
template <> __device__ __forceinline__ void dft8<long long, true>(longlong2* a) { fx::dft8<true>(a); }

// ---------------------------------------------------------------------------
// the transforms of the kernels: FP32 lines as they are, FP64 lines in fixed
// point.  `tw` of an FP64 transform of length L is followed by its L
// fixed-point twiddles (TwiddleCache).
// ---------------------------------------------------------------------------
template <int L>
__device__ __forceinline__ const longlong2* fx_table(const double2* tw) {
  return reinterpret_cast<const longlong2*>(tw + L);
}

// partial norms that the threads of a CTA exchange: one block of shared memory
// per kernel, however many transforms it has (a second one cost the fused z pass
// at H = 144 a CTA per SM, 6 % of five products at 192^3)
template <int COUNT>
struct NormParts {
  float l1[COUNT];
  int mx[COUNT];
};
template <int COUNT>
__device__ __forceinline__ NormParts<COUNT>& norm_parts() {
  __shared__ NormParts<COUNT> p;
  return p;
}

// norm of each column of a strided tile, block (NCOL, TPL), to all its threads.
// each(f) calls f with every value of the thread.
template <int NCOL, int TPL, class EACH>
__device__ __forceinline__ fx::Norm col_norm(int t, int c, EACH each) {
  constexpr bool WARP = NCOL < 32;  // a warp holds 32 / NCOL elements of a column
  constexpr int ROWS = WARP ? (NCOL * TPL + 31) / 32 : TPL;
  float* l1 = norm_parts<ROWS * NCOL>().l1;
  int* mx = norm_parts<ROWS * NCOL>().mx;
  fx::Norm n;
  each([&](double2 v) { n.add(v); });
  if constexpr (WARP) {
#pragma unroll
    for (int o = NCOL; o < 32; o <<= 1) n.add(n.shfl_xor(o));
  }
  const int row = WARP ? (t * NCOL + c) >> 5 : t;
  l1[row * NCOL + c] = n.l1;  // (a warp's lanes of one column write the same values)
  mx[row * NCOL + c] = n.mx;
  const bool again = __syncthreads_or(n.sum_again());
  fx::Norm r;
#pragma unroll 8
  for (int i = 0; i < ROWS; ++i) {
    r.l1 += l1[i * NCOL + c];
    r.mx = max(r.mx, mx[i * NCOL + c]);
  }
  if (again) {
    float s = 0.f;
    each([&](double2 v) { s += r.rebased(v); });
    if constexpr (WARP) {
#pragma unroll
      for (int o = NCOL; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    __syncthreads();  // the first sums have been read
    l1[row * NCOL + c] = s;
    __syncthreads();
    s = 0.f;
    for (int i = 0; i < ROWS; ++i) s += l1[i * NCOL + c];
    r.set_rebased(s);
  }
  return r;
}

// Transform of the columns of a tile of double2 in fixed point, exchanged in
// the tile, F the FP64 plan: on entry every thread's own elements (t + i TPL,
// i < E) hold the inputs, on exit its own elements hold the outputs q, value
// q 2^-xs with the returned xs.  The conversions run as rolled loops over the
// tile: unrolled over registers they are ~1000 instructions each, and the
// kernels then waited on instruction fetch (3.7 of 8 stall cycles per issue).
template <class F, int NCOL>
__device__ __forceinline__ int tile_slot(int t, int i) {
  return pidx<F::kLayout>(t + i * F::TPL) * NCOL;
}
template <class F, int NCOL>
__device__ __forceinline__ void col_fx_run(longlong2* tile, int t, int c, const double2* tw) {
  using FX = typename F::template with_type<long long>;
  longlong2 q[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) q[s] = tile[F::in_slot(t, s) * NCOL + c];
  FX::run(q, t, tile + c, NCOL, fx_table<F::LEN>(tw), SyncBlock{});
  __syncthreads();  // the last exchange has been read
#pragma unroll
  for (int s = 0; s < F::E; ++s) tile[F::out_slot(t, s) * NCOL + c] = q[s];
}
template <class F, int NCOL>
__device__ __forceinline__ int col_fx(double2* tile, int t, int c, const double2* tw) {
  longlong2* tx = reinterpret_cast<longlong2*>(tile);
  const fx::Norm n = col_norm<NCOL, F::TPL>(t, c, [&](auto f) {
#pragma unroll 2
    for (int i = 0; i < F::E; ++i) f(tile[tile_slot<F, NCOL>(t, i) + c]);
  });
  const int xs = fx::scale(n, fx::ceil_log2(F::LEN), 0);
#pragma unroll 2
  for (int i = 0; i < F::E; ++i) {
    const int o = tile_slot<F, NCOL>(t, i) + c;
    tx[o] = fx::from_c(tile[o], xs);
  }
  col_fx_run<F, NCOL>(tx, t, c, tw);
  return xs;
}

// norm of each line of a contiguous-line pass, TPL threads per line, to all of
// them.  Summed in an order that is fixed by the line alone: the sum decides the
// scale, so another order could round every output of the line differently.
// (At most 256 threads per CTA; the callers have a barrier between two calls.)
template <int TPL, class SYNC, class EACH>
__device__ __forceinline__ fx::Norm line_norm(int t, int lg, SYNC sync, EACH each) {
  fx::Norm n;
  each([&](double2 v) { n.add(v); });
  auto again = [&](const fx::Norm& m) {
    float s = 0.f;
    each([&](double2 v) { s += m.rebased(v); });
    return s;
  };
  if constexpr (std::is_same<SYNC, SyncWarp>::value) {
#pragma unroll
    for (int o = 1; o < TPL; o <<= 1) n.add(n.shfl_xor(o));
    if (__any_sync(0xffffffffu, n.sum_again())) {
      float s = again(n);
#pragma unroll
      for (int o = 1; o < TPL; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      n.set_rebased(s);
    }
    return n;
  } else {
    float* l1 = norm_parts<256>().l1;
    int* mx = norm_parts<256>().mx;
    l1[lg * TPL + t] = n.l1;
    mx[lg * TPL + t] = n.mx;
    const bool any = __syncthreads_or(n.sum_again());
    fx::Norm r;
#pragma unroll
    for (int i = 0; i < TPL; ++i) {
      r.l1 += l1[lg * TPL + i];
      r.mx = max(r.mx, mx[lg * TPL + i]);
    }
    if (any) {
      const float s = again(r);
      sync();  // the first sums have been read
      l1[lg * TPL + t] = s;
      sync();
      float sum = 0.f;
      for (int i = 0; i < TPL; ++i) sum += l1[lg * TPL + i];
      r.set_rebased(sum);
    }
    return r;
  }
}

// a staged half-complex line (kin values, kz >= kin zero) to fixed point in
// place; returns its scale.  A c2r ignores the imaginary parts of kz = 0 and
// kz = H, however large they are: they count in neither the norm nor the
// transform.
template <int H, int TPL, class SYNC>
__device__ __forceinline__ int c2r_line_to_fx(double2* src, int kin, int t, int lg, SYNC sync) {
  const fx::Norm n = line_norm<TPL>(t, lg, sync, [&](auto f) {
#pragma unroll 2
    for (int k = t; k < kin; k += TPL) {
      double2 v = src[k];
      if (k == 0 || k == H) v.y = 0.0;
      f(v);
    }
  });
  // inputs of the transform are E + iO: at most twice the moduli of two terms each
  const int xs = fx::scale(n, fx::ceil_log2(H), 2);
#pragma unroll 2
  for (int k = t; k < kin; k += TPL) {
    longlong2 q = fx::from_c(src[k], xs);
    if (k == 0 || k == H) q.y = 0;
    reinterpret_cast<longlong2*>(src)[k] = q;
  }
  sync();
  return xs;
}

// a staged line of H real pairs in layout LIN to fixed point in place;
// returns its scale (the post-processing doubles the values)
template <int H, int TPL, int LIN, class SYNC>
__device__ __forceinline__ int r2c_line_to_fx(double2* src, int t, int lg, SYNC sync) {
  const fx::Norm n = line_norm<TPL>(t, lg, sync, [&](auto f) {
#pragma unroll 2
    for (int k = t; k < H; k += TPL) f(src[pidx<LIN>(k)]);
  });
  const int xs = fx::scale(n, fx::ceil_log2(H), 1);
#pragma unroll 2
  for (int k = t; k < H; k += TPL)
    reinterpret_cast<longlong2*>(src)[pidx<LIN>(k)] = fx::from_c(src[pidx<LIN>(k)], xs);
  return xs;
}

// one c2r pre-processed input of the half-length transform
template <int H>
__device__ __forceinline__ longlong2 c2r_pre_fx(const longlong2* src, int k, int kin,
                                                const longlong2* __restrict__ twM) {
  const longlong2 A = (k < kin) ? src[k] : make_longlong2(0, 0);
  const longlong2 B = (H - k < kin) ? cconj(src[H - k]) : make_longlong2(0, 0);
  const longlong2 Ev = cadd(A, B);
  const longlong2 Ov = cmulc(csub(A, B), twM[k]);
  return make_longlong2(Ev.x - Ov.y, Ev.y + Ov.x);
}
// r2c post-processing: twice E + w O from Z[k] and Z[H-k]
__device__ __forceinline__ longlong2 r2c_post_fx(longlong2 zk, longlong2 zh, longlong2 w) {
  const longlong2 zc = cconj(zh);
  const longlong2 d = csub(zk, zc);
  return cadd(cadd(zk, zc), cmul(make_longlong2(d.y, -d.x), w));
}

// c2r of a staged line in fixed point (c2r_line_to_fx) into the line area xl:
// on exit every thread's own elements (t + i TPL) hold the outputs.  xl may be
// src itself (it is read before the first exchange).
template <class F, int H, class SYNC>
__device__ __forceinline__ void c2r_line_fx(const longlong2* src, int kin, longlong2* xl, int t, const double2* twH,
                                            const double2* twM, SYNC sync) {
  using FX = typename F::template with_type<long long>;
  longlong2 q[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) q[s] = c2r_pre_fx<H>(src, F::in_index(t, s), kin, fx_table<2 * H>(twM));
  FX::run(q, t, xl, 1, fx_table<H>(twH), sync);
  sync();
#pragma unroll
  for (int s = 0; s < F::E; ++s) xl[F::out_slot(t, s)] = q[s];
}
// forward transform of a staged line of H pairs in fixed point, src (layout
// LIN) into xl, which may be src; the outputs are visible to the line on exit
template <class F, int H, int LIN, class SYNC>
__device__ __forceinline__ void r2c_line_fx(const longlong2* src, longlong2* xl, int t, const double2* twH, SYNC sync) {
  using FX = typename F::template with_type<long long>;
  longlong2 q[F::E];
#pragma unroll
  for (int s = 0; s < F::E; ++s) q[s] = src[pidx_split<LIN>(t, F::in_const(s), F::TBITS)];
  FX::run(q, t, xl, 1, fx_table<H>(twH), sync);
  sync();
#pragma unroll
  for (int s = 0; s < F::E; ++s) xl[F::out_slot(t, s)] = q[s];
  sync();
}
// output k of the r2c of a transformed line
template <int H, int LAY>
__device__ __forceinline__ double2 r2c_line_out(const longlong2* xl, int k, int xs, const double2* twM) {
  const longlong2 zk = xl[pidx<LAY>(k == H ? 0 : k)], zh = xl[pidx<LAY>(k == 0 || k == H ? 0 : H - k)];
  return fx::to_c(r2c_post_fx(zk, zh, fx_table<2 * H>(twM)[k]), xs + 1);
}

}  // namespace mf
