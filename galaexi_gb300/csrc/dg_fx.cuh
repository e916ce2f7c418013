// Block fixed-point arithmetic on the integer pipes, for the FP64 form.
//
// GB300 issues two FP64 instructions per clock and SM: a warp-wide FP64 instruction holds its
// sub-partition for 64 cycles (65 measured, for DFMA and for the FP64 <-> integer conversions alike),
// a 32 x 32 -> 64-bit multiply-add (IMAD.WIDE) for 2, a 64-bit addition for 3.  The kernels built on
// this header hold the values of one element as 64-bit integers with one power-of-two scale per
// quantity and element, X = x * 2^s, chosen from the element's largest magnitude so that |X| < 2^59 .. 2^61:
// 6 to 8 more significant bits than a double of the largest magnitude, and every value within that factor
// of it is held exactly.  Sums are exact; a product keeps the upper 64 bits, after a shift that uses the
// range up, of the 128-bit product (three multiply-adds; the low x low partial product is dropped).  A
// product costs about 14 cycles and a sum 3, instead of 65 each.
//
// Values are split into limbs (h, l), X = h 2^32 + l with l signed, so that all partial products are
// signed 32 x 32 products.  The bounds that keep every intermediate value inside 64 bits are stated
// where the scales are chosen.
#pragma once
#include <cuda_runtime.h>

namespace gx {

typedef long long fx64;

struct FxLimb {
  int h, l;
};
__device__ __forceinline__ FxLimb fx_limb(fx64 x) {
  const int l = (int)x;
  return {(int)(x >> 32) - (l >> 31), l};
}
// the limbs of x + y from xh = x + 2^31: the carry of the lower words then rounds the upper limb
constexpr fx64 kFxHalf = 1ll << 31;
__device__ __forceinline__ FxLimb fx_sum(fx64 xh, fx64 y) {
  const fx64 s = (fx64)((unsigned long long)xh + (unsigned long long)y);
  return {(int)(s >> 32), (int)s ^ (int)0x80000000};
}
// (sums wrap: the biased partial sums below use the whole 64 bits)
__device__ __forceinline__ fx64 fx_add(fx64 a, fx64 b) { return (fx64)((unsigned long long)a + (unsigned long long)b); }
__device__ __forceinline__ fx64 fx_sub(fx64 a, fx64 b) { return (fx64)((unsigned long long)a - (unsigned long long)b); }
// a * b + c as one instruction (the expression in C++ came out as up to eight)
__device__ __forceinline__ fx64 fx_mad(int a, int b, fx64 c) {
  fx64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
// the two mixed partial products of a * b, added to m
__device__ __forceinline__ fx64 fx_mid(FxLimb a, FxLimb b, fx64 m) { return fx_mad(a.l, b.h, fx_mad(a.h, b.l, m)); }
// the 96-bit number (t, lower word of m) shifted left by S (0 .. 31), its upper 64 bits
__device__ __forceinline__ fx64 fx_shift(fx64 t, fx64 m, int S) {
  const unsigned tl = (unsigned)t, th = (unsigned)((unsigned long long)t >> 32);
  return (fx64)(((unsigned long long)__funnelshift_l(tl, th, S) << 32) | __funnelshift_l((unsigned)m, tl, S));
}
// (a b [+ c d [+ e f]]) / 2^(64-S) + 2^(31+S): the mixed products start from 2^63, so that their upper
// word is unsigned and joins the chain of the upper products without a sign extension; the bias is taken
// off with the limbs (fx_unbias) or cancels.  1 <= S <= 31.
constexpr fx64 kFxMid = (fx64)(1ull << 63);
__device__ __forceinline__ fx64 fx_up(fx64 m) { return (fx64)((unsigned long long)m >> 32); }
__device__ __forceinline__ fx64 fx_mul(FxLimb a, FxLimb b, int S) {
  const fx64 m = fx_mid(a, b, kFxMid);
  return fx_shift(fx_mad(a.h, b.h, fx_up(m)), m, S);
}
__device__ __forceinline__ fx64 fx_dot(FxLimb a, FxLimb b, FxLimb c, FxLimb d, int S) {
  const fx64 m = fx_mid(c, d, fx_mid(a, b, kFxMid));
  return fx_shift(fx_mad(c.h, d.h, fx_mad(a.h, b.h, fx_up(m))), m, S);
}
__device__ __forceinline__ fx64 fx_dot(FxLimb a, FxLimb b, FxLimb c, FxLimb d, FxLimb e, FxLimb f, int S) {
  const fx64 m = fx_mid(e, f, fx_mid(c, d, fx_mid(a, b, kFxMid)));
  return fx_shift(fx_mad(e.h, f.h, fx_mad(c.h, d.h, fx_mad(a.h, b.h, fx_up(m)))), m, S);
}
__device__ __forceinline__ FxLimb fx_unbias(fx64 x, int S) {
  const int l = (int)x;
  return {(int)((unsigned)(x >> 32) - (unsigned)(l >> 31) - (1u << (S - 1))), l};
}
__device__ __forceinline__ fx64 fx_unbias64(fx64 x, int S) { return fx_sub(x, (fx64)(1ull << (31 + S))); }
// arithmetic right shift by 0 .. 63
__device__ __forceinline__ fx64 fx_sar(fx64 x, int k) {
  fx64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(k));
  return r;
}

// the word of |x| that orders magnitudes: exponent and upper mantissa
__device__ __forceinline__ unsigned fx_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// e with |x| < 2^e for every x whose fx_mag is at most mag (at least -150: zeros)
__device__ __forceinline__ int fx_exp(unsigned mag) { return max((int)(mag >> 20) - 1022, -150); }
// log2 of the largest |x| with this fx_mag, rounded up by about 1e-5
__device__ __forceinline__ float fx_log2(unsigned mag) {
  const float f = __int_as_float(0x3f800000u | ((mag & 0xfffffu) << 3));
  return fmaxf((float)((int)(mag >> 20) - 1023) + __log2f(f) + 1e-5f, -150.f);
}
// |x| from its fx_mag as a float (truncated), 2^-60 .. 2^60
__device__ __forceinline__ float fx_float(unsigned mag) {
  const unsigned lo = (1023u - 60u) << 20, hi = (1023u + 60u) << 20;
  mag = mag < lo ? lo : (mag > hi ? hi : mag);
  return __uint_as_float((mag - (896u << 20)) << 3);
}

// x * 2^s, towards zero, from r0 = fx_r0(s); |x 2^s| < 2^63, s < 1022.  Zeros and subnormal numbers give 0.
__device__ __forceinline__ int fx_r0(int s) { return 64 + 1022 - s; }
__device__ __forceinline__ fx64 fx_from(double x, int r0) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int eb = (hi >> 20) & 0x7ff;
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, 11) << 32) | (lo << 11);
  unsigned long long v;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(r0 - eb));  // amounts above 63 give 0
  return hi < 0 ? -(fx64)v : (fx64)v;
}

// the 96-bit number (t, lower word of m) in units of t as a double, with all its bits: normalised by the
// count s of redundant sign bits before the conversion
__device__ __forceinline__ double fx_to_double(fx64 t, fx64 m) {
  const int th = (int)(t >> 32);
  const int s = __clz(th ^ (th >> 31)) - 1;
  const double d = __ll2double_rn(fx_shift(t, m, s));
  const int dh = __double2hiint(d);
  return __hiloint2double((dh & 0x7ff00000) ? dh - (s << 20) : 0, __double2loint(d));
}

// log2 of the ratio of the largest and smallest |M_d| of an element, from MetL
__device__ __forceinline__ float fx_flatness(const float* MetL) {
  return fmaxf(MetL[0], fmaxf(MetL[1], MetL[2])) - fminf(MetL[0], fminf(MetL[1], MetL[2]));
}

// warp maximum / minimum of a magnitude word, combined over the block in shared memory (initialised by
// the caller; a block barrier follows)
__device__ __forceinline__ void fx_block_max(unsigned v, unsigned* s) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) atomicMax(s, v);
}
__device__ __forceinline__ void fx_block_min(unsigned v, unsigned* s) {
  v = __reduce_min_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) atomicMin(s, v);
}

// ---- digits: X = h 2^30 + l with |l| < 2^30 (same sign as h or 0 <= l), |X| < 2^60.  Sums are taken digit by
// digit (two additions, |l| < 2^31), products are a.h b.h + (a.h b.l + a.l b.h) / 2^30, in units of 2^60.
struct FxDig {
  int h, l;
};
__device__ __forceinline__ FxDig fd_split(fx64 x) { return {(int)(x >> 30), (int)x & 0x3fffffff}; }
__device__ __forceinline__ FxDig operator+(FxDig a, FxDig b) { return {a.h + b.h, a.l + b.l}; }
__device__ __forceinline__ FxDig operator-(FxDig a, FxDig b) { return {a.h - b.h, a.l - b.l}; }
struct FxDot {
  fx64 hh, mid, ll;
  __device__ __forceinline__ FxDot() : hh(0), mid(0), ll(0) {}
  __device__ __forceinline__ void add(FxDig a, FxDig b) {
    hh = fx_mad(a.h, b.h, hh);
    mid = fx_mad(a.l, b.h, fx_mad(a.h, b.l, mid));
    ll = fx_mad(a.l, b.l, ll);
  }
  // the low products' carry, before more than four of them (2^61 each) have been added
  __device__ __forceinline__ void carry() { mid += ll >> 30; ll = 0; }
  // the sum * 2^K in units of 2^60
  template <int K = 0> __device__ __forceinline__ fx64 sum() const {
    const fx64 m = mid + (ll >> 30);
    return K == 0 ? hh + (m >> 30) : (hh << K) + (m >> (30 - K));
  }
};
// the same without the low products, which are below one unit of the sum each: where |a| and |b| use the range
struct FxDotU {
  fx64 hh, mid;
  __device__ __forceinline__ FxDotU() : hh(0), mid(0) {}
  __device__ __forceinline__ void add(FxDig a, FxDig b) {
    hh = fx_mad(a.h, b.h, hh);
    mid = fx_mad(a.l, b.h, fx_mad(a.h, b.l, mid));
  }
  __device__ __forceinline__ fx64 sum() const { return hh + (mid >> 30); }
};
// digits of x * 2^K, K = max(k, 0) up to 30 (k < 0: of x / 2^-k); |x 2^k| < 2^60
__device__ __forceinline__ FxDig fd_scaled(fx64 x, int k) {
  if (k < 0) { x = fx_sar(x, -k); k = 0; }
  const unsigned lo = (unsigned)x, hi = (unsigned)((unsigned long long)x >> 32);
  return {(int)__funnelshift_r(lo, hi, 30 - k), (int)((lo << k) & 0x3fffffffu)};
}
__device__ __forceinline__ fx64 fd_pack(FxDig a) { return (fx64)(((unsigned long long)(unsigned)a.h << 32) | (unsigned)a.l); }
__device__ __forceinline__ FxDig fd_unpack(fx64 x) { return {(int)(x >> 32), (int)x}; }
// x * 2^s towards zero in digits, from r0 = fx_r0(s); |x 2^s| < 2^60, s < 1022
__device__ __forceinline__ FxDig fd_from(double x, int r0) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int eb = (hi >> 20) & 0x7ff;
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const unsigned long long m = ((unsigned long long)__funnelshift_l(lo, mh, 11) << 32) | (lo << 11);
  unsigned long long v;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(r0 - eb));
  const int sg = (hi >> 31) | 1;
  return {(int)(v >> 30) * sg, (int)((unsigned)v & 0x3fffffffu) * sg};
}
// the word of |x| that orders magnitudes of integers, and b with |x| < 2^b for every x whose word is at most mag
__device__ __forceinline__ unsigned fx_mag64(fx64 x) { return (unsigned)abs((int)(x >> 32)); }
__device__ __forceinline__ int fx_bits(unsigned mag) { return 64 - __clz((int)(mag + 1u)); }
// x as a double times 2^k
__device__ __forceinline__ double fx_scaled(fx64 x, int k) {
  const double d = __ll2double_rn(x);
  const int dh = __double2hiint(d);
  return __hiloint2double((dh & 0x7ff00000) ? dh + (k << 20) : 0, __double2loint(d));
}

}  // namespace gx
