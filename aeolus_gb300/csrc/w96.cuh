// 96-bit integers and limb pairs: the arithmetic of the FP64 plans' row
// transforms (rows_w.cuh), built from 32-bit additions with carry and 32 x 32 ->
// 64-bit multiply-adds.  GB300 executes those at up to 64 times the rate of its
// FP64 pipe.
#pragma once

#include "fx.cuh"

namespace aeolus {

// ------------------------------------------------------- 96-bit integers
struct w96 {
  unsigned l, m;
  int h;
};
struct cw {
  w96 re, im;
};

__device__ __forceinline__ w96 w_add(w96 a, w96 b) {
  w96 r;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=r"(r.l), "=r"(r.m), "=r"(r.h)
      : "r"(a.l), "r"(a.m), "r"(a.h), "r"(b.l), "r"(b.m), "r"(b.h));
  return r;
}
__device__ __forceinline__ w96 w_sub(w96 a, w96 b) {
  w96 r;
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=r"(r.l), "=r"(r.m), "=r"(r.h)
      : "r"(a.l), "r"(a.m), "r"(a.h), "r"(b.l), "r"(b.m), "r"(b.h));
  return r;
}
__device__ __forceinline__ w96 w_neg(w96 a) { return w_sub(w96{0u, 0u, 0}, a); }
__device__ __forceinline__ w96 w_half(w96 a) {
  return w96{__funnelshift_r(a.l, a.m, 1), __funnelshift_r(a.m, (unsigned)a.h, 1), a.h >> 1};
}
// v 2^s for a 64-bit v, 0 <= s < 32.
__device__ __forceinline__ w96 w_shl64(long long v, int s) {
  const unsigned lo = (unsigned)v, hi = (unsigned)((unsigned long long)v >> 32);
  return w96{lo << s, __funnelshift_l(lo, hi, s), (int)__funnelshift_l(hi, (unsigned)((int)hi >> 31), s)};
}

// 30-bit limbs x = x2 2^60 + (X1 / 2) 2^30 + X0 / 2 (|x| < 2^90): the two low
// ones doubled, to pair with the 31-bit limbs of a Q61 factor.
struct wlimbs {
  int x2, x1, X1, X0;
};
__device__ __forceinline__ wlimbs w_limbs(w96 x) {
  const int X1 = (int)(__funnelshift_r(x.l, x.m, 29) & 0x7FFFFFFEu);
  return wlimbs{(int)__funnelshift_r(x.m, (unsigned)x.h, 28), X1 >> 1, X1, (int)((x.l << 1) & 0x7FFFFFFEu)};
}
// (H 2^31 + T2) / 2 with H = sum of x2 wh, T2 = sum of x2 wl + X1 wh + carry.
__device__ __forceinline__ w96 w_recombine(long long H, long long T2) {
  const unsigned hl = (unsigned)H, hh = (unsigned)((unsigned long long)H >> 32);
  const unsigned tl = (unsigned)T2, th = (unsigned)((unsigned long long)T2 >> 32);
  return w_add(w96{hl << 30, __funnelshift_r(hl, hh, 2), (int)hh >> 2},
               w96{__funnelshift_r(tl, th, 1), (unsigned)((int)th >> 1), (int)th >> 31});
}
// x k, |k| <= 1.
__device__ __forceinline__ w96 w_mulk(w96 x, FxK k) {
  const wlimbs a = w_limbs(x);
  const long long t1 = fx_madw(a.X0, k.h, fx_madw(a.x1, k.l, 0LL));
  const long long t2 = fx_madw(a.X1, k.h, fx_madw(a.x2, k.l, t1 >> 30));
  return w_recombine(fx_madw(a.x2, k.h, 0LL), t2);
}
// x w (CONJ: x conj(w)), |w| = 1.
template <bool CONJ>
__device__ __forceinline__ cw w_cmul(cw x, FxW w) {
  const wlimbs a = w_limbs(x.re), b = w_limbs(x.im);
  // re = a c -+ b s, im = +-a s + b c: the sign goes to s
  const int sh = w.sh, sl = w.sl, nh = -w.sh, nl = -w.sl;
  const int rh = CONJ ? sh : nh, rl = CONJ ? sl : nl;  // factor of b in re
  const int ih = CONJ ? nh : sh, il = CONJ ? nl : sl;  // factor of a in im
  const long long r1 = fx_madw(b.X0, rh, fx_madw(b.x1, rl, fx_madw(a.X0, w.ch, fx_madw(a.x1, w.cl, 0LL))));
  const long long r2 =
      fx_madw(b.X1, rh, fx_madw(b.x2, rl, fx_madw(a.X1, w.ch, fx_madw(a.x2, w.cl, r1 >> 30))));
  const long long i1 = fx_madw(b.X0, w.ch, fx_madw(b.x1, w.cl, fx_madw(a.X0, ih, fx_madw(a.x1, il, 0LL))));
  const long long i2 =
      fx_madw(b.X1, w.ch, fx_madw(b.x2, w.cl, fx_madw(a.X1, ih, fx_madw(a.x2, il, i1 >> 30))));
  return cw{w_recombine(fx_madw(b.x2, rh, fx_madw(a.x2, w.ch, 0LL)), r2),
            w_recombine(fx_madw(b.x2, w.ch, fx_madw(a.x2, ih, 0LL)), i2)};
}
__device__ __forceinline__ cw cw_add(cw a, cw b) { return cw{w_add(a.re, b.re), w_add(a.im, b.im)}; }
__device__ __forceinline__ cw cw_sub(cw a, cw b) { return cw{w_sub(a.re, b.re), w_sub(a.im, b.im)}; }
// a + sg i b and a - sg i b (sg = +1 for POS) without a negation
template <bool POS>
__device__ __forceinline__ cw cw_add_i(cw a, cw b) {
  return POS ? cw{w_sub(a.re, b.im), w_add(a.im, b.re)} : cw{w_add(a.re, b.im), w_sub(a.im, b.re)};
}

// ------------------------------------------------- FP64 <-> fixed point
// Key of |x|: its high word (exponent and 20 mantissa bits).
__device__ __forceinline__ unsigned f64_key(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
constexpr unsigned kNonFinite = 0x7FF00000u;  // keys from here on are infinities and NaNs
// Exponent E with |x| < 2^E for every finite x whose key is at most `key`.
__device__ __forceinline__ int f64_key_exp(unsigned key) { return max((int)(key >> 20), 1) - 1022; }

// x 2^-S towards zero, for |x 2^-S| < 2^84.
__device__ __forceinline__ w96 w_of_f64(double x, int S) {
  const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
  const int ex = (int)((xh >> 20) & 0x7FFu);
  const unsigned mh = (xh & 0xFFFFFu) | (ex ? 0x100000u : 0u);
  // mantissa left-aligned in 96 bits (2^43 times its value), then shifted down
  unsigned h = __funnelshift_l(xl, mh, 11), m = xl << 11, l = 0u;
  int r = 1118 + S - max(ex, 1);  // 43 - (ex - 1075 - S)
  if (r >= 64) l = h, m = 0u, h = 0u, r -= 64;
  else if (r >= 32) l = m, m = h, h = 0u, r -= 32;
  if (r >= 32) l = 0u, r = 0;  // below one unit
  l = __funnelshift_r(l, m, r);
  m = __funnelshift_r(m, h, r);
  h = h >> r;
  const w96 v{l, m, (int)h};
  return (int)xh < 0 ? w_neg(v) : v;
}

// X 2^S rounded to FP64 (half up in magnitude; subnormal results are truncated,
// those above the range infinite), integer instructions only.
__device__ __forceinline__ double f64_of_w(w96 x, int S) {
  const int s = x.h >> 31;
  unsigned h = (unsigned)(x.h ^ s), m = x.m ^ (unsigned)s, l = x.l ^ (unsigned)s;  // |x| (one unit less if negative)
  int top = 95;
  if (h == 0u) h = m, m = l, l = 0u, top = 63;
  if (h == 0u) h = m, m = 0u, top -= 32;
  const int c = __clz((int)h);
  if (c == 32) return 0.0;
  h = __funnelshift_l(m, h, c);
  m = __funnelshift_l(l, m, c);
  const int e = top - c + S + 1022;  // biased exponent less one: the leading bit adds it back
  unsigned lo = __funnelshift_r(m, h, 11), hi = h >> 11;
  const unsigned long long t = (((unsigned long long)hi << 32) | lo) + ((m >> 10) & 1u);
  const unsigned sg = (unsigned)s & 0x80000000u;
  if (e < 0) {  // subnormal: truncated
    const unsigned long long d = -e < 64 ? t >> -e : 0ull;
    return __longlong_as_double((long long)(d | ((unsigned long long)sg << 32)));
  }
  if (e >= 2046) return __hiloint2double((int)(0x7FF00000u | sg), 0);
  const unsigned long long b = t + ((unsigned long long)(unsigned)e << 52);
  return __longlong_as_double((long long)(b | ((unsigned long long)((unsigned)s & 0x80000000u) << 32)));
}

// ------------------------------------------------------------ limb pairs
// x 2^-S as a 64-bit integer, towards zero (|x 2^-S| < 2^62).
__device__ __forceinline__ long long i64_of_f64(double x, int S) {
  const w96 v = w_of_f64(x, S);
  return (long long)(((unsigned long long)v.m << 32) | v.l);
}
// The same, rounded (half up).
__device__ __forceinline__ long long i64_of_f64_rn(double x, int S) { return (i64_of_f64(x, S - 1) + 1) >> 1; }
// v = h 2^LB + l, l in [-2^(LB-1), 2^(LB-1)).
template <int LB>
__device__ __forceinline__ int2 limbs(long long v) {
  const int h = (int)((v + (1LL << (LB - 1))) >> LB);
  return make_int2(h, (int)(v - ((long long)h << LB)));
}
// A sum of products of limb pairs from its two accumulators (high x high, and
// the mixed products; low x low is dropped), in units of 2^LB times the product
// of the factors' units; DROP more bits off.
template <int LB, int DROP = 0>
__device__ __forceinline__ w96 limb_total(long long hh, long long x) {
  return w_add(w_shl64(hh, LB - DROP), w_shl64(x >> DROP, 0));
}

}  // namespace aeolus
