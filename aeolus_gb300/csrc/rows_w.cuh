// Longitude stage of FP64 plans, one CTA per (latitude row, member rows):
//   order spectrum F_m (m <= L) --c2r--> grid row --FP64 products--> row
//   --r2c--> weighted order spectrum G_m,
// with the transforms in 96-bit fixed point.  GB300's FP64 pipe does two
// additions per clock and SM against 128 integer ones, so a 96-bit integer
// addition (three instructions) costs a tenth of an FP64 one and is exact:
//   * the row of one field is rounded to integers X at one block exponent S
//     (value X 2^S) with |X| < 2^hb, hb = 86 - ceil(log2 n) (78 at n = 192), so
//     an FP64 value keeps all 53 bits down to 2^-25 of the row's largest and
//     the absolute error elsewhere is 2^-78 of it;
//   * a twiddle product is x w with x in 30-bit limbs and w = Q61 (two 31-bit
//     limbs): ten wide multiply-adds per real part, within a few units of X;
//   * no operand of a product reaches 2^90 whatever the data: the bound on hb
//     covers the growth of a length-n transform and the factor 4 of the
//     real-FFT pre- and post-processing.
// The transform's error is then that of the FP64 twiddle table alone, below
// that of an FP64 FFT, which adds a rounding of 2^-53 per operation.  Grid
// values and order spectra are rounded once to FP64 (integer instructions);
// only the pointwise products run on the FP64 pipe.  A row with an infinity or
// a NaN comes out as NaN, as from FP64 arithmetic.
//
// Row lengths without a 2/3/5 transform (the 3/2-rule grids of state grids
// that just resolve l_max: 3 l_max + 1 points) use a direct sum, folded about
// the middle of the row, over 30-bit limb pairs with 64-bit accumulators:
// six wide multiply-adds per order and pair of points (row_w_dft_body).
//
// Row stage per RK4 stage against FP64 transforms and sums: 8 members at 192 x
// 384, l_max 127 367 -> 124 us; 3 members on 95 x 190 points, l_max 63 (direct
// sums) 238 -> 39 us; one member at 128 x 256, l_max 85 28.9 -> 23.9 us (128
// CTAs, bound by the latency of one row); 82 fields on 64 x 128 points (grid
// output) 66 -> 17 us.  Bound by instruction issue (42 k warp instructions per
// 9 + 4 field row at n = 192; 38 % issue-active at 14 warps per SM, which the
// 128 registers of a radix-8 butterfly allow); the FP64 pipe is 28 % busy.
// Error of an SWE tendency against 64-bit sums at l_max 127: zeta 3.37e-15 ->
// 3.34e-15, delta 9.04e-13 -> 9.01e-13, phi 1.95e-15 -> 1.93e-15.
#pragma once

#include "rows.cuh"
#include "w96.cuh"

namespace aeolus {

// ------------------------------------------------------------ transforms
template <bool INV, int R>
__device__ __forceinline__ void butterfly_w(cw* v, const FxConst& k) {
  if constexpr (R == 2) {
    const cw a = v[0], b = v[1];
    v[0] = cw_add(a, b);
    v[1] = cw_sub(a, b);
  } else if constexpr (R == 4) {
    const cw s02 = cw_add(v[0], v[2]), d02 = cw_sub(v[0], v[2]);
    const cw s13 = cw_add(v[1], v[3]), d13 = cw_sub(v[1], v[3]);
    v[0] = cw_add(s02, s13);
    v[2] = cw_sub(s02, s13);
    v[1] = cw_add_i<INV>(d02, d13);
    v[3] = cw_add_i<!INV>(d02, d13);
  } else if constexpr (R == 3) {
    const cw s = cw_add(v[1], v[2]), d = cw_sub(v[1], v[2]);
    const cw t = cw{w_sub(v[0].re, w_half(s.re)), w_sub(v[0].im, w_half(s.im))};
    const cw e = cw{w_mulk(d.re, k.h3), w_mulk(d.im, k.h3)};
    v[0] = cw_add(v[0], s);
    v[1] = cw_add_i<INV>(t, e);
    v[2] = cw_add_i<!INV>(t, e);
  } else if constexpr (R == 8) {
    cw e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    butterfly_w<INV, 4>(e, k);
    butterfly_w<INV, 4>(o, k);
    // o1 (1 +- i)/sqrt2, o2 (+- i), o3 (-1 +- i)/sqrt2 (+: inverse)
    const w96 s1 = w_mulk(w_add(o[1].re, o[1].im), k.r2), d1 = w_mulk(w_sub(o[1].re, o[1].im), k.r2);
    const w96 s3 = w_mulk(w_add(o[3].re, o[3].im), k.r2), d3 = w_mulk(w_sub(o[3].re, o[3].im), k.r2);
    v[0] = cw_add(e[0], o[0]);
    v[4] = cw_sub(e[0], o[0]);
    v[2] = cw_add_i<INV>(e[2], o[2]);
    v[6] = cw_add_i<!INV>(e[2], o[2]);
    if (INV) {
      v[1] = cw{w_add(e[1].re, d1), w_add(e[1].im, s1)};
      v[5] = cw{w_sub(e[1].re, d1), w_sub(e[1].im, s1)};
      v[3] = cw{w_sub(e[3].re, s3), w_add(e[3].im, d3)};
      v[7] = cw{w_add(e[3].re, s3), w_sub(e[3].im, d3)};
    } else {
      v[1] = cw{w_add(e[1].re, s1), w_sub(e[1].im, d1)};
      v[5] = cw{w_sub(e[1].re, s1), w_add(e[1].im, d1)};
      v[3] = cw{w_sub(e[3].re, d3), w_sub(e[3].im, s3)};
      v[7] = cw{w_add(e[3].re, d3), w_add(e[3].im, s3)};
    }
  } else {  // R == 5
    const cw a1 = cw_add(v[1], v[4]), a2 = cw_add(v[2], v[3]);
    const cw b1 = cw_sub(v[1], v[4]), b2 = cw_sub(v[2], v[3]);
    const cw t1 = cw{w_add(v[0].re, w_add(w_mulk(a1.re, k.c1), w_mulk(a2.re, k.c2))),
                     w_add(v[0].im, w_add(w_mulk(a1.im, k.c1), w_mulk(a2.im, k.c2)))};
    const cw t2 = cw{w_add(v[0].re, w_add(w_mulk(a1.re, k.c2), w_mulk(a2.re, k.c1))),
                     w_add(v[0].im, w_add(w_mulk(a1.im, k.c2), w_mulk(a2.im, k.c1)))};
    const cw u1 = cw{w_add(w_mulk(b1.re, k.s1), w_mulk(b2.re, k.s2)), w_add(w_mulk(b1.im, k.s1), w_mulk(b2.im, k.s2))};
    const cw u2 = cw{w_sub(w_mulk(b1.re, k.s2), w_mulk(b2.re, k.s1)), w_sub(w_mulk(b1.im, k.s2), w_mulk(b2.im, k.s1))};
    v[0] = cw_add(v[0], cw_add(a1, a2));
    v[1] = cw_add_i<INV>(t1, u1);
    v[4] = cw_add_i<!INV>(t1, u1);
    v[2] = cw_add_i<INV>(t2, u2);
    v[3] = cw_add_i<!INV>(t2, u2);
  }
}

// Row buffers: a complex slot is 16 bytes (re.m, re.h, im.m, im.h) plus 8
// (re.l, im.l) in a second array; the first part alone also holds two FP64
// grid values.
struct WRows {
  uint4* H;
  uint2* L;
  __device__ __forceinline__ cw get(int i) const {
    const uint4 a = H[i];
    const uint2 b = L[i];
    return cw{w96{b.x, a.x, (int)a.y}, w96{b.y, a.z, (int)a.w}};
  }
  __device__ __forceinline__ void put(int i, cw v) const {
    H[i] = make_uint4(v.re.m, (unsigned)v.re.h, v.im.m, (unsigned)v.im.h);
    L[i] = make_uint2(v.re.l, v.im.l);
  }
  __device__ __forceinline__ double2 get_f64(int i) const { return *reinterpret_cast<const double2*>(&H[i]); }
  __device__ __forceinline__ void put_f64(int i, double2 v) const { *reinterpret_cast<double2*>(&H[i]) = v; }
};

// One in-place stage (see fft_stage_ip in rows_fx.cuh); CONV: the rows still
// hold FP64 values, rounded at their field's block exponent as they are read.
// Transform f sits in slot row (f / PER) STR + f mod PER (PER fields of each
// member row's STR slots).
template <int PER, int STR>
__device__ __forceinline__ int w_slot(int f) {
  return PER == STR ? f : f / PER * STR + f % PER;
}
template <bool INV, int R, bool TW, bool CONV, int PER, int STR>
__device__ __forceinline__ void w_stage(const WRows& x, int nf, int n, int fs, int Ls, unsigned nb_rcp,
                                        unsigned ls_rcp, const FxW* __restrict__ tw, const FxConst& kc, const int* sS) {
  const int nb = n / R, stride = n / (Ls * R);
#pragma unroll 1
  for (int idx = threadIdx.x; idx < nf * nb; idx += blockDim.x) {
    const int fi = div_rcp(idx, nb, nb_rcp), jj = idx - fi * nb, f = w_slot<PER, STR>(fi);
    const int g = div_rcp(jj, Ls, ls_rcp), k = jj - g * Ls;
    const int base = f * fs + g * Ls * R + k;
    cw v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      if constexpr (CONV) {
        const double2 d = x.get_f64(base + t * Ls);
        v[t] = cw{w_of_f64(d.x, sS[f]), w_of_f64(d.y, sS[f])};
      } else {
        v[t] = x.get(base + t * Ls);
      }
    }
    if (INV && TW) {
#pragma unroll
      for (int t = 1; t < R; ++t) v[t] = w_cmul<INV>(v[t], fx_ldw(&tw[2 * (k * t * stride)]));
    }
    butterfly_w<INV, R>(v, kc);
    if (!INV && TW) {
#pragma unroll
      for (int t = 1; t < R; ++t) v[t] = w_cmul<INV>(v[t], fx_ldw(&tw[2 * (k * t * stride)]));
    }
#pragma unroll
    for (int t = 0; t < R; ++t) x.put(base + t * Ls, v[t]);
  }
}

template <bool INV, bool TW, bool CONV, int PER, int STR>
__device__ __forceinline__ void w_stage_r(int r, const WRows& x, int nf, int n, int fs, int Ls, unsigned nbm,
                                          unsigned lsm, const FxW* __restrict__ tw, const FxConst& kc, const int* sS) {
  switch (r) {
    case 8: w_stage<INV, 8, TW, CONV, PER, STR>(x, nf, n, fs, Ls, nbm, lsm, tw, kc, sS); break;
    case 4: w_stage<INV, 4, TW, CONV, PER, STR>(x, nf, n, fs, Ls, nbm, lsm, tw, kc, sS); break;
    case 2: w_stage<INV, 2, TW, CONV, PER, STR>(x, nf, n, fs, Ls, nbm, lsm, tw, kc, sS); break;
    case 3: w_stage<INV, 3, TW, CONV, PER, STR>(x, nf, n, fs, Ls, nbm, lsm, tw, kc, sS); break;
    default: w_stage<INV, 5, TW, CONV, PER, STR>(x, nf, n, fs, Ls, nbm, lsm, tw, kc, sS); break;
  }
}

// Inverse by decimation in time (digit-reversed input), forward by decimation
// in frequency (digit-reversed output; its first stage reads FP64 rows).
template <int NIN>
__device__ __forceinline__ void w_fft_inv(const WRows& x, int nf, int fs, const FftInfo& fi,
                                          const FxW* __restrict__ tw, const FxConst& kc) {
  int Ls = 1;
  for (int s = 0; s < fi.nfac; ++s) {
    if (s == 0)
      w_stage_r<true, false, false, NIN, NIN>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, nullptr);
    else
      w_stage_r<true, true, false, NIN, NIN>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, nullptr);
    __syncthreads();
    Ls *= fi.fac[s];
  }
}
template <int NOUT, int OS>
__device__ __forceinline__ void w_fft_fwd(const WRows& x, int nf, int fs, const FftInfo& fi,
                                          const FxW* __restrict__ tw, const FxConst& kc, const int* sS) {
  int Ls = fi.n;
  for (int s = fi.nfac - 1; s >= 0; --s) {
    Ls /= fi.fac[s];
    const bool conv = s == fi.nfac - 1;
    if (conv && s == 0)
      w_stage_r<false, false, true, NOUT, OS>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, sS);
    else if (conv)
      w_stage_r<false, true, true, NOUT, OS>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, sS);
    else if (s == 0)
      w_stage_r<false, false, false, NOUT, OS>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, sS);
    else
      w_stage_r<false, true, false, NOUT, OS>(fi.fac[s], x, nf, fi.n, fs, Ls, fi.nbm[s], fi.lsm[s], tw, kc, sS);
    __syncthreads();
  }
}

// Member rows per CTA of a batch that fills the chip: functors with few fields
// take several, so every phase has work for all threads (a batch that does
// not takes one).
template <class Pw>
constexpr int w_rows_per_cta() {
  constexpr int NF = Pw::NIN > Pw::NOUT ? Pw::NIN : Pw::NOUT;
  return NF >= 5 ? 1 : NF >= 3 ? 2 : NF == 2 ? 4 : 8;
}
constexpr int kWideMaxThreads = 256;

// Where the row stage of an FP64 plan finds input field f of a functor:
// spectra block src(f), times i m / R for a longitude derivative (lam(f)),
// which is diagonal in m and needs no contraction of its own.  Default: field
// f in block f.
template <class Pw, class = void>
struct RowSrc {
  static constexpr int NBLK = Pw::NIN;
  __device__ static constexpr int src(int f) { return f; }
  __device__ static constexpr bool lam(int) { return false; }
};
template <class Pw>
struct RowSrc<Pw, std::void_t<decltype(Pw::NBLK64)>> {
  static constexpr int NBLK = Pw::NBLK64;
  __device__ static constexpr int src(int f) { return Pw::src64(f); }
  __device__ static constexpr bool lam(int f) { return Pw::lam64(f); }
};

// Per-CTA scalars.
template <int N>
struct WScratch {
  unsigned bits[N];
  unsigned key[N];  // largest input / output key of each (row, field)
  int S[N];         // its block exponent
};

template <class Pw, int NR, int IN_MODE, int OUT_MODE>
__device__ __forceinline__ void row_w_body(const RowArgs& a, const Pw& pw, const FxW* __restrict__ twfx,
                                           const FxConst& kc, int bx, int by) {
  constexpr int NIN = Pw::NIN, NOUT = Pw::NOUT;
  constexpr int NF = NIN > NOUT ? NIN : NOUT;
  constexpr int NRI = NR * NIN, NRO = NR * NOUT;
  static_assert(NR == 1 || NIN == NF, "several member rows: the outputs take input slots");
  extern __shared__ uint4 smem_w[];
  __shared__ WScratch<NR * NF> sc;
  const int j = bx, b0 = by * NR, T = blockDim.x, tid = threadIdx.x;
  const int nrow = min(NR, a.batch - b0);
  const int N = a.fft.N, n = a.fft.n, L = a.L, fs = n + 1;
  const int hb = 86 - (32 - __clz(max(n - 1, 1)));
  const WRows x{smem_w, reinterpret_cast<uint2*>(smem_w + NR * NF * fs)};
  const long sq = (long)a.nblk * a.nlat, sb = sq * (L + 1);  // order and member stride of the blocks
  double2* block = nullptr;
  if (IN_MODE == kInF || OUT_MODE == kOutG) block = a.FG + fg_index(b0, 0, 0, j, L, a.nblk, a.nlat);
  for (int i = tid; i < NR * NF; i += T) sc.bits[i] = 0u, sc.key[i] = 0u;
  __syncthreads();

  // ---- 1. grid rows of the NIN input fields in fixed point
  if constexpr (IN_MODE == kInF) {
    // each thread keeps one (row, field): its orders to their digit-reversed
    // slots as FP64, the largest key on the way
    const int TQ = T / NRI;
    if (tid < TQ * NRI) {
      const int rf = tid % NRI, row = rf / NIN, f = rf - row * NIN;
      if (row < nrow) {
        const double2* src = block + row * sb + RowSrc<Pw>::src(f);
        const bool lam = RowSrc<Pw>::lam(f);
        unsigned mx = 0u;
#pragma unroll 4
        for (int q = tid / NRI; q <= L; q += TQ) {
          double2 v = src[(long)q * sq];
          if (lam) v = cscale((double)q * a.ir, ci(v));
          if (q == 0) v.y = 0.0;
          mx = max(mx, max(f64_key(v.x), f64_key(v.y)));
          x.put_f64(rf * fs + __ldg(&a.irev[q]), v);
        }
        if (mx) atomicMax(&sc.key[rf], mx);
      }
    }
    __syncthreads();
    for (int i = tid; i < NRI; i += T) sc.S[i] = f64_key_exp(sc.key[i]) - hb;
    __syncthreads();
    // Z_q = A + P, Z_{n-q} = conj(A - P), A = H_q + conj H_{n-q}, P = i conj(e_q) (H_q - conj H_{n-q})
#pragma unroll 1
    for (int idx = tid; idx < NRI * (n / 2 + 1); idx += T) {
      const int q = idx / NRI, rf = idx - q * NRI, S = sc.S[rf];
      if (NR > 1 && rf >= nrow * NIN) continue;
      const int qn = n - q, s0 = rf * fs + __ldg(&a.irev[q]), s1 = q == 0 ? s0 : rf * fs + __ldg(&a.irev[qn]);
      cw hq{}, hn{};
      if (q <= L) {
        const double2 d = x.get_f64(s0);
        hq = cw{w_of_f64(d.x, S), w_of_f64(d.y, S)};
      }
      if (q > 0 && qn <= L) {
        const double2 d = x.get_f64(s1);
        hn = cw{w_of_f64(d.x, S), w_of_f64(d.y, S)};
      }
      const cw A{w_add(hq.re, hn.re), w_sub(hq.im, hn.im)};
      const cw B{w_sub(hq.re, hn.re), w_add(hq.im, hn.im)};
      const cw C = w_cmul<true>(B, fx_ldw(&twfx[q]));
      x.put(s0, cw_add_i<true>(A, C));
      if (q > 0 && qn > q) {
        const cw Z = cw_add_i<false>(A, C);
        x.put(s1, cw{Z.re, w_neg(Z.im)});
      }
    }
    __syncthreads();
    w_fft_inv<NIN>(x, nrow * NIN, fs, a.fft, twfx, kc);
  }

  // ---- 2. pointwise products, two grid points (one complex slot) at a time,
  // in place; grid output leaves directly
  {
    const double c = a.coslat[j];
    const double fg = a.fgrid ? a.fgrid[j] : 0.0;
    const double nan = __hiloint2double(0x7FF80000, 0);
#pragma unroll 1
    for (int i = tid; i < nrow * n; i += T) {
      const int row = NR == 1 ? 0 : i / n, k = i - row * n;
      double i0[NIN], i1[NIN], o0[NOUT], o1[NOUT];
#pragma unroll
      for (int f = 0; f < NIN; ++f) {
        const int rf = row * NIN + f;
        if constexpr (IN_MODE == kInF) {
          const cw v = x.get(rf * fs + k);
          const bool bad = sc.key[rf] >= kNonFinite;
          i0[f] = bad ? nan : f64_of_w(v.re, sc.S[rf]);
          i1[f] = bad ? nan : f64_of_w(v.im, sc.S[rf]);
        } else {
          const double* g = a.gin + (long)(b0 + row) * a.gin_b + (long)f * a.gin_f + (long)j * N + 2 * k;
          i0[f] = g[0];
          i1[f] = g[1];
        }
      }
      const unsigned bits = pw(c, fg, i0, o0) | pw(c, fg, i1, o1);
      if (a.status && bits) atomicOr(&sc.bits[row], bits);
      if constexpr (OUT_MODE == kOutGrid) {
#pragma unroll
        for (int f = 0; f < NOUT; ++f) {
          double* g = a.gout + (long)(b0 + row) * a.gout_b + (long)f * a.gout_f + (long)j * N + 2 * k;
          g[0] = o0[f];
          g[1] = o1[f];
        }
      } else {
        // only this thread touches slot k of the member row's fields, so the
        // outputs take the place of its first inputs
#pragma unroll
        for (int f = 0; f < NOUT; ++f) x.put_f64((row * NF + f) * fs + k, make_double2(o0[f], o1[f]));
      }
    }
  }
  if (OUT_MODE == kOutGrid && !a.status) return;
  __syncthreads();
  if (a.status && tid < nrow && sc.bits[tid]) atomicOr(&a.status[b0 + tid], sc.bits[tid]);

  // ---- 3. weighted order spectra
  if constexpr (OUT_MODE == kOutG) {
    for (int i = tid; i < NR * NF; i += T) sc.key[i] = 0u;
    __syncthreads();
    constexpr int OS = NF;  // slot rows per member row
    for (int rf = tid >> 5; rf < nrow * NOUT; rf += T >> 5) {  // one warp per row and field
      const int row = rf / NOUT, f = rf - row * NOUT, o = row * OS + f;
      unsigned mx = 0u;
      for (int k = tid & 31; k < n; k += 32) {
        const double2 v = x.get_f64(o * fs + k);
        mx = max(mx, max(f64_key(v.x), f64_key(v.y)));
      }
      mx = __reduce_max_sync(0xffffffffu, mx);
      if ((tid & 31) == 0) {
        sc.key[o] = mx;
        sc.S[o] = f64_key_exp(mx) - hb;
      }
    }
    __syncthreads();
    w_fft_fwd<NOUT, OS>(x, nrow * NOUT, fs, a.fft, twfx, kc, sc.S);
    const double wj = a.wq ? a.wq[j] : 1.0;
    const double nan = __hiloint2double(0x7FF80000, 0);
#pragma unroll 1
    for (int idx = tid; idx < NRO * (L + 1 - a.drop); idx += T) {
      const int q = idx / NRO, rf = idx - q * NRO;  // fields fastest: contiguous global writes
      const int row = rf / NOUT, f = rf - row * NOUT, o = row * OS + f;
      if (NR > 1 && row >= nrow) continue;
      const cw zq = x.get(o * fs + __ldg(&a.irev[q])), zn = x.get(o * fs + __ldg(&a.irev[q == 0 ? 0 : n - q]));
      // R_q = (Z_q + conj Z_{n-q})/2 - (i/2) e^{-2 pi i q/N} (Z_q - conj Z_{n-q})
      const cw E{w_add(zq.re, zn.re), w_sub(zq.im, zn.im)};
      const cw D{w_sub(zq.re, zn.re), w_add(zq.im, zn.im)};
      const cw C = w_cmul<false>(D, fx_ldw(&twfx[q]));
      const cw R = cw_add_i<false>(E, C);
      const int S = sc.S[o] - 1;
      const bool bad = sc.key[o] >= kNonFinite;
      block[row * sb + (long)q * sq + f] =
          bad ? make_double2(nan, nan) : make_double2(wj * f64_of_w(R.re, S), wj * f64_of_w(R.im, S));
    }
  }
}

// ------------------------------------------------------------ direct sums
// |data|, |twiddle| <= 2^59 in limb pairs of 30 low bits (|high|, |low| <= 2^29).
// A term's two mixed products add up to at most 2^59, so 16 terms stay within
// 64 bits; the flushed sums drop their last 10 bits (2^78 a term: 2^14 terms and
// the factor 4 of both signs and both halves).
// Rounded so, the data carry 2^-60 of their row's largest value and the products
// dropped (low x low) are as small, against the 2^-53 to which an FP64 sum of
// the row rounds; 55 bits and truncation raised the error of fields with steep
// spectra by a quarter over FP64 sums.
constexpr int kDftLow = 30, kDftBits = 59, kDftTerms = 16, kDftDrop = 10;
constexpr int kDftUnit = kDftBits - kDftLow - kDftDrop;  // sums are in 2^-kDftUnit of the data's unit

// Twiddle q (cos, -sin of 2 pi q / N) in limb pairs of Q59, from the shared
// table or (rows too long for one) from the plan's Q61 table.
template <bool GTAB>
__device__ __forceinline__ int4 dft_twiddle(const int4* tab, const FxW* __restrict__ twfx, int q) {
  if constexpr (!GTAB) return tab[q];
  const FxW w = fx_ldw(&twfx[q]);
  constexpr int cut = 61 - kDftBits;
  auto q59 = [](int h, int l) { return limbs<kDftLow>((((long long)h << 31) + l + (1 << (cut - 1))) >> cut); };
  const int2 c = q59(w.ch, w.cl), s = q59(w.sh, w.sl);
  return make_int4(c.x, c.y, s.x, s.y);
}

// (sum_j a_j cos, sum_j b_j (-sin)) of angle 2 pi i j / N, j = 1..J, for FT
// fields: in units of 2^-kDftUnit of the data's unit.
template <int FT, bool GTAB>
__device__ __forceinline__ void dft_sums(const int4* __restrict__ d, int ld, int J, int i, int N, const int4* tab,
                                         const FxW* __restrict__ twfx, w96* C, w96* S) {
#pragma unroll
  for (int f = 0; f < FT; ++f) C[f] = S[f] = w96{0u, 0u, 0};
  int e = 0;
#pragma unroll 1
  for (int j0 = 1; j0 <= J; j0 += kDftTerms) {
    long long chh[FT], cx[FT], shh[FT], sx[FT];
#pragma unroll
    for (int f = 0; f < FT; ++f) chh[f] = cx[f] = shh[f] = sx[f] = 0LL;
    const int j1 = min(J + 1, j0 + kDftTerms);
#pragma unroll 2
    for (int j = j0; j < j1; ++j) {
      e += i;
      if (e >= N) e -= N;
      const int4 w = dft_twiddle<GTAB>(tab, twfx, e);
#pragma unroll
      for (int f = 0; f < FT; ++f) {
        const int4 v = d[f * ld + j];
        chh[f] = fx_madw(v.x, w.x, chh[f]);
        cx[f] = fx_madw(v.y, w.x, fx_madw(v.x, w.y, cx[f]));
        shh[f] = fx_madw(v.z, w.z, shh[f]);
        sx[f] = fx_madw(v.w, w.z, fx_madw(v.z, w.w, sx[f]));
      }
    }
#pragma unroll
    for (int f = 0; f < FT; ++f) {
      C[f] = w_add(C[f], limb_total<kDftLow, kDftDrop>(chh[f], cx[f]));
      S[f] = w_add(S[f], limb_total<kDftLow, kDftDrop>(shh[f], sx[f]));
    }
  }
}

template <int NFLD>
constexpr int dft_fields() {  // fields per thread (they share the twiddle)
  return NFLD % 3 == 0 ? 3 : NFLD % 2 == 0 ? 2 : 1;
}

template <class Pw, int IN_MODE, int OUT_MODE, bool GTAB>
__device__ __forceinline__ void row_w_dft_body(const RowArgs& a, const Pw& pw, const FxW* __restrict__ twfx, int gf,
                                               int bx, int by) {
  constexpr int NIN = Pw::NIN, NOUT = Pw::NOUT;
  constexpr int NF = NIN > NOUT ? NIN : NOUT;
  extern __shared__ uint4 smem_w[];
  __shared__ WScratch<NF> sc;
  const int j = bx, b = by, T = blockDim.x, tid = threadIdx.x;
  const int N = a.fft.N, L = a.L, half = N / 2, J = (N - 1) / 2;
  const int ld = max(L, J) + 1;  // staged values per field
  int4* tab = reinterpret_cast<int4*>(smem_w);
  int4* data = tab + (GTAB ? 0 : N);                          // [gf][ld]
  double* grid = reinterpret_cast<double*>(data + gf * ld);   // [NF][N]
  const long sq = (long)a.nblk * a.nlat;
  double2* block = nullptr;
  if (IN_MODE == kInF || OUT_MODE == kOutG) block = a.FG + fg_index(b, 0, 0, j, L, a.nblk, a.nlat);
  const double nan = __hiloint2double(0x7FF80000, 0);
  if (!GTAB)
    for (int q = tid; q < N; q += T) tab[q] = dft_twiddle<true>(nullptr, twfx, q);
  if (tid < NF) sc.bits[tid] = 0u, sc.key[tid] = 0u;
  __syncthreads();

  auto load = [&](int f, int q) {
    double2 v = block[(long)q * sq + RowSrc<Pw>::src(f)];
    if (RowSrc<Pw>::lam(f)) v = cscale((double)q * a.ir, ci(v));
    if (q == 0) v.y = 0.0;
    return v;
  };
  if constexpr (IN_MODE == kInF) {
    const int TQ = T / NIN;
    if (tid < TQ * NIN) {
      const int f = tid % NIN;
      unsigned mx = 0u;
#pragma unroll 4
      for (int q = tid / NIN; q <= L; q += TQ) {
        const double2 v = load(f, q);
        mx = max(mx, max(f64_key(v.x), f64_key(v.y)));
      }
      if (mx) atomicMax(&sc.key[f], mx);
    }
    __syncthreads();
    if (tid < NIN) sc.S[tid] = f64_key_exp(sc.key[tid]) - kDftBits;
    __syncthreads();
    constexpr int FT = dft_fields<NIN>();
    for (int g0 = 0; g0 < NIN; g0 += gf) {
      const int ng = min(gf, NIN - g0);
      for (int idx = tid; idx < ng * (L + 1); idx += T) {
        const int q = idx / ng, f = idx - q * ng;
        const double2 v = load(g0 + f, q);
        const int2 re = limbs<kDftLow>(i64_of_f64_rn(v.x, sc.S[g0 + f])), im = limbs<kDftLow>(i64_of_f64_rn(v.y, sc.S[g0 + f]));
        data[f * ld + q] = make_int4(re.x, re.y, im.x, im.y);
      }
      __syncthreads();
      // x_k, x_{N-k} = F_0 + 2 (sum Re F_m cos +- sum Im F_m (-sin))
      for (int idx = tid; idx < ng / FT * (half + 1); idx += T) {
        const int s = idx / (half + 1), k = idx - s * (half + 1);
        const int4* d = data + s * FT * ld;
        w96 C[FT], S[FT];
        dft_sums<FT, GTAB>(d, ld, L, k, N, tab, twfx, C, S);
#pragma unroll
        for (int u = 0; u < FT; ++u) {
          const int f = g0 + s * FT + u, e = sc.S[f] - kDftUnit;
          const bool bad = sc.key[f] >= kNonFinite;
          const int4 v0 = d[u * ld];
          const w96 V0 = w_shl64(((long long)v0.x << kDftLow) + v0.y, kDftUnit);
          const w96 p = w_add(C[u], S[u]), r = w_sub(C[u], S[u]);
          grid[f * N + k] = bad ? nan : f64_of_w(w_add(V0, w_add(p, p)), e);
          if (k > 0 && N - k > k) grid[f * N + N - k] = bad ? nan : f64_of_w(w_add(V0, w_add(r, r)), e);
        }
      }
      __syncthreads();
    }
  }

  {
    const double c = a.coslat[j];
    const double fg = a.fgrid ? a.fgrid[j] : 0.0;
    unsigned bits = 0u;
    for (int k = tid; k < N; k += T) {
      double in[NIN], out[NOUT];
#pragma unroll
      for (int f = 0; f < NIN; ++f)
        in[f] = IN_MODE == kInF ? grid[f * N + k] : a.gin[(long)b * a.gin_b + (long)f * a.gin_f + (long)j * N + k];
      bits |= pw(c, fg, in, out);
#pragma unroll
      for (int f = 0; f < NOUT; ++f) {
        if (OUT_MODE == kOutGrid) a.gout[(long)b * a.gout_b + (long)f * a.gout_f + (long)j * N + k] = out[f];
        else grid[f * N + k] = out[f];
      }
    }
    if (a.status && bits) atomicOr(&sc.bits[0], bits);
  }
  __syncthreads();
  if (a.status && tid == 0 && sc.bits[0]) atomicOr(&a.status[b], sc.bits[0]);

  if constexpr (OUT_MODE == kOutG) {
    constexpr int FT = dft_fields<NOUT>();
    constexpr int fb = kDftBits - 1;  // pairs x_j +- x_{N-j} take one bit more
    for (int f = tid >> 5; f < NOUT; f += T >> 5) {
      unsigned mx = 0u;
      for (int k = tid & 31; k < N; k += 32) mx = max(mx, f64_key(grid[f * N + k]));
      mx = __reduce_max_sync(0xffffffffu, mx);
      if ((tid & 31) == 0) {
        sc.key[f] = mx;
        sc.S[f] = f64_key_exp(mx) - fb;
      }
    }
    __syncthreads();
    const double wj = a.wq ? a.wq[j] : 1.0;
    const int nq = L + 1 - a.drop;
    for (int g0 = 0; g0 < NOUT; g0 += gf) {
      const int ng = min(gf, NOUT - g0);
      for (int idx = tid; idx < ng * (J + 1); idx += T) {
        const int f = idx / (J + 1), i = idx - f * (J + 1), S = sc.S[g0 + f];
        const double* x = grid + (g0 + f) * N;
        const long long X = i64_of_f64_rn(x[i], S);
        int2 p, r;
        if (i > 0) {
          const long long Y = i64_of_f64_rn(x[N - i], S);
          p = limbs<kDftLow>(X + Y);
          r = limbs<kDftLow>(X - Y);
        } else {  // x_0 and, for an even row, the point opposite
          p = limbs<kDftLow>(X);
          r = limbs<kDftLow>(N % 2 == 0 ? i64_of_f64_rn(x[half], S) : 0LL);
        }
        data[f * ld + i] = make_int4(p.x, p.y, r.x, r.y);
      }
      __syncthreads();
      for (int idx = tid; idx < ng / FT * nq; idx += T) {
        const int s = idx / nq, q = idx - s * nq;
        const int4* d = data + s * FT * ld;
        w96 C[FT], S[FT];
        dft_sums<FT, GTAB>(d, ld, J, q % N, N, tab, twfx, C, S);
#pragma unroll
        for (int u = 0; u < FT; ++u) {
          const int f = g0 + s * FT + u, e = sc.S[f] - kDftUnit;
          const int4 v0 = d[u * ld];
          const long long x0 = ((long long)v0.x << kDftLow) + v0.y, xh = ((long long)v0.z << kDftLow) + v0.w;
          const w96 re = w_add(C[u], w_shl64(x0 + (q & 1 ? -xh : xh), kDftUnit));
          const bool bad = sc.key[f] >= kNonFinite;
          block[(long)q * sq + f] =
              bad ? make_double2(nan, nan) : make_double2(wj * f64_of_w(re, e), wj * f64_of_w(S[u], e));
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- kernels
template <class Pw, int NR, int IN_MODE, int OUT_MODE>
__global__ void __launch_bounds__(kWideMaxThreads, 2) row_kernel_w(RowArgs a, Pw pw, const FxW* __restrict__ twfx,
                                                                   FxConst kc) {
  pdl_wait();
  row_w_body<Pw, NR, IN_MODE, OUT_MODE>(a, pw, twfx, kc, blockIdx.x, blockIdx.y);
}
template <class Pw, int IN_MODE, int OUT_MODE, bool GTAB>
__global__ void __launch_bounds__(kWideMaxThreads, 2) row_kernel_w_dft(RowArgs a, Pw pw, const FxW* __restrict__ twfx,
                                                                       int gf) {
  pdl_wait();
  row_w_dft_body<Pw, IN_MODE, OUT_MODE, GTAB>(a, pw, twfx, gf, blockIdx.x, blockIdx.y);
}

template <class Pw>
constexpr int w_fields() {
  return Pw::NIN > Pw::NOUT ? Pw::NIN : Pw::NOUT;
}
template <class Pw>
inline size_t row_w_smem_bytes(const FftInfo& f, int nr) {
  return (size_t)nr * w_fields<Pw>() * (f.n + 1) * (sizeof(uint4) + sizeof(uint2));
}
// Shared memory of the direct sums with `gf` staged fields.
template <class Pw>
inline size_t row_w_dft_smem(const FftInfo& f, int L, int gf, bool gtab) {
  const size_t ld = std::max(L, (f.N - 1) / 2) + 1;
  return ((gtab ? 0 : f.N) + gf * ld) * sizeof(int4) + (size_t)w_fields<Pw>() * f.N * sizeof(double);
}
// Staged fields: all of them when the row fits 96 KB (two CTAs per SM), else
// as few as one thread takes.
template <class Pw>
inline int row_w_dft_group(const FftInfo& f, int L) {
  constexpr int all = w_fields<Pw>();
  constexpr int ti = dft_fields<Pw::NIN>(), to = dft_fields<Pw::NOUT>();
  if (row_w_dft_smem<Pw>(f, L, all, false) <= 96 * 1024) return all;
  return ti > to ? (ti % to ? ti * to : ti) : (to % ti ? ti * to : to);  // a multiple of both
}

}  // namespace aeolus
