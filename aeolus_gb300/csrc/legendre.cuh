// Legendre stage of the Gauss transform of FP64 plans.
//
// Synthesis: F_m(x_j) = sum_{l=m..L} a_lm Pbar_lm(x_j), split by the parity
// of l - m so one pass over the northern rows gives both hemispheres
// (Pbar_lm(-x) = (-1)^(l-m) Pbar_lm(x)).  Analysis: a_lm = sum_j Pbar_lm(x_j)
// G_m(j) over the folded even/odd row sums.  CTAs take the order pair
// (i, L - i) so every CTA contracts the same L + 2 degrees.
//
// Functor contracts (shared with the point-set path):
//   Derive:   NF fields; column(b, l, m, double2 v[NF]) gives the spectral
//             coefficients to synthesise (derived from the caller's input).
//   Epilogue: NF analysed fields; finish(b, l, m, const double2 acc[NF])
//             consumes a_lm for l >= m; zero(b, l, m) handles l < m slots.
#pragma once

#include <type_traits>
#include <utility>

#include "common.cuh"
#include "w96.cuh"

namespace aeolus {

// Highest degree and order an epilogue uses of the analysed fields.  The
// tendencies and the Jacobian cut their products to the 2/3 rule (degrees and
// orders up to 2L/3), so 56 % of the triangle of an analysis would be thrown
// away: their epilogues declare kCut, the row stage then writes no order above
// the cut and the contraction runs over the kept triangle only (an epilogue
// still visits every slot, with zeros for the cut ones).
template <class E, class = void>
struct EpiTop {
  __host__ __device__ static int top(int L) { return L; }
};
template <class E>
struct EpiTop<E, std::enable_if_t<E::kCut>> {
  __host__ __device__ static int top(int L) { return (2 * L) / 3; }
};
// kCutPlus: one degree more, which the weak-form curl and divergence of the
// degrees up to the cut read.
template <class E>
struct EpiTop<E, std::enable_if_t<E::kCutPlus>> {
  __host__ __device__ static int top(int L) { return (2 * L) / 3 + 1 < L ? (2 * L) / 3 + 1 : L; }
};

struct LegArgs {
  int L, nlat, nh, batch, bc;
  int ss;            // CTAs that share the items of one (order pair, member chunk)
  int rb;            // synthesis: rows per warp (8, 16 or 32)
  int js;            // analysis: lanes that share the rows of one degree
  int solo;          // analysis: one order per CTA (rows too many for a pair's shared memory)
  const int2* P;     // synthesis table, limb pairs (row index fastest)
  const int* eP;     // [m][nh] exponents of its (order, row) columns
  const int2* PT;    // analysis table, limb pairs (degree fastest)
  const int* ePT;    // exponents of its (order, degree) columns, packed triangle
  double2* FG;       // F / G blocks [b][j][nblk][L+1]
  int nblk;
};

__host__ __device__ inline int n_pairs(int L) { return L / 2 + 1; }

// FP64 contraction in integers.  The FP64 pipe's 2 DFMA per clock and SM bound
// these sums (8 members at l_max 127: 184 and 93 us per stage), while the 32 x
// 32 -> 64-bit multiply-add runs at up to 32 times that rate.  So every factor
// is held as a 59-bit integer in two limbs, the basis at one exponent
// per (order, row) or (order, degree) and the data at one per (member, field,
// order) column; a product is three multiply-adds into two 64-bit sums, which
// stay exact, and each result is rounded to FP64 once.  The error is that of
// the limbs, 2^-60 of the largest factors per term, against a rounding of
// 2^-53 of the running sum per FP64 multiply-add; an infinity or NaN in a
// column makes all its results NaN, as in FP64.  The sums being exact, results
// depend neither on the launch shape nor on the batch.
// Work items are the smallest independent ones, packed densely over the
// threads:
//   synthesis  (northern row, data column) per item;
//   analysis   (degree, one of js row slices) per item, the slices of a degree
//              in neighbouring lanes and added by shuffles;
// and the items of one (order pair, member chunk) are shared by `ss` CTAs when
// there are too few of those to fill the chip (leg_shares, pipeline.cuh).
// Measured per stage (7 or 4 fields, before -> after): synthesis 184 -> 85 us
// and analysis 93 -> 51 us at 8 members, l_max 127, 192 rows; 14 -> 10.6 and
// 14 -> 14.8 us at one member, l_max 85, 128 rows, where the preparation (the
// derived columns and their limbs, 10 us of serial latency) is what is left.
// At 8 members the multiply-adds would take 21 us of the synthesis; the
// preparation takes 29 and the sums 55, at 1.5 of 4 instructions per clock and
// 11 warps per SM, which neither other unrollings, residencies nor a prefetch
// of the basis moved (80 to 94 us).
template <class Derive, int CPT>
__device__ __forceinline__ void legendre_synth_body(const LegArgs& a, const Derive& d, int bx, int by) {
  constexpr int NF = Derive::NF;
  extern __shared__ double2 s_a[];
  const int L = a.L, nh = a.nh;
  const int share = bx % a.ss, b0 = by * a.bc;
  const int i = bx / a.ss;
  const int mA = i, mB = L - i;
  const bool two = mB != mA;
  const int KA = L + 1 - mA, KB = two ? L + 1 - mB : 0;
  const int nb = min(a.bc, a.batch - b0);
  const int ncols = nb * NF;
  double2* sA = s_a;                     // [ncols][KA], FP64, then limb pairs
  double2* sB = s_a + (long)ncols * KA;  // [ncols][KB]
  unsigned* key = reinterpret_cast<unsigned*>(s_a + (long)ncols * (KA + KB));  // [2][ncols]

  // derived coefficient columns of both orders, then their largest keys
  for (int idx = threadIdx.x; idx < nb * (KA + KB); idx += blockDim.x) {
    const int bl = idx / (KA + KB);
    const int t = idx - bl * (KA + KB);
    const bool isA = t < KA;
    const int m = isA ? mA : mB;
    const int tt = isA ? t : t - KA;
    const int K = isA ? KA : KB;
    double2 v[NF];
    d.column(b0 + bl, m + tt, m, v);
    double2* dst = isA ? sA : sB;
#pragma unroll
    for (int f = 0; f < NF; ++f) dst[(long)(bl * NF + f) * K + tt] = v[f];
  }
  __syncthreads();
  for (int c = threadIdx.x >> 5; c < (two ? 2 : 1) * ncols; c += blockDim.x >> 5) {  // one warp per column
    const int K = c < ncols ? KA : KB;
    const double2* v = c < ncols ? sA + (long)c * KA : sB + (long)(c - ncols) * KB;
    unsigned k = 0u;
    for (int t = threadIdx.x & 31; t < K; t += 32) k = max(k, max(f64_key(v[t].x), f64_key(v[t].y)));
    k = __reduce_max_sync(0xffffffffu, k);
    if ((threadIdx.x & 31) == 0) key[c] = k;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < ncols * (KA + KB); idx += blockDim.x) {  // to limb pairs, in place
    const bool isA = idx < ncols * KA;
    const int c = isA ? idx / KA : (idx - ncols * KA) / KB;
    const int S = f64_key_exp(key[(isA ? 0 : ncols) + c]) - kLegBits;
    const double2 v = s_a[idx];
    const int2 re = limbs<kLegLow>(i64_of_f64_rn(v.x, S)), im = limbs<kLegLow>(i64_of_f64_rn(v.y, S));
    reinterpret_cast<int4*>(s_a)[idx] = make_int4(re.x, re.y, im.x, im.y);
  }
  __syncthreads();

  // A warp takes rb rows of 32 / rb neighbouring slots of CPT columns; the
  // columns of one row block follow each other, so the warps of a CTA read the
  // same basis lines about the same time.
  const int rb = a.rb, cpw = 32 / rb * CPT, cg = (ncols + cpw - 1) / cpw;
  const int units = (nh + rb - 1) / rb * cg, per = (units + a.ss - 1) / a.ss;
  const int lane = threadIdx.x & 31;
  for (int u = share * per + (threadIdx.x >> 5); u < min(units, (share + 1) * per); u += blockDim.x >> 5) {
    const int jb = u / cg, c = (u - jb * cg) * cpw + lane / rb * CPT, jn = jb * rb + lane % rb;
    if (c >= ncols || jn >= nh) continue;
    const int jS = a.nlat - 1 - jn;
#pragma unroll 1
    for (int pass = 0; pass < (two ? 2 : 1); ++pass) {
      const int m = pass ? mB : mA;
      const int K = pass ? KB : KA;
      // the last slot of an odd column count repeats its column (stored once)
      const int4* sc[CPT];
#pragma unroll
      for (int q = 0; q < CPT; ++q)
        sc[q] = reinterpret_cast<const int4*>(pass ? sB : sA) + (long)min(c + q, ncols - 1) * K;
      const int2* Pm = a.P + tri_off(m, L) * nh + jn;
      w96 Ex[CPT], Ey[CPT], Ox[CPT], Oy[CPT];
#pragma unroll
      for (int q = 0; q < CPT; ++q) Ex[q] = Ey[q] = Ox[q] = Oy[q] = w96{0u, 0u, 0};
#pragma unroll 1
      for (int t0 = 0; t0 < K; t0 += 2 * kLegTerms) {
        const int t1 = min(K, t0 + 2 * kLegTerms);
        long long eh[CPT][2], el[CPT][2], oh[CPT][2], ol[CPT][2];
#pragma unroll
        for (int q = 0; q < CPT; ++q) eh[q][0] = eh[q][1] = el[q][0] = el[q][1] = oh[q][0] = oh[q][1] = ol[q][0] = ol[q][1] = 0LL;
        auto term = [&](int2 p, int4 v, long long* h, long long* l) {
          h[0] = fx_madw(p.x, v.x, h[0]);
          l[0] = fx_madw(p.x, v.y, fx_madw(p.y, v.x, l[0]));
          h[1] = fx_madw(p.x, v.z, h[1]);
          l[1] = fx_madw(p.x, v.w, fx_madw(p.y, v.z, l[1]));
        };
        const int2* pt = Pm + (long)t0 * nh;
        int t = t0;
#pragma unroll 4
        for (; t + 1 < t1; t += 2) {
          const int2 pe = __ldg(pt), po = __ldg(pt + nh);
          pt += 2 * nh;
#pragma unroll
          for (int q = 0; q < CPT; ++q) {
            term(pe, sc[q][t], eh[q], el[q]);
            term(po, sc[q][t + 1], oh[q], ol[q]);
          }
        }
        if (t < t1) {
          const int2 pe = __ldg(pt);
#pragma unroll
          for (int q = 0; q < CPT; ++q) term(pe, sc[q][t], eh[q], el[q]);
        }
#pragma unroll
        for (int q = 0; q < CPT; ++q) {
          Ex[q] = w_add(Ex[q], limb_total<kLegLow, kLegDrop>(eh[q][0], el[q][0]));
          Ey[q] = w_add(Ey[q], limb_total<kLegLow, kLegDrop>(eh[q][1], el[q][1]));
          Ox[q] = w_add(Ox[q], limb_total<kLegLow, kLegDrop>(oh[q][0], ol[q][0]));
          Oy[q] = w_add(Oy[q], limb_total<kLegLow, kLegDrop>(oh[q][1], ol[q][1]));
        }
      }
      const int eP = __ldg(a.eP + (long)m * nh + jn);
      const double nan = __hiloint2double(0x7FF80000, 0);
#pragma unroll
      for (int q = 0; q < CPT; ++q) {
        if (c + q >= ncols) break;
        const int bl = (c + q) / NF, f = c + q - bl * NF;
        const unsigned k = key[(pass ? ncols : 0) + c + q];
        const int S = f64_key_exp(k) + eP - 2 * kLegBits + kLegLow + kLegDrop;
        const bool bad = k >= kNonFinite;
        double2* out = a.FG + fg_index(b0 + bl, m, f, jn, L, a.nblk, a.nlat);
        *out = bad ? make_double2(nan, nan)
                   : make_double2(f64_of_w(w_add(Ex[q], Ox[q]), S), f64_of_w(w_add(Ey[q], Oy[q]), S));
        if (jS != jn)
          out[(long)(jS - jn) * a.nblk] =
              bad ? make_double2(nan, nan)
                  : make_double2(f64_of_w(w_sub(Ex[q], Ox[q]), S), f64_of_w(w_sub(Ey[q], Oy[q]), S));
      }
    }
  }
}

template <class Derive, int CPT>
__global__ void __launch_bounds__(256, 2) legendre_synth_kernel(LegArgs a, Derive d) {
  pdl_wait();
  legendre_synth_body<Derive, CPT>(a, d, blockIdx.x, blockIdx.y);
}

template <class Derive>
inline size_t synth_smem_bytes(int L, int bc) {
  return (size_t)bc * Derive::NF * ((L + 2) * sizeof(double2) + 2 * sizeof(unsigned));
}

template <class Epi>
__device__ __forceinline__ void legendre_analysis_body(const LegArgs& a, const Epi& e, int bx, int by) {
  constexpr int NF = Epi::NF;
  extern __shared__ double2 s_g[];  // [2 orders][nb][NF][2 parities][nh], FP64 rows, then limb pairs; keys
  const int L = a.L, nh = a.nh, top = EpiTop<Epi>::top(L);
  const int share = bx % a.ss, b0 = by * a.bc;
  const int i = bx / a.ss;
  const int mA = i, mB = a.solo ? i : top - i;
  const bool two = mB != mA;
  const int KA = top + 1 - mA, KB = two ? top + 1 - mB : 0;
  const int nb = min(a.bc, a.batch - b0);
  const int JS = a.js;
  const int per_order = a.bc * NF * 2 * nh;
  unsigned* key = reinterpret_cast<unsigned*>(s_g + (a.solo ? 1 : 2) * (long)per_order);  // [2][bc][NF]

  const int nrows = (two ? 2 : 1) * nb * NF * nh;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < nrows; idx += blockDim.x) {
    int r = idx;
    const int f = r % NF; r /= NF;
    const int jn = r % nh; r /= nh;
    const int bl = r % nb; r /= nb;
    const int which = r;
    const int m = which ? mB : mA;
    const long bb = b0 + bl;
    const int jS = a.nlat - 1 - jn;
    const double2 gN = a.FG[fg_index(bb, m, f, jn, L, a.nblk, a.nlat)];
    const double2 gS = jS != jn ? a.FG[fg_index(bb, m, f, jS, L, a.nblk, a.nlat)] : make_double2(0.0, 0.0);
    double2* dst = s_g + which * per_order + ((bl * NF + f) * 2) * nh;
    dst[jn] = gN;
    dst[nh + jn] = gS;
  }
  __syncthreads();
  for (int c = threadIdx.x >> 5; c < (two ? 2 : 1) * nb * NF; c += blockDim.x >> 5) {  // one warp per (order, field)
    const int which = c / (nb * NF), cc = c - which * nb * NF;
    const double2* v = s_g + which * per_order + cc * 2 * nh;
    unsigned k = 0u;
    for (int r = threadIdx.x & 31; r < 2 * nh; r += 32) k = max(k, max(f64_key(v[r].x), f64_key(v[r].y)));
    k = __reduce_max_sync(0xffffffffu, k);
    if ((threadIdx.x & 31) == 0) key[which * a.bc * NF + cc] = k;
  }
  __syncthreads();
  // fold the hemispheres (exactly, in integers) into even and odd limb pairs
  for (int idx = threadIdx.x; idx < nrows; idx += blockDim.x) {
    int r = idx;
    const int jn = r % nh; r /= nh;
    const int c = r % (nb * NF), which = r / (nb * NF);  // c = bl NF + f
    double2* src = s_g + which * per_order + c * 2 * nh + jn;
    const double2 gN = src[0], gS = src[nh];
    const int S = f64_key_exp(key[which * a.bc * NF + c]) - (kLegBits - 1);  // a sum has one bit more
    const long long nx = i64_of_f64_rn(gN.x, S), ny = i64_of_f64_rn(gN.y, S);
    const long long sx = i64_of_f64_rn(gS.x, S), sy = i64_of_f64_rn(gS.y, S);
    const int2 er = limbs<kLegLow>(nx + sx), ei = limbs<kLegLow>(ny + sy);
    const int2 or_ = limbs<kLegLow>(nx - sx), oi = limbs<kLegLow>(ny - sy);
    *reinterpret_cast<int4*>(src) = make_int4(er.x, er.y, ei.x, ei.y);
    *reinterpret_cast<int4*>(src + nh) = make_int4(or_.x, or_.y, oi.x, oi.y);
  }
  __syncthreads();

  // degrees of this CTA: [d0, d1) of the nb (KA + KB) (member, degree) pairs;
  // every lane of a warp runs the same number of rounds (the shuffles)
  const int KT = KA + KB;
  const int per = (nb * KT + a.ss - 1) / a.ss;
  const int d0 = share * per, d1 = min(nb * KT, d0 + per);
  const int nitem = max(0, d1 - d0) * JS;
  for (int base = threadIdx.x & ~31; base < nitem; base += blockDim.x) {
    const int item = base + (threadIdx.x & 31);
    const bool on = item < nitem;
    const int di = on ? item / JS : 0, js = item % JS;
    const int bl = (d0 + di) / KT;
    const int t0 = d0 + di - bl * KT;
    const bool isA = t0 < KA;
    const int m = isA ? mA : mB;
    const int t = isA ? t0 : t0 - KA;
    const int K = L + 1 - m;
    const int4* sg = reinterpret_cast<const int4*>(s_g) + (isA ? 0 : per_order) + (bl * NF * 2 + (t & 1)) * nh;
    const int2* pt = a.PT + tri_off(m, L) * nh + t;
    w96 sx[NF], sy[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) sx[f] = sy[f] = w96{0u, 0u, 0};
#pragma unroll 1
    for (int j0 = js; j0 < (on ? nh : 0); j0 += kLegTerms * JS) {
      long long xh[NF], xl[NF], yh[NF], yl[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) xh[f] = xl[f] = yh[f] = yl[f] = 0LL;
      const int j1 = min(nh, j0 + kLegTerms * JS);
#pragma unroll 4
      for (int jn = j0; jn < j1; jn += JS) {
        const int2 p = __ldg(pt + (long)jn * K);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          const int4 g = sg[f * 2 * nh + jn];
          xh[f] = fx_madw(p.x, g.x, xh[f]);
          xl[f] = fx_madw(p.x, g.y, fx_madw(p.y, g.x, xl[f]));
          yh[f] = fx_madw(p.x, g.z, yh[f]);
          yl[f] = fx_madw(p.x, g.w, fx_madw(p.y, g.z, yl[f]));
        }
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        sx[f] = w_add(sx[f], limb_total<kLegLow, kLegDrop>(xh[f], xl[f]));
        sy[f] = w_add(sy[f], limb_total<kLegLow, kLegDrop>(yh[f], yl[f]));
      }
    }
    const int eP = on ? __ldg(a.ePT + tri_off(m, L) + t) : 0;
    const double nan = __hiloint2double(0x7FF80000, 0);
    auto result = [&](w96 v, int f) {
      const unsigned k = key[((isA ? 0 : a.bc) + bl) * NF + f];
      return k >= kNonFinite ? nan : f64_of_w(v, f64_key_exp(k) + eP - (2 * kLegBits - 1) + kLegLow + kLegDrop);
    };
    double2 acc[NF];
    if (JS == 1) {
#pragma unroll
      for (int f = 0; f < NF; ++f) acc[f] = make_double2(result(sx[f], f), result(sy[f], f));
    } else {
      // add the slices; the lanes of a degree round its 2 NF sums in turn
      // (value v by lane v mod JS) and share them
      auto add = [&](w96 v) {
        for (int o = JS >> 1; o > 0; o >>= 1)
          v = w_add(v, w96{__shfl_xor_sync(0xffffffffu, v.l, o), __shfl_xor_sync(0xffffffffu, v.m, o),
                           __shfl_xor_sync(0xffffffffu, v.h, o)});
        return v;
      };
#pragma unroll
      for (int f = 0; f < NF; ++f) sx[f] = add(sx[f]), sy[f] = add(sy[f]);
#pragma unroll 1
      for (int v0 = 0; v0 < 2 * NF; v0 += JS) {
        w96 mine = sx[0];
        const int want = v0 + js;
#pragma unroll
        for (int v = 1; v < 2 * NF; ++v)
          if (v == want) mine = v & 1 ? sy[v >> 1] : sx[v >> 1];
        const double r = result(mine, min(want, 2 * NF - 1) >> 1);
#pragma unroll
        for (int v = 0; v < 2 * NF; ++v) {
          const double x = __shfl_sync(0xffffffffu, r, v - v0, JS);
          if (v >= v0 && v < v0 + JS) (v & 1 ? acc[v >> 1].y : acc[v >> 1].x) = x;
        }
      }
    }
    if (on && js == 0) e.finish(b0 + bl, m + t, m, acc);
  }
  // the slots outside the kept triangle, shared by every CTA of these members
  const int n2 = (L + 1) * (L + 1), ncta = (a.solo ? top + 1 : n_pairs(top)) * a.ss;
  const double2 none[NF] = {};
  for (int idx = bx * blockDim.x + threadIdx.x; idx < nb * n2; idx += ncta * blockDim.x) {
    const int bl = idx / n2, r = idx - bl * n2;
    const int l = r / (L + 1), m = r - l * (L + 1);
    if (m > l) e.zero(b0 + bl, l, m);
    else if (l > top) e.finish(b0 + bl, l, m, none);
  }
}

template <class Epi>
__global__ void __launch_bounds__(256, Epi::NF <= 4 ? 2 : 1) legendre_analysis_kernel(LegArgs a, Epi e) {
  pdl_wait();
  legendre_analysis_body<Epi>(a, e, blockIdx.x, blockIdx.y);
}

template <class Epi>
inline size_t analysis_smem_bytes(int nh, int bc, int solo) {
  return (size_t)(solo ? 1 : 2) * bc * Epi::NF * 2 * nh * sizeof(double2) + (size_t)2 * bc * Epi::NF * sizeof(unsigned);
}

// ------------------------------------------------------------ plain functors
struct DeriveCopy {  // synthesis input: dense [b][L+1][L+1]
  static constexpr int NF = 1;
  const double2* in;
  int L;
  long bstride;
  __device__ void column(int b, int l, int m, double2* v) const {
    v[0] = in[(long)b * bstride + (long)l * (L + 1) + m];
  }
};

struct EpiStore {  // analysis output: dense [b][L+1][L+1]
  static constexpr int NF = 1;
  double2* out;
  int L;
  long bstride;
  __device__ void finish(int b, int l, int m, const double2* acc) const {
    out[(long)b * bstride + (long)l * (L + 1) + m] = acc[0];
  }
  __device__ void zero(int b, int l, int m) const {
    out[(long)b * bstride + (long)l * (L + 1) + m] = make_double2(0.0, 0.0);
  }
};

}  // namespace aeolus
