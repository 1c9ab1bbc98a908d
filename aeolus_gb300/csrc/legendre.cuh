// Legendre stage of the Gauss transform (FP64 contraction).
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
  int solo;          // analysis: one order per CTA (rows too many for a pair's shared memory)
  const double* P;   // synthesis table (row index fastest)
  const double* PT;  // analysis table (degree fastest)
  double2* FG;       // F / G blocks [b][j][nblk][L+1]
  int nblk;
};

__host__ __device__ inline int n_pairs(int L) { return L / 2 + 1; }

// Both kernels are bound by the FP64 pipe (2 DFMA per clock and SM: a warp's
// DFMA occupies its sub-partition for 64 cycles, so one warp with two
// independent sums per sub-partition already saturates it and the loads that
// feed it are free).  What costs is idle lanes and idle SMs, so the work items
// are the smallest independent ones, packed densely over the threads:
//   synthesis  (northern row, data column) per item;
//   analysis   (degree, one of JS row slices) per item, the slices added
//              through shared memory; JS depends on the grid alone, so a
//              member's result does not depend on the batch;
// and the items of one (order pair, member chunk) are shared by `ss` CTAs when
// there are too few of those to fill the chip (leg_shares, pipeline.cuh).
// FP64 SWE RK4 steps with these kernels and the kept-triangle analysis: one
// member at 128 x 256, l_max 85 505 -> 377 us (analysis 30.4 -> 14.6 us per
// stage), 8 members at 192 x 384, l_max 127 3.30 -> 2.91 ms (analysis 142 -> 93 us
// per stage; synthesis of 7 fields 184 us).
// The sums are in FP64 because rows and degrees of one order differ by many
// decades: P_mm next to a pole is 1e-70 of its equatorial value at m = 40, and a
// steep spectrum falls as far.  59-bit integers at one exponent per column (85 and
// 51 us) keep the norm of a field but not its rows: a field of the single
// coefficient l = m = 20 came out as zeros next to the poles and 3e-5 off at row 12
// of 192, where these sums are 9e-15 off.
template <class Derive>
__device__ __forceinline__ void legendre_synth_body(const LegArgs& a, const Derive& d, int bx, int by) {
  constexpr int NF = Derive::NF;
  extern __shared__ double2 s_a[];
  const int L = a.L, nh = a.nh;
  const int i = bx / a.ss;
  const int mA = i, mB = L - i;
  const bool two = mB != mA;
  const int KA = L + 1 - mA, KB = two ? L + 1 - mB : 0;
  const int share = bx % a.ss, b0 = by * a.bc;
  const int nb = min(a.bc, a.batch - b0);
  const int ncols = nb * NF;
  double2* sA = s_a;                   // [ncols][KA]
  double2* sB = s_a + (long)ncols * KA;  // [ncols][KB]

  // derived coefficient columns of both orders
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

  const int items = nh * ncols, per = (items + a.ss - 1) / a.ss;
  for (int item = share * per + threadIdx.x; item < min(items, (share + 1) * per); item += blockDim.x) {
    const int c = item / nh, jn = item - c * nh;
    const int jS = a.nlat - 1 - jn;
    const int bl = c / NF, f = c - bl * NF;
    for (int pass = 0; pass < (two ? 2 : 1); ++pass) {
      const int m = pass ? mB : mA;
      const int K = pass ? KB : KA;
      const double2* sc = (pass ? sB : sA) + (long)c * K;
      const double* Pm = a.P + tri_off(m, L) * nh + jn;
      double2 E = make_double2(0.0, 0.0), O = E;
      int t = 0;
#pragma unroll 4
      for (; t + 1 < K; t += 2) {
        const double pe = __ldg(Pm + (long)t * nh);
        const double po = __ldg(Pm + (long)(t + 1) * nh);
        const double2 ae = sc[t], ao = sc[t + 1];
        E.x = fma(pe, ae.x, E.x);
        E.y = fma(pe, ae.y, E.y);
        O.x = fma(po, ao.x, O.x);
        O.y = fma(po, ao.y, O.y);
      }
      if (t < K) {
        const double pe = __ldg(Pm + (long)t * nh);
        const double2 ae = sc[t];
        E.x = fma(pe, ae.x, E.x);
        E.y = fma(pe, ae.y, E.y);
      }
      const long bb = b0 + bl;
      a.FG[fg_index(bb, m, f, jn, L, a.nblk, a.nlat)] = cadd(E, O);
      if (jS != jn) a.FG[fg_index(bb, m, f, jS, L, a.nblk, a.nlat)] = csub(E, O);
    }
  }
}

template <class Derive>
__global__ void __launch_bounds__(256) legendre_synth_kernel(LegArgs a, Derive d) {
  pdl_wait();
  legendre_synth_body<Derive>(a, d, blockIdx.x, blockIdx.y);
}

template <class Derive>
inline size_t synth_smem_bytes(int L, int bc) {
  return (size_t)bc * Derive::NF * (L + 2) * sizeof(double2);
}

// Row slices per degree of the analysis (a power of two, from the grid and the
// field count alone).  Rows that fill most of the shared memory by themselves
// (above 160 KB) leave no room for partial sums: one slice, finished directly.
__host__ __device__ inline int leg_row_slices(int nh, int nf) {
  return (long)64 * nf * nh > 160 * 1024 ? 1 : nh >= 32 ? 8 : nh >= 8 ? 4 : 1;
}

template <class Epi>
__device__ __forceinline__ void legendre_analysis_body(const LegArgs& a, const Epi& e, int bx, int by) {
  constexpr int NF = Epi::NF;
  extern __shared__ double2 s_g[];  // [2 orders, solo: 1][nb][NF][2 parities][nh], then [items / JS][JS][NF] partial sums
  const int L = a.L, nh = a.nh, top = EpiTop<Epi>::top(L);
  const int i = bx / a.ss;
  const int mA = i, mB = a.solo ? i : top - i;
  const bool two = mB != mA;
  const int KA = top + 1 - mA, KB = two ? top + 1 - mB : 0;
  const int share = bx % a.ss, b0 = by * a.bc;
  const int nb = min(a.bc, a.batch - b0);
  const int JS = leg_row_slices(nh, NF);
  const long per_order = (long)a.bc * NF * 2 * nh;

  for (int idx = threadIdx.x; idx < (two ? 2 : 1) * nb * NF * nh; idx += blockDim.x) {
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
    double2* dst = s_g + which * per_order + ((long)(bl * NF + f) * 2) * nh;
    dst[jn] = cadd(gN, gS);
    dst[nh + jn] = csub(gN, gS);
  }
  __syncthreads();

  // degrees of this CTA: [d0, d1) of the nb (KA + KB) (member, degree) pairs
  const int KT = KA + KB;
  const int per = (nb * KT + a.ss - 1) / a.ss;
  const int d0 = share * per, d1 = min(nb * KT, d0 + per);
  double2* part = s_g + (a.solo ? 1 : 2) * per_order;
  for (int item = threadIdx.x; item < (d1 - d0) * JS; item += blockDim.x) {
    const int di = item / JS, js = item - di * JS;
    const int bl = (d0 + di) / KT;
    const int t0 = d0 + di - bl * KT;
    const bool isA = t0 < KA;
    const int m = isA ? mA : mB;
    const int t = isA ? t0 : t0 - KA;
    const int K = L + 1 - m;
    const int par = t & 1;
    const double2* sg = s_g + (isA ? 0 : per_order) + ((long)bl * NF * 2 + par) * nh;
    const double* pt = a.PT + tri_off(m, L) * nh + t;
    double2 acc[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int jn = js; jn < nh; jn += JS) {
      const double p = __ldg(pt + (long)jn * K);
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const double2 g = sg[(long)f * 2 * nh + jn];
        acc[f].x = fma(p, g.x, acc[f].x);
        acc[f].y = fma(p, g.y, acc[f].y);
      }
    }
    if (JS == 1) {
      e.finish(b0 + bl, m + t, m, acc);
    } else {
#pragma unroll
      for (int f = 0; f < NF; ++f) part[(long)item * NF + f] = acc[f];
    }
  }
  if (JS > 1) {
    __syncthreads();
    // the slices of one (degree, field) added in slice order, dense over the threads
    for (int idx = threadIdx.x; idx < (d1 - d0) * NF; idx += blockDim.x) {
      const int di = idx / NF, f = idx - di * NF;
      double2* q = part + (long)di * JS * NF + f;
      double2 s = q[0];
      for (int js = 1; js < JS; ++js) s = cadd(s, q[js * NF]);
      q[0] = s;
    }
    __syncthreads();
    for (int di = threadIdx.x; di < d1 - d0; di += blockDim.x) {
      const int bl = (d0 + di) / KT;
      const int t0 = d0 + di - bl * KT;
      const bool isA = t0 < KA;
      const int m = isA ? mA : mB;
      const double2* q = part + (long)di * JS * NF;
      double2 acc[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) acc[f] = q[f];
      e.finish(b0 + bl, m + (isA ? t0 : t0 - KA), m, acc);
    }
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
__global__ void __launch_bounds__(256) legendre_analysis_kernel(LegArgs a, Epi e) {
  pdl_wait();
  legendre_analysis_body<Epi>(a, e, blockIdx.x, blockIdx.y);
}

template <class Epi>
inline size_t analysis_smem_bytes(int L, int nh, int bc, int ss, int solo) {
  const int top = EpiTop<Epi>::top(L);
  const size_t degrees = ((size_t)bc * (top + 2) + ss - 1) / ss;
  const int js = leg_row_slices(nh, Epi::NF);
  return ((size_t)(solo ? 1 : 2) * bc * Epi::NF * 2 * nh + (js > 1 ? degrees * js * Epi::NF : 0)) * sizeof(double2);
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
