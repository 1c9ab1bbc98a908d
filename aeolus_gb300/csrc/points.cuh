// Point-set (e.g. icosahedral geodesic) transform: dense real basis product.
//
// Real basis columns, m-major: for each order m the cosine columns
// Pbar_lm cos(m lon) for l = m..L, then (m > 0) the sine columns
// Pbar_lm sin(m lon); (L+1)^2 columns in all, stored column-major
// (point index fastest).  With that basis the reference's complex forms
// (fast_geodesic_sh.py:68-107) become real GEMMs:
//   synthesis  f = B v,  v[cos(l,0)] = Re a_l0, v[cos(l,m)] = 2 Re a_lm,
//                        v[sin(l,m)] = -2 Im a_lm;
//   analysis   c = B^T (w f),  a_lm = c[cos(l,m)] - i c[sin(l,m)].
#pragma once

#include "common.cuh"

namespace aeolus {

__host__ __device__ inline long col_base(int m, int L) { return m == 0 ? 0 : 2 * tri_off(m, L) - (L + 1); }
__host__ __device__ inline long col_cos(int l, int m, int L) { return col_base(m, L) + (l - m); }
__host__ __device__ inline long col_sin(int l, int m, int L) { return col_base(m, L) + (L + 1 - m) + (l - m); }

// V[(b*NF + f) * ncol + col] from Derive columns (one thread per (b, l, m) of
// the dense square, orders fastest: coalesced reads, no search for the order).
template <class Derive>
__global__ void derive_cols_kernel(int L, int batch, long ncol, double* __restrict__ V, Derive d) {
  pdl_wait();
  constexpr int NF = Derive::NF;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n2 * batch) return;
  const int b = (int)(idx / n2);
  const int r = (int)(idx - (long)b * n2);
  const int l = r / (L + 1), m = r - l * (L + 1);
  if (m > l) return;
  double2 v[NF];
  d.column(b, l, m, v);
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    double* col = V + ((long)b * NF + f) * ncol;
    if (m == 0) {
      col[col_cos(l, 0, L)] = v[f].x;
    } else {
      col[col_cos(l, m, L)] = 2.0 * v[f].x;
      col[col_sin(l, m, L)] = -2.0 * v[f].y;
    }
  }
}

// Pointwise op over points.  in: Gr[b * in_b + f * in_f + p];
// out: Out[b * out_b + f * out_f + p] = scale_p * out_f with scale_p = w_p
// (analysis input) or 1 (grid output).
template <class Pw>
__global__ void points_pointwise_kernel(long npts, int batch, const double* __restrict__ Gr, long in_b, long in_f,
                                        double* __restrict__ Out, long out_b, long out_f,
                                        const double* __restrict__ coslat, const double* __restrict__ fgrid,
                                        const double* __restrict__ w, unsigned* status, Pw pw) {
  pdl_wait();
  constexpr int NIN = Pw::NIN, NOUT = Pw::NOUT;
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= npts * batch) return;
  const int b = (int)(idx / npts);
  const long p = idx - (long)b * npts;
  double in[NIN], out[NOUT];
#pragma unroll
  for (int f = 0; f < NIN; ++f) in[f] = __ldcg(Gr + (long)b * in_b + (long)f * in_f + p);
  const unsigned bits = pw(coslat[p], fgrid[p], in, out);
  if (status && bits) atomicOr(&status[b], bits);
  const double sc = w ? w[p] : 1.0;
#pragma unroll
  for (int f = 0; f < NOUT; ++f) Out[(long)b * out_b + (long)f * out_f + p] = sc * out[f];
}

// a_lm from real analysis columns; one thread per (b, l, m) of the dense square.
template <class Epi>
__global__ void epilogue_cols_kernel(int L, int batch, long ncol, const double* __restrict__ C, Epi e) {
  pdl_wait();
  constexpr int NF = Epi::NF;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n2 * batch) return;
  const int b = (int)(idx / n2);
  const int r = (int)(idx - (long)b * n2);
  const int l = r / (L + 1), m = r - l * (L + 1);
  if (m > l) {
    e.zero(b, l, m);
    return;
  }
  double2 acc[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    const double* col = C + ((long)b * NF + f) * ncol;
    acc[f] = make_double2(__ldcg(col + col_cos(l, m, L)), m == 0 ? 0.0 : -__ldcg(col + col_sin(l, m, L)));
  }
  e.finish(b, l, m, acc);
}

// FP64 basis products.  GB300's FP64 pipe does 2 DFMA per clock and SM
// (629 G/s at 2070 MHz) while HBM delivers 840 G basis values/s, so from two
// data columns on the products are bound by the multiply-adds themselves:
// what counts is to issue only useful ones, on every SM.  Each CTA takes
// exactly the columns there are (NT <= 8 per pass, a template argument) and
// the contraction is split over its threads, so one field on a small point
// set (a resolution-4 run: 10,242 product points x 441 columns, 4 + 1 columns
// per stage) still covers the chip.  The order of each output's sum depends
// on the plan's sizes only, not on the batch.  Against the square 64 x 32
// tile this replaces (padded to 32 columns, 7 CTAs in the analysis), a BVE
// RK4 step of that run went from 29.84 to 0.275 ms; its multiply-adds alone
// take 0.145 ms at the FP64 rate.
constexpr int kPtThreads = 256;
constexpr int kPtCols = 8;      // data columns per pass
constexpr int kPtRows = 16;     // synthesis: points per CTA (one 128-byte line per basis column)
constexpr int kPtSlices = kPtThreads / kPtRows;
constexpr int kPtChunk = 256;   // synthesis: basis columns per staged chunk

// out[n * M + p] = sum_k B[k * M + p] V[n * K + k]: 16 points x 16 slices of
// the basis columns per CTA; the chunk's coefficients sit in shared memory.
template <int NT>
__global__ void __launch_bounds__(kPtThreads) points_synth_kernel(long M, int K, int N, const double* __restrict__ B,
                                                                  const double* __restrict__ V,
                                                                  double* __restrict__ out) {
  pdl_wait();
  __shared__ double sV[kPtChunk][NT];
  __shared__ double sR[kPtThreads / 32][kPtRows][NT];
  const unsigned rb = (unsigned)((M + kPtRows - 1) / kPtRows);  // row blocks; passes are the slow grid index
  const int n0 = (int)(blockIdx.x / rb) * NT, nn = min(NT, N - n0);
  const long p0 = (long)(blockIdx.x % rb) * kPtRows;
  const int pt = threadIdx.x % kPtRows, sl = threadIdx.x / kPtRows;
  const long p = p0 + pt;
  const double* Bp = B + min(p, M - 1);
  double acc[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) acc[q] = 0.0;
  for (int k0 = 0; k0 < K; k0 += kPtChunk) {
    const int kn = min(kPtChunk, K - k0);
    __syncthreads();
    for (int e = threadIdx.x; e < NT * kPtChunk; e += kPtThreads) {
      const int k = e % kPtChunk, q = e / kPtChunk;
      if (k < kn) sV[k][q] = q < nn ? __ldcg(V + (long)(n0 + q) * K + k0 + k) : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = sl; k < kn; k += kPtSlices) {
      const double bv = __ldg(Bp + (long)(k0 + k) * M);
#pragma unroll
      for (int q = 0; q < NT; ++q) acc[q] = fma(bv, sV[k][q], acc[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < NT; ++q) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], kPtRows);
  if ((threadIdx.x & 31) < kPtRows)
#pragma unroll
    for (int q = 0; q < NT; ++q) sR[threadIdx.x >> 5][pt][q] = acc[q];
  __syncthreads();
  for (int e = threadIdx.x; e < kPtRows * NT; e += kPtThreads) {
    const int r = e % kPtRows, q = e / kPtRows;
    const long pr = p0 + r;
    if (q >= nn || pr >= M) continue;
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kPtThreads / 32; ++w) v += sR[w][r][q];
    out[(long)(n0 + q) * M + pr] = v;
  }
}

// C[n * M + c] = sum_p B[c * K + p] W[n * K + p]: one basis column per CTA, its
// threads stride over the points (contiguous in B and W).  Four basis columns per
// CTA, which share each point's data values, are slower or equal: 40,962 points,
// 2,809 columns and 8 data columns 1,664 against 1,588 us, 6,561 and 8 3,643
// against 3,653, 6,561 and 32 14,515 against 14,334.
template <int NT>
__global__ void __launch_bounds__(kPtThreads) points_analysis_kernel(int M, long K, int N, const double* __restrict__ B,
                                                                     const double* __restrict__ W,
                                                                     double* __restrict__ C) {
  pdl_wait();
  __shared__ double sR[kPtThreads / 32][NT];
  const int n0 = (int)(blockIdx.x / (unsigned)M) * NT, nn = min(NT, N - n0);
  const int c = (int)(blockIdx.x % (unsigned)M);
  const double* Bc = B + (long)c * K;
  const double* Wn[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) Wn[q] = W + (long)(n0 + min(q, nn - 1)) * K;
  double acc[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) acc[q] = 0.0;
#pragma unroll 2
  for (long p = threadIdx.x; p < K; p += kPtThreads) {
    const double b = __ldg(Bc + p);
    double w[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) w[q] = __ldcg(Wn[q] + p);
#pragma unroll
    for (int q = 0; q < NT; ++q) acc[q] = fma(b, w[q], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    double v = acc[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sR[threadIdx.x >> 5][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < nn) {
    const int q = threadIdx.x;
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kPtThreads / 32; ++w) v += sR[w][q];
    C[(long)(n0 + q) * M + c] = v;
  }
}

int points_gemm_synth(const aeolus_plan_impl* p, const double* V, double* out, int ncols, cudaStream_t st);
int points_gemm_analysis(const aeolus_plan_impl* p, const double* W, double* C, int ncols, cudaStream_t st);

}  // namespace aeolus
