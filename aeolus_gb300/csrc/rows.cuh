// Longitude stage of the Gauss transform: what its FP64 (rows_w.cuh) and
// split-precision (rows_fx.cuh, rows_pfa.cuh) bodies share.
#pragma once

#include "common.cuh"
#include "df.cuh"

namespace aeolus {

// Row inputs and outputs: order spectra, an FP64 grid, or (split-precision
// plans) a grid of double-floats, which saves the conversions on both sides
// of a double-float kernel.
enum { kInF = 0, kInGrid = 1, kInGridDf = 2 };
enum { kOutGrid = 0, kOutG = 1, kOutGridDf = 2 };

struct RowArgs {
  int L, nlat, batch;
  FftInfo fft;
  const int* irev;        // [n] digit-reversed position of index q (fixed-point in-place FFTs)
  const double* coslat;   // [nlat] clamped cos(latitude)
  const double* fgrid;    // [nlat] synthesis of the unit (1,0) mode
  const double* wq;       // [nlat] quadrature weight of a point of row j (NULL: unit weights)
  int unit_weights;       // launch_rows: leave wq NULL (adjoint of synthesis)
  // kInF: spectra F[b][j][nblk][L+1]; kOutG writes G into the same blocks,
  // or (fixed-point rows, G != NULL) into G with gblk fields per block
  double2* FG;
  int nblk;
  double2* G;
  int gblk;
  // kInGrid: grid[b * gin_b + f * gin_f + j * N + k]
  const double* gin;
  long gin_b, gin_f;
  // kOutGrid: out[b * gout_b + f * gout_f + j * N + k]
  double* gout;
  long gout_b, gout_f;
  template <int MODE>
  __device__ __forceinline__ df in_df(long i) const {  // grid value i as a double-float
    return MODE == kInGridDf ? reinterpret_cast<const df*>(gin)[i] : df_of_f64(gin[i]);
  }
  template <int MODE>
  __device__ __forceinline__ void put_df(long i, df v) const {
    if (MODE == kOutGridDf) reinterpret_cast<df*>(gout)[i] = v;
    else gout[i] = f64_of_df(v);
  }
  // grid values i (even) and i + 1 on the packed lanes
  template <int MODE>
  __device__ __forceinline__ df2 in_df2(long i) const {
    if (MODE == kInGridDf) {
      const float4 w = *reinterpret_cast<const float4*>(reinterpret_cast<const df*>(gin) + i);
      return df2{f2_pack(w.x, w.z), f2_pack(w.y, w.w)};
    }
    return df2_pack(df_of_f64(gin[i]), df_of_f64(gin[i + 1]));
  }
  template <int MODE>
  __device__ __forceinline__ void put_df2(long i, df2 v) const {
    df a, b;
    df2_unpack(v, a, b);
    if (MODE == kOutGridDf) {
      *reinterpret_cast<float4*>(reinterpret_cast<df*>(gout) + i) = make_float4(a.hi, a.lo, b.hi, b.lo);
    } else {
      gout[i] = f64_of_df(a);
      gout[i + 1] = f64_of_df(b);
    }
  }
  unsigned* status;       // optional per-member state bits
  double ir;              // 1 / R of the functor's longitude derivatives (RowSrc)
  int drop;               // kOutG: orders above L - drop are not written (EpiTop)
};

// x / d through the stage's 32-bit reciprocal (exact for x * d < 2^32).
__device__ __forceinline__ int div_rcp(int x, int d, unsigned rcp) {
  return d == 1 ? x : (int)__umulhi((unsigned)x, rcp);
}

// Identity pointwise op for plain synthesis / analysis.
struct PwCopy {
  static constexpr int NIN = 1, NOUT = 1;
  static constexpr bool kIdentity = true;
  __device__ unsigned operator()(double, double, const double* in, double* out) const {
    out[0] = in[0];
    return 0u;
  }
  __device__ RowDf df_row(double c, double) const { return RowDf{df{0.f, 0.f}, df{0.f, 0.f}, (float)c}; }
  __device__ unsigned df_op(const RowDf&, const df* in, df* out) const {
    out[0] = in[0];
    return 0u;
  }
  __device__ unsigned df_op2(const RowDf&, const df2* in, df2* out) const {  // two grid points (packed)
    out[0] = in[0];
    return 0u;
  }
};

}  // namespace aeolus
