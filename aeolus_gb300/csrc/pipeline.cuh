// Launch helpers that chain the three Gauss stages
//   legendre_synth<Derive>  ->  row_kernel<Pointwise>  ->  legendre_analysis<Epilogue>
// and the equivalent point-set chain (points.cu) behind one interface.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "legendre.cuh"
#include "rows.cuh"
#include "rows_fx.cuh"
#include "rows_pfa.cuh"
#include "rows_w.cuh"

namespace aeolus {

inline int pick_bc(int L, int batch) {
  const long ctas = (long)n_pairs(L) * batch;
  int bc = (int)std::max(1L, std::min(4L, ctas / 608));
  return std::min(bc, std::max(batch, 1));
}

// Raises a kernel's dynamic shared-memory limit once per (kernel, device):
// later calls -- including calls made while a stream is being captured
// into a CUDA graph -- do not touch the function attributes again.
int allow_smem_raw(const void* kern, size_t bytes);  // plan.cu

// A kernel's static shared memory counts towards both limits (48 KB without the
// attribute, 227 KB with it): sizes that leave kStaticSmemMax of room need no look
// at the kernel.
template <class K>
inline int allow_smem(K kern, size_t bytes) {
  if (bytes + kStaticSmemMax <= 48 * 1024) return AEOLUS_OK;
  if (bytes > 227 * 1024) return fail(AEOLUS_ERR_ARG, "shared-memory tile exceeds 227 KB for this size");
  return allow_smem_raw(reinterpret_cast<const void*>(kern), bytes);
}

// Launch shapes of the three Gauss stages (the autotuner's knobs are the
// plan's tune_* fields; 0 keeps the built-in heuristic).
struct LegCfg {
  int bc;          // members per CTA
  int ss;          // CTAs per (order pair, member chunk)
  int solo;        // analysis: one order per CTA
  int threads;
  size_t smem;
  dim3 grid;
};

// Warps of a CTA with `warps` warps of items: at most 8, with the fewest idle
// ones in the last round.
inline int leg_warps(int warps) {
  int best = 1, cost = warps;
  for (int w = 2; w <= 8; ++w) {
    const int c = (warps + w - 1) / w * w;
    if (c <= cost || best < 4) best = w, cost = c;
  }
  return best;
}

// CTAs that share one (order pair, member chunk) of `warps` warps of items:
// enough for six CTAs per SM, which even out the last wave (24 members at l_max
// 127 4306 us a step against 4443 with three to five, 8 members 1542 against 1517
// to 1542), and none with fewer than four warps: each repeats the derivation or the
// folding of the whole pair.  Against two warps at least: 423 -> 364 us for 4
// members at l_max 85, 533 -> 507 for 2 at 127, 563 -> 533 for 8 at 63, but 138 ->
// 142 for one at 42 and 226 -> 238 for 2 at 85; against eight: 246 -> 193 us for
// one at 85, 308 -> 341 for one at 127.
inline int leg_shares(const aeolus_plan_impl* p, long ctas, int warps) {
  const long want = (6L * p->sm_count + ctas - 1) / std::max(ctas, 1L);
  return (int)std::max(1L, std::min<long>(want, warps / 4));
}

template <class Derive>
LegCfg synth_cfg(const aeolus_plan_impl* p, int batch) {
  const int L = p->lmax;
  int bc = p->tune_bc_synth > 0 ? std::min(p->tune_bc_synth, std::max(batch, 1)) : pick_bc(L, batch);
  while (bc > 1 && synth_smem_bytes<Derive>(L, bc) > 200 * 1024) --bc;
  const int gy = (batch + bc - 1) / bc, items = p->nh * bc * Derive::NF;
  const int ss = leg_shares(p, (long)n_pairs(L) * gy, (items + 31) / 32);
  const int per = (items + ss - 1) / ss;
  return LegCfg{bc, ss, 0, 32 * leg_warps((per + 31) / 32), synth_smem_bytes<Derive>(L, bc), dim3(n_pairs(L) * ss, gy)};
}

template <class Epi>
LegCfg analysis_cfg(const aeolus_plan_impl* p, int batch) {
  const int L = p->lmax, top = EpiTop<Epi>::top(L), js = leg_row_slices(p->nh, Epi::NF);
  int bc = p->tune_bc_anal > 0 ? std::min(p->tune_bc_anal, std::max(batch, 1)) : pick_bc(top, batch);
  while (bc > 1 && analysis_smem_bytes<Epi>(L, p->nh, bc, 1, 0) > 160 * 1024) --bc;
  const int solo = analysis_smem_bytes<Epi>(L, p->nh, bc, top + 2, 0) > 227 * 1024;
  const int pairs = solo ? top + 1 : n_pairs(top);
  const int gy = (batch + bc - 1) / bc, degrees = bc * (top + 2), q = 32 / js;  // q degrees fill a warp
  const int want = leg_shares(p, (long)pairs * gy, (degrees * js + 31) / 32);
  int per = (degrees + want - 1) / want;
  per = std::max(std::min(q, degrees), per / q * q);
  int ss = (degrees + per - 1) / per;
  while (js > 1 && ss < degrees && analysis_smem_bytes<Epi>(L, p->nh, bc, ss, solo) > 220 * 1024) ++ss;  // partial sums that fit
  per = (degrees + ss - 1) / ss;
  return LegCfg{bc, ss, solo, std::max(128, 32 * leg_warps((per * js + 31) / 32)),
                analysis_smem_bytes<Epi>(L, p->nh, bc, ss, solo), dim3(pairs * ss, gy)};
}

inline LegArgs leg_args(const aeolus_plan_impl* p, const LegCfg& c, int batch, double2* FG, int nblk) {
  return LegArgs{p->lmax, p->nlat, p->nh, batch, c.bc, c.ss, c.solo, p->P, p->PT, FG, nblk};
}

inline int row_threads(const aeolus_plan_impl* p) { return p->tune_row_threads > 0 ? p->tune_row_threads : 256; }

template <class Derive>
int launch_synth(const aeolus_plan_impl* p, const Derive& d, double2* FG, int nblk, int batch,
                 cudaStream_t st) {
  const LegCfg c = synth_cfg<Derive>(p, batch);
  const LegArgs a = leg_args(p, c, batch, FG, nblk);
  auto kern = legendre_synth_kernel<Derive>;
  int s = allow_smem(kern, c.smem);
  if (s) return s;
  ProfScope prof("legendre_synth_f64", st);
  launch_pdl(kern, c.grid, dim3(c.threads), c.smem, st, a, d);
  AE_LAUNCH("legendre_synth_kernel");
  return AEOLUS_OK;
}

template <class Epi>
int launch_analysis(const aeolus_plan_impl* p, const Epi& e, double2* FG, int nblk, int batch,
                    cudaStream_t st) {
  const LegCfg c = analysis_cfg<Epi>(p, batch);
  const LegArgs a = leg_args(p, c, batch, FG, nblk);
  auto kern = legendre_analysis_kernel<Epi>;
  int s = allow_smem(kern, c.smem);
  if (s) return s;
  ProfScope prof("legendre_analysis_f64", st);
  launch_pdl(kern, c.grid, dim3(c.threads), c.smem, st, a, e);
  AE_LAUNCH("legendre_analysis_kernel");
  return AEOLUS_OK;
}

// Fills the plan-derived fields of a row stage's arguments.
inline void row_args(const aeolus_plan_impl* p, RowArgs& a) {
  a.L = p->lmax;
  a.nlat = p->nlat;
  a.fft = p->fftx;
  a.irev = p->fft_irev;
  a.coslat = p->coslat;
  a.fgrid = p->fgrid;
  a.wq = a.unit_weights ? nullptr : p->wq;
}

template <class Pw, int IN_MODE, int OUT_MODE, class FFT>
int launch_rows_fx(const aeolus_plan_impl* p, const Pw& pw, const RowArgs& a, cudaStream_t st) {
  const size_t sm = row_fx_smem_bytes<Pw>(p->fftx, p->lmax);
  auto kern = row_kernel_fx<Pw, IN_MODE, OUT_MODE, FFT>;
  int s = allow_smem(kern, sm);
  if (s) return s;
  ProfScope prof(IN_MODE == kInF ? (OUT_MODE == kOutG ? "rows_fx_c2r_products_r2c" : "rows_fx_c2r") : "rows_fx_r2c",
                 st);
  launch_pdl(kern, dim3(p->nlat, a.batch), dim3(row_threads(p)), sm, st, a, pw, static_cast<const FxW*>(p->twfx),
             static_cast<const float4*>(p->twdf), fx_consts());
  AE_LAUNCH("row_kernel_fx");
  return AEOLUS_OK;
}

// At most two row CTAs per SM: 320 threads instead of 128 shorten every phase
// of a row (each pass of 9 fields then takes one or two rounds).  Tendency
// chains only, whose rows have the most phases.  SWE RK4 per stage: 47.2 ->
// 43.9 us at one CTA per SM (l_max 85, one member), 56.8 -> 54.4 at two; from
// three on it costs (86.6 -> 90.8 us at 3.8 per SM).
template <int IN_MODE, int OUT_MODE>
inline bool split_few_rows(const aeolus_plan_impl* p, dim3 grid) {
  return IN_MODE == kInF && OUT_MODE == kOutG && (long)grid.x * grid.y <= 2L * p->sm_count;
}
template <int IN_MODE, int OUT_MODE>
constexpr int few_row_threads() { return IN_MODE == kInF && OUT_MODE == kOutG ? kFewRowThreads : kFx8Threads; }

// Fixed radix sequence (R0, 8, 8): compile-time lengths, kFx8Threads threads
// (the plan's row-thread knob does not apply).
template <class Pw, int IN_MODE, int OUT_MODE, int R0>
int launch_rows_fx8(const aeolus_plan_impl* p, const Pw& pw, const RowArgs& a, cudaStream_t st) {
  const size_t sm = row_fx8_smem_bytes<Pw>(R0);
  const dim3 grid(p->nlat, a.batch);
  const bool few = split_few_rows<IN_MODE, OUT_MODE>(p, grid);
  auto kern = few ? row_kernel_fx8<Pw, IN_MODE, OUT_MODE, R0, few_row_threads<IN_MODE, OUT_MODE>()> : row_kernel_fx8<Pw, IN_MODE, OUT_MODE, R0, kFx8Threads>;
  int s = allow_smem(kern, sm);
  if (s) return s;
  ProfScope prof(IN_MODE == kInF ? (OUT_MODE == kOutG ? "rows_fx_c2r_products_r2c" : "rows_fx_c2r") : "rows_fx_r2c",
                 st);
  launch_pdl(kern, grid, dim3(few ? kFewRowThreads : kFx8Threads), sm, st, a, pw, static_cast<const FxW*>(p->twfx),
             fx_consts());
  AE_LAUNCH("row_kernel_fx8");
  return AEOLUS_OK;
}

// nlon = 2 R0 R1 R2: prime-factor transforms (rows_pfa.cuh), kPfaThreads
// threads (the plan's row-thread knob does not apply).
template <class Pw, int IN_MODE, int OUT_MODE, class S>
int launch_rows_pfa(const aeolus_plan_impl* p, const Pw& pw, const RowArgs& a, cudaStream_t st) {
  const size_t sm = row_pfa_smem_bytes<Pw, S>();
  const dim3 grid = row_pfa_grid<Pw>(p->nlat, a.batch);
  const bool few = split_few_rows<IN_MODE, OUT_MODE>(p, grid);
  auto kern = few ? row_kernel_pfa<Pw, IN_MODE, OUT_MODE, S, few_row_threads<IN_MODE, OUT_MODE>()> : row_kernel_pfa<Pw, IN_MODE, OUT_MODE, S, kPfaThreads>;
  int s = allow_smem(kern, sm);
  if (s) return s;
  ProfScope prof(IN_MODE == kInF ? (OUT_MODE == kOutG ? "rows_fx_c2r_products_r2c" : "rows_fx_c2r") : "rows_fx_r2c",
                 st);
  launch_pdl(kern, grid, dim3(few ? kFewRowThreads : kPfaThreads), sm, st, a, pw,
             static_cast<const FxW*>(p->twfx), fx_consts());
  AE_LAUNCH("row_kernel_pfa");
  return AEOLUS_OK;
}

// Row-stage body of the split-precision path for a plan: every caller (the
// single-plan chains and the grouped ensemble kernels) picks the same one,
// so a plan's results do not depend on the route.
enum SplitRowKind {
  kRowsRuntime = 0,  // runtime radix sequence (row_fx_body)
  kRowsFx8R2,        // nlon 256: 2 x 8 x 8 Cooley-Tukey (row_fx8_body)
  kRowsPfa192,       // nlon 384: prime-factor 3 x (8 x 8)
  kRowsPfa160,       // nlon 320: 5 x (4 x 8)
  kRowsPfa96,        // nlon 192: 3 x (4 x 8)
  kRowsPfa64,        // nlon 128: 8 x 8
  kRowsPfa32,        // nlon 64: 4 x 8
};
inline int split_row_kind(const aeolus_plan_impl* p) {
  const FftInfo& f = p->fftx;
  if (Pfa192::matches(f)) return kRowsPfa192;
  if (Pfa160::matches(f)) return kRowsPfa160;
  if (Pfa96::matches(f)) return kRowsPfa96;
  if (Pfa64::matches(f)) return kRowsPfa64;
  if (Pfa32::matches(f)) return kRowsPfa32;
  if (FftFixed<2, 8, 8>::matches(f)) return kRowsFx8R2;
  return kRowsRuntime;
}
template <class Pw>
size_t split_row_smem_bytes(const aeolus_plan_impl* p) {
  switch (split_row_kind(p)) {
    case kRowsPfa192: return row_pfa_smem_bytes<Pw, Pfa192>();
    case kRowsPfa160: return row_pfa_smem_bytes<Pw, Pfa160>();
    case kRowsPfa96: return row_pfa_smem_bytes<Pw, Pfa96>();
    case kRowsPfa64: return row_pfa_smem_bytes<Pw, Pfa64>();
    case kRowsPfa32: return row_pfa_smem_bytes<Pw, Pfa32>();
    case kRowsFx8R2: return row_fx8_smem_bytes<Pw>(2);
    default: return row_fx_smem_bytes<Pw>(p->fftx, p->lmax);
  }
}

// Launch shape of the FP64 row stage (results do not depend on it).
struct WideRowCfg {
  int nr;       // member rows per CTA (FFT lengths)
  int gf;       // staged fields (direct sums)
  bool gtab;    // twiddles from global memory (rows too long for a shared table)
  int threads;
  size_t smem;
  dim3 grid;
};
template <class Pw>
WideRowCfg wide_row_cfg(const aeolus_plan_impl* p, int batch) {
  WideRowCfg c{1, 0, false, 128, 0, dim3(p->nlat, batch)};
  const FftInfo& f = p->fftx;
  if (f.use_fft) {
    constexpr int NR = w_rows_per_cta<Pw>();
    const long grouped = (long)p->nlat * ((batch + NR - 1) / NR);
    if (grouped >= 4L * p->sm_count && row_w_smem_bytes<Pw>(f, NR) <= 72 * 1024) {
      c.nr = NR;
      c.grid.y = (batch + NR - 1) / NR;
    }
    c.smem = row_w_smem_bytes<Pw>(f, c.nr);
    // few rows: twice the threads shorten each row; otherwise more CTAs per SM
    // (512 threads measured equal at one CTA per SM and 22 % slower at two)
    if ((long)c.grid.x * c.grid.y <= 2L * p->sm_count) c.threads = 256;
  } else {
    c.gf = row_w_dft_group<Pw>(f, p->lmax);
    c.gtab = row_w_dft_smem<Pw>(f, p->lmax, c.gf, false) > 220 * 1024;
    c.smem = row_w_dft_smem<Pw>(f, p->lmax, c.gf, c.gtab);
    const int items = (std::min(c.gf, Pw::NIN) + dft_fields<Pw::NIN>() - 1) / dft_fields<Pw::NIN>() * (f.N / 2 + 1);
    c.threads = 32 * leg_warps((items + 31) / 32);
  }
  if (p->tune_row_threads > 0) c.threads = std::min(p->tune_row_threads, kWideMaxThreads);
  return c;
}

template <class Pw, int IN_MODE, int OUT_MODE>
int launch_rows(const aeolus_plan_impl* p, const Pw& pw, RowArgs a, cudaStream_t st) {
  row_args(p, a);
  if (p->precision == AEOLUS_PREC_SPLIT_BF16) {
    // split-precision path: fixed-point FFTs, double-float products; every
    // row stage gets kernels compiled for the common radix sequences
    switch (split_row_kind(p)) {
      case kRowsPfa192: return launch_rows_pfa<Pw, IN_MODE, OUT_MODE, Pfa192>(p, pw, a, st);
      case kRowsPfa160: return launch_rows_pfa<Pw, IN_MODE, OUT_MODE, Pfa160>(p, pw, a, st);
      case kRowsPfa96: return launch_rows_pfa<Pw, IN_MODE, OUT_MODE, Pfa96>(p, pw, a, st);
      case kRowsPfa64: return launch_rows_pfa<Pw, IN_MODE, OUT_MODE, Pfa64>(p, pw, a, st);
      case kRowsPfa32: return launch_rows_pfa<Pw, IN_MODE, OUT_MODE, Pfa32>(p, pw, a, st);
      case kRowsFx8R2: return launch_rows_fx8<Pw, IN_MODE, OUT_MODE, 2>(p, pw, a, st);
      default: return launch_rows_fx<Pw, IN_MODE, OUT_MODE, FftRuntime>(p, pw, a, st);
    }
  }
  if constexpr (IN_MODE == kInGridDf || OUT_MODE == kOutGridDf) {
    return fail(AEOLUS_ERR_ARG, "double-float grids need a split-precision Gauss plan");
  } else {
    const WideRowCfg c = wide_row_cfg<Pw>(p, a.batch);
    const char* name = IN_MODE == kInF ? (OUT_MODE == kOutG ? "rows_c2r_products_r2c" : "rows_c2r") : "rows_r2c";
    constexpr int NR = w_rows_per_cta<Pw>();
    auto kern = c.nr == 1 ? row_kernel_w<Pw, 1, IN_MODE, OUT_MODE> : row_kernel_w<Pw, NR, IN_MODE, OUT_MODE>;
    auto kdft = c.gtab ? row_kernel_w_dft<Pw, IN_MODE, OUT_MODE, true> : row_kernel_w_dft<Pw, IN_MODE, OUT_MODE, false>;
    int s = p->fftx.use_fft ? allow_smem(kern, c.smem) : allow_smem(kdft, c.smem);
    if (s) return s;
    ProfScope prof(name, st);
    const FxW* tw = p->twfx;
    if (p->fftx.use_fft) launch_pdl(kern, c.grid, dim3(c.threads), c.smem, st, a, pw, tw, fx_consts());
    else launch_pdl(kdft, c.grid, dim3(c.threads), c.smem, st, a, pw, tw, c.gf);
    AE_LAUNCH("row_kernel_w");
    return AEOLUS_OK;
  }
}

// Bytes of the F/G block area for `nblk` fields per (member, row).
inline size_t fg_bytes(const aeolus_plan_impl* p, int nblk, int batch) {
  return (size_t)batch * p->nlat * nblk * (p->lmax + 1) * sizeof(double2);
}

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace aeolus
