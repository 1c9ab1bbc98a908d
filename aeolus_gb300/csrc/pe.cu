// Dry hydrostatic primitive-equation tendency in sigma coordinates,
// src/planetary_sandbox/physics/primitive_equations.py:482-753 with the
// column operators of physics/sigma_coordinate.py:164-398, batched over
// levels and members on the library's transforms:
//
//   aeolus_pe_derive    spectral: per level u cos, v cos (from the inverse
//                       Laplacians of zeta, delta), zeta, delta, T, dT/dlambda,
//                       sin(theta) dT/dtheta / R, the same two of eta = zeta + f,
//                       eta; per member the two derivatives of ln p_s
//   (synthesis of all 10 K + 2 fields on the product plan)
//   aeolus_pe_columns   pointwise, one thread per product point and member,
//                       the whole column in registers: G = delta + V.grad ln p_s,
//                       d ln p_s/dt, interface sigma_dot, omega/p, centred
//                       vertical advection of u, v, T; the thermodynamic
//                       integrand, -div(eta V), curl(eta V), kinetic energy, and
//                       the residual vector Z = sigma_dot dV/dsigma + R_d T grad ln p_s
//   (analysis of the 4 K + 1 integrands; weak-form curl/div of Z on the
//   one-degree-extended plan)
//   aeolus_pe_spectral  spectral: 2/3 cuts, Simmons-Burridge geopotential of
//                       the spectral T, -lap(KE + Phi), l = 0 rows of the
//                       momentum tendencies pinned.
//
// These calls are the C ABI's pieces and the yardstick of the chain's tests; the
// package runs the whole tendency as one chain (aeolus_pe_tendency, below).
#include <type_traits>

#include "models.cuh"

namespace aeolus {
namespace {

constexpr int kPeMaxLevels = 64;
constexpr int kPeLevelFields = 10;  // U, V, zeta, delta, T, T_lam, T_snt, eta_lam, eta_snt, eta
constexpr int kPeOutFields = 4;     // thermodynamic integrand, -div(eta V), curl(eta V), KE

// Lorenz sigma grid, sigma_coordinate.py:43-149: interfaces s[0] = 0 (top)
// .. s[K] = 1 (surface), thickness, interface log ratios beta (beta[0], the
// infinite top entry, is never read) and the Simmons-Burridge alpha.
// The column kernel multiplies by host-computed reciprocals instead of
// dividing (FP64 divides would dominate its FP64 pipe): h2[k] = 1/(2 Dsigma_k)
// and bd[k] = beta_k / Dsigma_k, within an ulp of the reference's quotients.
struct PeSigma {
  int K;
  double s[kPeMaxLevels + 1], dsig[kPeMaxLevels], beta[kPeMaxLevels], alpha[kPeMaxLevels];
  double h2[kPeMaxLevels], bd[kPeMaxLevels];
};

int make_sigma(const double* interfaces, int nlev, PeSigma* g) {
  if (nlev < 1 || nlev > kPeMaxLevels)
    return fail(AEOLUS_ERR_ARG, "nlev must be in [1, " + std::to_string(kPeMaxLevels) + "], got " +
                                    std::to_string(nlev));
  if (!interfaces) return fail(AEOLUS_ERR_ARG, "NULL sigma interfaces");
  if (interfaces[0] != 0.0 || interfaces[nlev] != 1.0)
    return fail(AEOLUS_ERR_ARG, "sigma interfaces must start at exactly 0.0 and end at exactly 1.0");
  g->K = nlev;
  for (int k = 0; k <= nlev; ++k) {
    if (!std::isfinite(interfaces[k]) || (k > 0 && !(interfaces[k] > interfaces[k - 1])))
      return fail(AEOLUS_ERR_ARG, "sigma interfaces must be finite and strictly increasing");
    g->s[k] = interfaces[k];
  }
  for (int k = 0; k < nlev; ++k) {
    g->dsig[k] = g->s[k + 1] - g->s[k];
    g->h2[k] = 1.0 / (2.0 * g->dsig[k]);
  }
  g->beta[0] = 0.0;
  g->bd[0] = 0.0;
  g->alpha[0] = std::log(2.0);
  for (int k = 1; k < nlev; ++k) {
    g->beta[k] = std::log(g->s[k + 1] / g->s[k]);
    g->alpha[k] = 1.0 - (g->s[k] / g->dsig[k]) * g->beta[k];
    g->bd[k] = g->beta[k] / g->dsig[k];
  }
  return AEOLUS_OK;
}

int pe_check(const aeolus_pe_params* prm) {
  if (!prm) return fail(AEOLUS_ERR_ARG, "NULL primitive-equation parameters");
  if (!(std::isfinite(prm->radius) && prm->radius > 0) || !std::isfinite(prm->omega))
    return fail(AEOLUS_ERR_ARG, "primitive equations: bad radius/omega");
  if (!(std::isfinite(prm->r_dry) && prm->r_dry > 0))
    return fail(AEOLUS_ERR_ARG, "r_dry must be finite and > 0, got " + std::to_string(prm->r_dry));
  if (!(std::isfinite(prm->cp_dry) && prm->cp_dry > prm->r_dry))
    return fail(AEOLUS_ERR_ARG, "cp_dry must be finite and > r_dry, got " + std::to_string(prm->cp_dry));
  return AEOLUS_OK;
}

// One thread per (member, l, m): every level's derived spectra.
__global__ void pe_derive_kernel(Spec s, int K, int batch, double f10, const double2* __restrict__ st,
                                 double2* __restrict__ out) {
  const int L = s.L;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n2 * batch) return;
  const int b = (int)(idx / n2);
  const long r = idx - b * n2;
  const int l = (int)(r / (L + 1)), m = (int)(r - (long)l * (L + 1));
  const double2* S = st + (long)b * (3 * K + 1) * n2;
  double2* O = out + (long)b * (kPeLevelFields * K + 2) * n2 + r;
  const double2 zero = make_double2(0.0, 0.0);
  if (m > l) {
    for (int f = 0; f < kPeLevelFields * K + 2; ++f) O[f * n2] = zero;
    return;
  }
  const bool lo = l >= 1 && l - 1 >= m, hi = l + 1 <= L;
  auto val = [&](const double2* a, int ll) { return a[(long)ll * (L + 1) + m]; };
  auto inv = [&](const double2* a, int ll) { return s.invlap0(a, ll, m); };
  auto snt_r = [&](double2 vlo, double2 vhi) { return cscale(s.ir, s.snt(vlo, vhi, l, m)); };
  for (int k = 0; k < K; ++k) {
    const double2* z = S + (long)k * n2;
    const double2* d = S + (long)(K + k) * n2;
    const double2* T = S + (long)(2 * K + k) * n2;
    const double2 psi = inv(z, l), chi = inv(d, l);
    const double2 psi_lo = lo ? inv(z, l - 1) : zero, psi_hi = hi ? inv(z, l + 1) : zero;
    const double2 chi_lo = lo ? inv(d, l - 1) : zero, chi_hi = hi ? inv(d, l + 1) : zero;
    double2 e = val(z, l), e_lo = lo ? val(z, l - 1) : zero, e_hi = hi ? val(z, l + 1) : zero;
    if (m == 0) {  // eta = zeta + f, f = 2 Omega sin(lat): the (1, 0) mode
      if (l == 1) e.x += f10;
      if (l - 1 == 1) e_lo.x += f10;
      if (l + 1 == 1) e_hi.x += f10;
    }
    const double2 Tl = val(T, l);
    double2* o = O + (long)kPeLevelFields * k * n2;
    o[0 * n2] = cadd(snt_r(psi_lo, psi_hi), s.dlam(chi, m));   // u cos
    o[1 * n2] = csub(s.dlam(psi, m), snt_r(chi_lo, chi_hi));   // v cos
    o[2 * n2] = val(z, l);
    o[3 * n2] = val(d, l);
    o[4 * n2] = Tl;
    o[5 * n2] = s.dlam(Tl, m);
    o[6 * n2] = snt_r(lo ? val(T, l - 1) : zero, hi ? val(T, l + 1) : zero);
    o[7 * n2] = s.dlam(e, m);
    o[8 * n2] = snt_r(e_lo, e_hi);
    o[9 * n2] = e;
  }
  const double2* q = S + (long)3 * K * n2;
  O[(long)kPeLevelFields * K * n2] = s.dlam(val(q, l), m);
  O[((long)kPeLevelFields * K + 1) * n2] = snt_r(lo ? val(q, l - 1) : zero, hi ? val(q, l + 1) : zero);
}

// The same spectra for split-precision plans (their synthesis digits carry
// 48 bits) in packed double-float (lanes re, im): the coefficient products
// of the double-float derive table at the plan radius (Spec::dcoef_df: the
// same combinations of C+-, 1/lap and m/R as the SWE derive), the state
// converted by integer operations on its bits, each derived spectrum
// rounded to FP64 by one FP64 addition per word; zeta, delta, T and eta are
// copied in FP64 as they are.
__global__ void __launch_bounds__(128) pe_derive_df_kernel(Spec s, int K, int batch, double f10,
                                                           const double2* __restrict__ st, double2* __restrict__ out) {
  // one thread per (member, level, l, m); "level" K is the pair of ln p_s
  // spectra (the levels are independent, so the loads of all of them fly
  // at once instead of one level after another)
  const int L = s.L;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n2 * (K + 1) * batch) return;
  const long r = idx % n2;
  const int k = (int)((idx / n2) % (K + 1)), b = (int)(idx / (n2 * (K + 1)));
  const int l = (int)(r / (L + 1)), m = (int)(r - (long)l * (L + 1));
  const double2* S = st + (long)b * (3 * K + 1) * n2;
  double2* O = out + (long)b * (kPeLevelFields * K + 2) * n2 + r;
  const int nout = k < K ? kPeLevelFields : 2;
  double2* o = O + (long)kPeLevelFields * k * n2;  // level k's fields, or the two ln p_s ones at k = K
  if (m > l) {
    const double2 zero = make_double2(0.0, 0.0);
    for (int f = 0; f < nout; ++f) o[f * n2] = zero;
    return;
  }
  const bool lo = l >= 1 && l - 1 >= m, hi = l + 1 <= L;
  const float2* c = s.dcoef_df + r * 8;
  auto kc = [&](int i) { return df2_splat(df{c[i].x, c[i].y}); };
  const df2 zero = df2{0ull, 0ull};
  auto cv = [&](const double2* a, int ll) { return df2_of_f64x2(a[(long)ll * (L + 1) + m]); };
  auto cvlo = [&](const double2* a) { return lo ? cv(a, l - 1) : zero; };
  auto cvhi = [&](const double2* a) { return hi ? cv(a, l + 1) : zero; };
  const df2 B1 = kc(3), B2 = kc(4), B3 = kc(5);
  if (k == K) {
    const double2* q = S + (long)3 * K * n2;
    o[0] = f64x2_of_df2(df2_mul(B3, df2_times_i(cv(q, l))));
    o[n2] = f64x2_of_df2(df2_add_fast(df2_mul(B1, cvlo(q)), df2_mul(B2, cvhi(q))));
    return;
  }
  const df2 A1 = kc(0), A2 = kc(1), A3 = kc(2);
  // eta = zeta + f at the (1, 0) mode, in the neighbour slots
  auto add_f = [&](df2 v, bool at) {
    if (!at) return v;
    df re, im;
    df2_unpack(v, re, im);
    return df2_pack(df_add(re, df_of_f64(f10)), im);
  };
  const double2* z = S + (long)k * n2;
  const double2* d = S + (long)(K + k) * n2;
  const double2* T = S + (long)(2 * K + k) * n2;
  const double2 z64 = z[r], d64 = d[r], T64 = T[r];
  const df2 zl = df2_of_f64x2(z64), dl = df2_of_f64x2(d64), Tl = df2_of_f64x2(T64);
  const df2 z_lo = cvlo(z), z_hi = cvhi(z), d_lo = cvlo(d), d_hi = cvhi(d);
  o[0 * n2] = f64x2_of_df2(df2_add_fast(df2_add_fast(df2_mul(A1, z_lo), df2_mul(A2, z_hi)),
                                        df2_mul(A3, df2_times_i(dl))));    // u cos
  o[1 * n2] = f64x2_of_df2(df2_sub_fast(df2_mul(A3, df2_times_i(zl)),
                                        df2_add_fast(df2_mul(A1, d_lo), df2_mul(A2, d_hi))));  // v cos
  o[2 * n2] = z64;
  o[3 * n2] = d64;
  o[4 * n2] = T64;
  o[5 * n2] = f64x2_of_df2(df2_mul(B3, df2_times_i(Tl)));
  o[6 * n2] = f64x2_of_df2(df2_add_fast(df2_mul(B1, cvlo(T)), df2_mul(B2, cvhi(T))));
  o[7 * n2] = f64x2_of_df2(df2_mul(B3, df2_times_i(zl)));  // m = 0 (the only f slot) has B3 = 0
  o[8 * n2] = f64x2_of_df2(df2_add_fast(df2_mul(B1, add_f(z_lo, m == 0 && l == 2)),
                                        df2_mul(B2, add_f(z_hi, m == 0 && l == 0))));
  o[9 * n2] = (m == 0 && l == 1) ? make_double2(z64.x + f10, z64.y) : z64;
}

// One thread per (member, product point): the column in thread-local
// arrays.  The kernel is FP64-bound (84 % FP64-pipe active at 192x384,
// 20 levels); the arrays spill through L1 to L2, which doubles its DRAM
// traffic but not its time: a shared-memory column (occupancy-capped) and a
// two-pass form without arrays (recomputing the FP64 terms) both ran slower.
__global__ void __launch_bounds__(128) pe_columns_kernel(PeSigma sg, long np, int nlon, const double* __restrict__ coslat,
                                                         int batch, double r_dry, double kappa,
                                                         const double* __restrict__ grid, double* __restrict__ prod,
                                                         double* __restrict__ fen) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= np * batch) return;
  const int K = sg.K;
  const int b = (int)(idx / np);
  const long p = idx - b * np;
  const double ic = 1.0 / coslat[nlon > 0 ? p / nlon : p];
  const double* Gd = grid + (long)b * (kPeLevelFields * K + 2) * np + p;
  double* P = prod + (long)b * (kPeOutFields * K + 1) * np + p;
  const double lp_lam = Gd[(long)kPeLevelFields * K * np], lp_snt = Gd[((long)kPeLevelFields * K + 1) * np];
  double u[kPeMaxLevels], v[kPeMaxLevels], T[kPeMaxLevels], G[kPeMaxLevels], A[kPeMaxLevels];
  double part[kPeMaxLevels], sd[kPeMaxLevels + 1];
  double acc = 0.0, total = 0.0;
  for (int k = 0; k < K; ++k) {
    const double* f = Gd + (long)kPeLevelFields * k * np;
    u[k] = f[0] * ic;
    v[k] = f[np] * ic;
    T[k] = f[4 * np];
    A[k] = (u[k] * lp_lam - v[k] * lp_snt) * ic;      // V . grad(ln p_s)
    G[k] = f[3 * np] + A[k];                          // delta + A
    const double w = sg.dsig[k] * G[k];
    acc = k == 0 ? w : acc + w;                       // cumulative thickness-weighted G
    part[k] = acc;
  }
  total = part[K - 1];
  // interface sigma_dot: exact zeros at the top and (total - total) at the surface
  sd[0] = 0.0;
  for (int k = 1; k < K; ++k) sd[k] = sg.s[k] * total - part[k - 1];
  sd[K] = total - total;
  P[(long)kPeOutFields * K * np] = -total;            // d ln p_s / dt
  const double gu = lp_lam * ic, gv = -lp_snt * ic;   // grad(ln p_s)
  auto vadv = [&](const double* X, int k) {
    double a = 0.0;
    bool any = false;
    if (k < K - 1) {
      a = sd[k + 1] * (X[k + 1] - X[k]);
      any = true;
    }
    if (k > 0) {
      const double up = sd[k] * (X[k] - X[k - 1]);
      a = any ? a + up : up;
      any = true;
    }
    return any ? a * sg.h2[k] : 0.0;
  };
  for (int k = 0; k < K; ++k) {
    const double* f = Gd + (long)kPeLevelFields * k * np;
    const double wp = k == 0 ? A[0] - sg.alpha[0] * G[0]
                             : A[k] - sg.bd[k] * part[k - 1] - sg.alpha[k] * G[k];
    const double t_lam = f[5 * np], t_snt = f[6 * np];
    const double e_lam = f[7 * np], e_snt = f[8 * np], eta = f[9 * np];
    const double adv_t = (u[k] * t_lam - v[k] * t_snt) * ic;
    double* o = P + (long)kPeOutFields * k * np;
    o[0] = -adv_t - vadv(T, k) + kappa * T[k] * wp;
    o[np] = -((u[k] * e_lam - v[k] * e_snt) * ic + eta * f[3 * np]);
    o[2 * np] = eta * f[2 * np] + (v[k] * e_lam + u[k] * e_snt) * ic;
    o[3 * np] = 0.5 * (u[k] * u[k] + v[k] * v[k]);
    const double rt = r_dry * T[k];
    double* z = fen + ((long)b * K + k) * 2 * np + p;
    z[0] = vadv(u, k) + rt * gu;
    z[np] = vadv(v, k) + rt * gv;
  }
}

// ---------------------------------------------------------------------------
// The same column in double-float arithmetic, for split-precision plans (the
// rest of their tendency is computed to ~48 bits already): the FP64 grid
// values become double-floats through integer operations on their bits
// (df_of_f64) and the results FP64 with one FP64 addition each (f64_of_df),
// the only FP64 instructions of the kernel (GB300's FP64 pipe is ~1/64 of
// its f32 pipe).  Values below 2^-126 in magnitude are taken as 0, values
// beyond the float range as infinite.
struct PeSigmaDf {
  int K;
  df s[kPeMaxLevels + 1], dsig[kPeMaxLevels], alpha[kPeMaxLevels], h2[kPeMaxLevels], bd[kPeMaxLevels];
};

inline df host_df(double x) {
  const float h = static_cast<float>(x);
  return df{h, static_cast<float>(x - static_cast<double>(h))};
}

PeSigmaDf sigma_df(const PeSigma& g) {
  PeSigmaDf d;
  d.K = g.K;
  for (int k = 0; k <= g.K; ++k) d.s[k] = host_df(g.s[k]);
  for (int k = 0; k < g.K; ++k) {
    d.dsig[k] = host_df(g.dsig[k]);
    d.alpha[k] = host_df(g.alpha[k]);
    d.h2[k] = host_df(g.h2[k]);
    d.bd[k] = host_df(g.bd[k]);
  }
  return d;
}

// 1 / c as a double-float: f32 reciprocal refined by one double-float Newton step.
__device__ __forceinline__ df df_recip(df c) {
  const float r0 = 1.0f / c.hi;
  const df e = df_sub(df{1.0f, 0.0f}, df_mul(c, df{r0, 0.0f}));  // 1 - c r0
  return df_add(df{r0, 0.0f}, df_mul(df{r0, 0.0f}, e));
}

// Two passes over the levels and no per-level arrays (in double-float the
// recomputation is cheap, while thread-local column arrays would make the
// kernel wait on local memory): pass 1 forms the cumulative thickness-weighted
// G for the surface value; pass 2 repeats the same running sum for the
// interface sigma_dot and keeps a three-level window of u, v, T for the
// vertical advection (the same operations in the same order as one pass
// with arrays).
__global__ void __launch_bounds__(128) pe_columns_df_kernel(PeSigmaDf sg, long np, int nlon,
                                                            const double* __restrict__ coslat, int batch, df r_dry,
                                                            df kappa, const double* __restrict__ grid,
                                                            double* __restrict__ prod, double* __restrict__ fen) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= np * batch) return;
  const int K = sg.K;
  const int b = (int)(idx / np);
  const long p = idx - b * np;
  const df ic = df_recip(df_of_f64(coslat[nlon > 0 ? p / nlon : p]));
  const double* Gd = grid + (long)b * (kPeLevelFields * K + 2) * np + p;
  double* P = prod + (long)b * (kPeOutFields * K + 1) * np + p;
  const df lp_lam = df_of_f64(Gd[(long)kPeLevelFields * K * np]), lp_snt = df_of_f64(Gd[((long)kPeLevelFields * K + 1) * np]);
  auto lev = [&](int k) { return Gd + (long)kPeLevelFields * k * np; };
  auto AG = [&](int k, df uk, df vk, df& A, df& G) {
    A = df_mul(df_sub(df_mul(uk, lp_lam), df_mul(vk, lp_snt)), ic);  // V . grad(ln p_s)
    G = df_add(df_of_f64(lev(k)[3 * np]), A);                        // delta + A
  };
  // pass 1: the cumulative thickness-weighted G
  df acc = df{0.f, 0.f};
  for (int k = 0; k < K; ++k) {
    const double* f = lev(k);
    df A, G;
    AG(k, df_mul(df_of_f64(f[0]), ic), df_mul(df_of_f64(f[np]), ic), A, G);
    const df w = df_mul(sg.dsig[k], G);
    acc = k == 0 ? w : df_add(acc, w);
  }
  const df total = acc;
  P[(long)kPeOutFields * K * np] = f64_of_df(df_neg(total));  // d ln p_s / dt
  const df gu = df_mul(lp_lam, ic), gv = df_neg(df_mul(lp_snt, ic));
  const df zero = df{0.f, 0.f};
  // vertical advection of X at level k from (X[k-1], X[k], X[k+1]) with the
  // interface sigma_dot above (sdk) and below (sdk1) the level
  auto vadv = [&](df xm, df x0, df xp, int k, df sdk, df sdk1) {
    df a = zero;
    bool any = false;
    if (k < K - 1) {
      a = df_mul(sdk1, df_sub(xp, x0));
      any = true;
    }
    if (k > 0) {
      const df up = df_mul(sdk, df_sub(x0, xm));
      a = any ? df_add(a, up) : up;
      any = true;
    }
    return any ? df_mul(a, sg.h2[k]) : zero;
  };
  // pass 2
  df um = zero, vm = zero, Tm = zero;
  df u0 = df_mul(df_of_f64(lev(0)[0]), ic), v0 = df_mul(df_of_f64(lev(0)[np]), ic), T0 = df_of_f64(lev(0)[4 * np]);
  df run = zero, part_prev = zero;
  for (int k = 0; k < K; ++k) {
    const double* f = lev(k);
    df up = zero, vp = zero, Tp = zero;
    if (k + 1 < K) {
      const double* g = lev(k + 1);
      up = df_mul(df_of_f64(g[0]), ic);
      vp = df_mul(df_of_f64(g[np]), ic);
      Tp = df_of_f64(g[4 * np]);
    }
    df A, G;
    AG(k, u0, v0, A, G);
    const df w = df_mul(sg.dsig[k], G);
    run = k == 0 ? w : df_add(run, w);
    // interface sigma_dot: exact zeros at the top and (total - total) at the surface
    const df sdk = k == 0 ? zero : df_sub(df_mul(sg.s[k], total), part_prev);
    const df sdk1 = k + 1 == K ? zero : df_sub(df_mul(sg.s[k + 1], total), run);
    const df wp = k == 0 ? df_sub(A, df_mul(sg.alpha[0], G))
                         : df_sub(df_sub(A, df_mul(sg.bd[k], part_prev)), df_mul(sg.alpha[k], G));
    const df t_lam = df_of_f64(f[5 * np]), t_snt = df_of_f64(f[6 * np]);
    const df e_lam = df_of_f64(f[7 * np]), e_snt = df_of_f64(f[8 * np]), eta = df_of_f64(f[9 * np]);
    const df adv_t = df_mul(df_sub(df_mul(u0, t_lam), df_mul(v0, t_snt)), ic);
    double* o = P + (long)kPeOutFields * k * np;
    o[0] = f64_of_df(df_add(df_sub(df_neg(adv_t), vadv(Tm, T0, Tp, k, sdk, sdk1)), df_mul(df_mul(kappa, T0), wp)));
    o[np] = f64_of_df(df_neg(df_add(df_mul(df_sub(df_mul(u0, e_lam), df_mul(v0, e_snt)), ic),
                                    df_mul(eta, df_of_f64(f[3 * np])))));
    o[2 * np] = f64_of_df(df_add(df_mul(eta, df_of_f64(f[2 * np])),
                                 df_mul(df_add(df_mul(v0, e_lam), df_mul(u0, e_snt)), ic)));
    o[3 * np] = f64_of_df(df_scale2(df_add(df_mul(u0, u0), df_mul(v0, v0)), 0.5f));
    const df rt = df_mul(r_dry, T0);
    double* z = fen + ((long)b * K + k) * 2 * np + p;
    z[0] = f64_of_df(df_add(vadv(um, u0, up, k, sdk, sdk1), df_mul(rt, gu)));
    z[np] = f64_of_df(df_add(vadv(vm, v0, vp, k, sdk, sdk1), df_mul(rt, gv)));
    part_prev = run;
    um = u0;
    vm = v0;
    Tm = T0;
    u0 = up;
    v0 = vp;
    T0 = Tp;
  }
}

// One thread per (member, l, m): every level's tendencies.
__global__ void pe_spectral_kernel(PeSigma sg, int L, double R, double r_dry, int batch,
                                   const double2* __restrict__ st, const double2* __restrict__ an,
                                   const double2* __restrict__ cz, const double2* __restrict__ dz,
                                   const double2* __restrict__ phis, double2* __restrict__ out) {
  const int K = sg.K;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n2 * batch) return;
  const int b = (int)(idx / n2);
  const long r = idx - b * n2;
  const int l = (int)(r / (L + 1)), m = (int)(r - (long)l * (L + 1));
  double2* O = out + (long)b * (3 * K + 1) * n2 + r;
  const double2 zero = make_double2(0.0, 0.0);
  if (m > l) {
    for (int f = 0; f < 3 * K + 1; ++f) O[f * n2] = zero;
    return;
  }
  const int cut = (2 * L) / 3;
  const bool keep = l <= cut && m <= cut;
  const double lap = -(double)l * (l + 1.0) / (R * R);
  const double2* A = an + (long)b * (kPeOutFields * K + 1) * n2 + r;
  const double2* T = st + (long)b * (3 * K + 1) * n2 + (long)2 * K * n2 + r;
  // Simmons-Burridge on the spectral T, upward from Phi_s at the surface
  double2 below = phis[r];
  for (int k = K - 1; k >= 0; --k) {
    const double2 Tk = T[(long)k * n2];
    const double2 phi = cadd(below, cscale(r_dry * sg.alpha[k], Tk));
    if (k > 0) below = cadd(below, cscale(r_dry * sg.beta[k], Tk));
    const double2* a = A + (long)kPeOutFields * k * n2;
    const long zk = ((long)b * K + k) * n2 + r;
    const double2 ke = keep ? a[3 * n2] : zero;
    O[(long)(2 * K + k) * n2] = keep ? a[0] : zero;
    O[(long)k * n2] = (l == 0 || !keep) ? zero : csub(a[n2], cz[zk]);
    const double2 dd = keep ? csub(a[2 * n2], dz[zk]) : zero;
    O[(long)(K + k) * n2] = l == 0 ? zero : csub(dd, cscale(lap, cadd(ke, phi)));
  }
  O[(long)3 * K * n2] = keep ? A[(long)kPeOutFields * K * n2] : zero;
}

// --------------------------------------------------------------------------
// The whole tendency as one chain (aeolus_pe_tendency, aeolus_pe_rk4): the
// spectra of a member's K levels and ln p_s go through the transforms as
// K + 1 "levels" of the batch,
//   synthesis of 7 contracted fields per level (U, V, zeta, delta, T and the
//   latitude derivatives of T and eta; the longitude derivatives are formed
//   from the T and zeta order spectra, and eta = zeta + f on the grid),
//   column physics, analysis of 6 fields per level (the four integrands and
//   Z / cos, whose curl and divergence below the 2/3 cut read one degree
//   more than the cut, not one more than l_max), spectral kernel.
// Level K carries ln p_s in the T slot (its other fields are zero) and
// d ln p_s / dt in the first integrand.  Against the composition of the single
// calls (10 K + 2 fields synthesised, 6 K + 1 analysed to l_max + 1, FP64 grids
// between the kernels, 14 launches through Python): one FP64 RK4 step at 64 x
// 128, l_max 42, 8 levels 1.45 -> 0.27 ms; the split tendency of 4 members at
// 192 x 384, l_max 127, 20 levels 2.13 -> 1.26 ms (columns 376 -> 265 us, bound
// by instruction issue; 110 us of it are the DRAM bytes).
constexpr int kPeGrid = 9;  // U, V, zeta, delta, T, T_lam, T_snt, eta_lam, eta_snt
constexpr int kPeProd = 6;  // the four integrands of kPeOutFields, Z_east / cos, Z_north / cos

struct PeDerive7;
struct PeDerive {  // every grid field (point-set plans)
  static constexpr int NF = kPeGrid;
  using Contracted = PeDerive7;
  Spec s;
  const double2* state;
  int K;
  double f10;
  struct Level {
    const double2 *z, *d, *T;  // null: the level of ln p_s
  };
  __device__ Level level(int bk) const {
    const long n2 = (long)(s.L + 1) * (s.L + 1);
    const int b = bk / (K + 1), k = bk - b * (K + 1);
    const double2* S = state + (long)b * (3 * K + 1) * n2;
    if (k == K) return Level{nullptr, nullptr, S + 3 * K * n2};
    return Level{S + k * n2, S + (K + k) * n2, S + (2 * K + k) * n2};
  }
  __device__ void column(int bk, int l, int m, double2* v) const {
    const Level f = level(bk);
    const int L = s.L;
    const long r = (long)l * (L + 1) + m;
    const bool lo = l >= 1 && l - 1 >= m, hi = l + 1 <= L;
    const double2 zero = make_double2(0.0, 0.0);
    // 1/R C+_{l-1} / lap, 1/R C-_{l+1} / lap, m/R / lap, then the same without 1 / lap
    double A1, A2, A3, B1, B2, B3;
    if (s.dcoef) {
      const double* c = s.dcoef + r * 8;
      A1 = c[0], A2 = c[1], A3 = c[2], B1 = c[3], B2 = c[4], B3 = c[5];
    } else {
      auto il = [&](int ll) { return ll <= 0 ? 0.0 : (s.invlap ? s.invlap[ll] : 1.0 / s.lap(ll)); };
      B1 = lo ? s.ir * s.cplus[r - (L + 1)] : 0.0;
      B2 = hi ? s.ir * s.cminus[r + (L + 1)] : 0.0;
      B3 = (double)m * s.ir;
      A1 = lo ? B1 * il(l - 1) : 0.0;
      A2 = hi ? B2 * il(l + 1) : 0.0;
      A3 = B3 * il(l);
    }
    auto at = [&](const double2* a, int off) { return a[r + off * (L + 1)]; };
    const double2 Tl = f.T[r], T_lo = lo ? at(f.T, -1) : zero, T_hi = hi ? at(f.T, 1) : zero;
    v[4] = Tl;
    v[5] = make_double2(-B3 * Tl.y, B3 * Tl.x);
    v[6] = make_double2(fma(B1, T_lo.x, B2 * T_hi.x), fma(B1, T_lo.y, B2 * T_hi.y));
    if (!f.z) {
      v[0] = v[1] = v[2] = v[3] = v[4] = v[7] = v[8] = zero;
      v[4] = Tl;
      return;
    }
    const double2 zl = f.z[r], dl = f.d[r];
    double2 z_lo = lo ? at(f.z, -1) : zero, z_hi = hi ? at(f.z, 1) : zero;
    const double2 d_lo = lo ? at(f.d, -1) : zero, d_hi = hi ? at(f.d, 1) : zero;
    v[0] = make_double2(fma(A1, z_lo.x, fma(A2, z_hi.x, -A3 * dl.y)), fma(A1, z_lo.y, fma(A2, z_hi.y, A3 * dl.x)));
    v[1] = make_double2(-fma(A1, d_lo.x, fma(A2, d_hi.x, A3 * zl.y)), fma(A3, zl.x, -fma(A1, d_lo.y, A2 * d_hi.y)));
    v[2] = zl;
    v[3] = dl;
    v[7] = make_double2(-B3 * zl.y, B3 * zl.x);  // f has m = 0: no longitude derivative
    if (m == 0) {                                // planetary vorticity of the (1, 0) mode in eta
      if (l - 1 == 1) z_lo.x += f10;
      if (l + 1 == 1) z_hi.x += f10;
    }
    v[8] = make_double2(fma(B1, z_lo.x, B2 * z_hi.x), fma(B1, z_lo.y, B2 * z_hi.y));
  }
};

struct PeDerive7 {  // the contracted fields of a Gauss plan
  static constexpr int NF = 7;
  static constexpr bool kColumnDf = true;
  static constexpr int NBLK = kPeGrid;
  __host__ __device__ static constexpr int blk(int f) { return f < 5 ? f : f == 5 ? 6 : 8; }
  __host__ __device__ static constexpr int lam_blk(int f) { return f == 4 ? 5 : f == 2 ? 7 : -1; }
  PeDerive d9;
  double lam_ir() const { return d9.s.ir; }
  __device__ void column(int bk, int l, int m, double2* v) const {
    double2 w[kPeGrid];
    d9.column(bk, l, m, w);
#pragma unroll
    for (int f = 0; f < 5; ++f) v[f] = w[f];
    v[5] = w[6];
    v[6] = w[8];
  }
  // The same fields in double-float (lanes re, im), as SweDerive7::column_df.
  __device__ void column_df(int bk, int l, int m, df2* v) const {
    const Spec& s = d9.s;
    if (!s.dcoef_df) {
      double2 w[NF];
      column(bk, l, m, w);
#pragma unroll
      for (int f = 0; f < NF; ++f) v[f] = df2_of_f64x2(w[f]);
      return;
    }
    const PeDerive::Level f = d9.level(bk);
    const int L = s.L;
    const long r = (long)l * (L + 1) + m;
    const float2* c = s.dcoef_df + r * 8;
    auto k = [&](int i) { return df2_splat(df{c[i].x, c[i].y}); };
    const bool lo = l >= 1 && l - 1 >= m, hi = l + 1 <= L;
    const df2 zero = df2{0ull, 0ull};
    auto at = [&](const double2* a, int off, bool in) { return in ? df2_of_f64x2(a[r + off * (L + 1)]) : zero; };
    const df2 B1 = k(3), B2 = k(4);
    v[4] = at(f.T, 0, true);
    v[5] = df2_add_fast(df2_mul(B1, at(f.T, -1, lo)), df2_mul(B2, at(f.T, 1, hi)));
    if (!f.z) {
      v[0] = v[1] = v[2] = v[3] = v[6] = zero;
      return;
    }
    const df2 zl = at(f.z, 0, true), dl = at(f.d, 0, true), d_lo = at(f.d, -1, lo), d_hi = at(f.d, 1, hi);
    df2 z_lo = at(f.z, -1, lo), z_hi = at(f.z, 1, hi);
    const df2 A1 = k(0), A2 = k(1), A3 = k(2);
    v[0] = df2_add_fast(df2_add_fast(df2_mul(A1, z_lo), df2_mul(A2, z_hi)), df2_mul(A3, df2_times_i(dl)));
    v[1] = df2_sub_fast(df2_mul(A3, df2_times_i(zl)), df2_add_fast(df2_mul(A1, d_lo), df2_mul(A2, d_hi)));
    v[2] = zl;
    v[3] = dl;
    if (m == 0 && (l == 2 || l == 0)) {  // planetary vorticity of the (1, 0) mode in eta
      df re, im;
      df2_unpack(l == 2 ? z_lo : z_hi, re, im);
      re = df_add(re, df_of_f64(d9.f10));
      (l == 2 ? z_lo : z_hi) = df2_pack(re, im);
    }
    v[6] = df2_add_fast(df2_mul(B1, z_lo), df2_mul(B2, z_hi));
  }
};

// Identity of N fields.
template <int N>
struct PwCopyN {
  static constexpr int NIN = N, NOUT = N;
  static constexpr bool kIdentity = true;
  __device__ unsigned operator()(double, double, const double* in, double* out) const {
#pragma unroll
    for (int f = 0; f < N; ++f) out[f] = in[f];
    return 0u;
  }
  __device__ RowDf df_row(double c, double) const { return RowDf{df{0.f, 0.f}, df{0.f, 0.f}, (float)c}; }
  __device__ unsigned df_op(const RowDf&, const df* in, df* out) const {
#pragma unroll
    for (int f = 0; f < N; ++f) out[f] = in[f];
    return 0u;
  }
  __device__ unsigned df_op2(const RowDf&, const df2* in, df2* out) const {
#pragma unroll
    for (int f = 0; f < N; ++f) out[f] = in[f];
    return 0u;
  }
};
struct PePw : PwCopyN<kPeGrid> {  // grid fields; FP64 Gauss plans: T_lam, eta_lam from T, zeta (RowSrc)
  static constexpr int NBLK64 = 7;
  __device__ static constexpr int src64(int f) {
    constexpr int b[kPeGrid] = {0, 1, 2, 3, 4, 4, 5, 2, 6};
    return b[f];
  }
  __device__ static constexpr bool lam64(int f) { return f == 5 || f == 7; }
};

// Analysed fields of a level, [bk][kPeProd][L+1][L+1]: only the triangle the
// spectral kernel reads is written.
struct PeEpi {
  static constexpr int NF = kPeProd;
  static constexpr bool kCutPlus = true;
  double2* out;
  int L;
  __device__ void finish_field(int bk, int f, int l, int m, double2 a) const {
    if (l <= EpiTop<PeEpi>::top(L)) out[(((long)bk * NF + f) * (L + 1) + l) * (L + 1) + m] = a;
  }
  __device__ void finish(int bk, int l, int m, const double2* acc) const {
#pragma unroll
    for (int f = 0; f < NF; ++f) finish_field(bk, f, l, m, acc[f]);
  }
  __device__ void zero(int, int, int) const {}
};

// Arithmetic of the column kernel: FP64, or double-float on split-precision
// plans (whose transforms carry ~48 bits).
__device__ __forceinline__ double pe_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double pe_add(double a, double b) { return a + b; }
__device__ __forceinline__ double pe_sub(double a, double b) { return a - b; }
__device__ __forceinline__ double pe_neg(double a) { return -a; }
__device__ __forceinline__ double pe_half(double a) { return 0.5 * a; }
__device__ __forceinline__ df pe_mul(df a, df b) { return df_mul(a, b); }
__device__ __forceinline__ df pe_add(df a, df b) { return df_add(a, b); }
__device__ __forceinline__ df pe_sub(df a, df b) { return df_sub(a, b); }
__device__ __forceinline__ df pe_neg(df a) { return df_neg(a); }
__device__ __forceinline__ df pe_half(df a) { return df_scale2(a, 0.5f); }
__device__ __forceinline__ void pe_const(double x, double& v) { v = x; }
__device__ __forceinline__ void pe_const(double x, df& v) { v = df_of_f64(x); }
__device__ __forceinline__ void pe_recip(double c, double& v) { v = 1.0 / c; }
__device__ __forceinline__ void pe_recip(double c, df& v) { v = df_recip(df_of_f64(c)); }
// Grid values as stored: in the kernel's arithmetic, or FP64 around a
// double-float column (split-precision point-set plans).
template <class V>
__device__ __forceinline__ V pe_ld(V v) { return v; }
template <class V, class = std::enable_if_t<std::is_same<V, df>::value>>
__device__ __forceinline__ df pe_ld(double v) { return df_of_f64(v); }
__device__ __forceinline__ void pe_st(double& o, double v) { o = v; }
__device__ __forceinline__ void pe_st(df& o, df v) { o = v; }
__device__ __forceinline__ void pe_st(double& o, df v) { o = f64_of_df(v); }
struct PeCol {  // column constants of either arithmetic
  template <class V>
  using Sigma = std::conditional_t<std::is_same<V, df>::value, PeSigmaDf, PeSigma>;
};

constexpr int kPeColWarps = 8;

// One warp per 32 points and every eighth level, the column of each point in
// shared memory: u, v, T and the running sum are exchanged there, A and G
// kept for the second pass.  A thread per column (levels in sequence) left
// 64 x 128 points on a third of the chip and spilled the FP64 column to local
// memory; the double-float form had to run the first pass twice.
template <class V, class G>
__global__ void __launch_bounds__(32 * kPeColWarps) pe_level_columns_kernel(
    typename PeCol::Sigma<V> sg, long np, int nlon, const double* __restrict__ coslat, const double* __restrict__ fgrid,
    double f10, long ncolumns, double r_dry, double kappa, const G* grid, G* prod) {
  extern __shared__ char smem_pe[];
  V* sh = reinterpret_cast<V*>(smem_pe);  // [6][K][32]: u, v, T, A, G, running sum
  pdl_wait();
  const int K = sg.K, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long col = (long)blockIdx.x * 32 + lane;
  const bool in = col < ncolumns;
  const long cc = in ? col : ncolumns - 1;
  const long b = cc / np, p = cc - b * np;
  const G* Gd = grid + b * (K + 1) * kPeGrid * np + p;
  G* P = prod + b * (K + 1) * kPeProd * np + p;
  V ic, f, kap, rd, zero;
  pe_recip(coslat[nlon > 0 ? p / nlon : p], ic);
  pe_const(f10 * fgrid[nlon > 0 ? p / nlon : p], f);
  pe_const(kappa, kap);
  pe_const(r_dry, rd);
  pe_const(0.0, zero);
  const G* Gs = Gd + (long)K * kPeGrid * np;
  const V lp_lam = pe_ld<V>(Gs[5 * np]), lp_snt = pe_ld<V>(Gs[6 * np]);
  auto S = [&](int a, int k) -> V& { return sh[(a * K + k) * 32 + lane]; };
  for (int k = warp; k < K; k += kPeColWarps) {
    const G* g = Gd + (long)kPeGrid * k * np;
    const V u = pe_mul(pe_ld<V>(g[0]), ic), v = pe_mul(pe_ld<V>(g[np]), ic);
    const V A = pe_mul(pe_sub(pe_mul(u, lp_lam), pe_mul(v, lp_snt)), ic);  // V . grad(ln p_s)
    const V D = pe_add(pe_ld<V>(g[3 * np]), A);                            // delta + A
    S(0, k) = u;
    S(1, k) = v;
    S(2, k) = pe_ld<V>(g[4 * np]);
    S(3, k) = A;
    S(4, k) = D;
    S(5, k) = pe_mul(sg.dsig[k], D);
  }
  __syncthreads();
  if (warp == 0) {  // cumulative thickness-weighted G, top to bottom
    V acc = S(5, 0);
    for (int k = 1; k < K; ++k) {
      acc = pe_add(acc, S(5, k));
      S(5, k) = acc;
    }
  }
  __syncthreads();
  const V total = S(5, K - 1);
  const V gu = pe_mul(lp_lam, ic), gv = pe_neg(pe_mul(lp_snt, ic));  // grad(ln p_s)
  if (!in) return;
  if (warp == K % kPeColWarps) {  // the level of ln p_s
    G* o = P + (long)K * kPeProd * np;
    pe_st(o[0], pe_neg(total));  // d ln p_s / dt
#pragma unroll
    for (int q = 1; q < kPeProd; ++q) pe_st(o[q * np], zero);
  }
  for (int k = warp; k < K; k += kPeColWarps) {
    const G* g = Gd + (long)kPeGrid * k * np;
    const V zeta = pe_ld<V>(g[2 * np]), delta = pe_ld<V>(g[3 * np]);
    const V t_lam = pe_ld<V>(g[5 * np]), t_snt = pe_ld<V>(g[6 * np]);
    const V e_lam = pe_ld<V>(g[7 * np]), e_snt = pe_ld<V>(g[8 * np]);
    const V u = S(0, k), v = S(1, k), T = S(2, k), A = S(3, k), D = S(4, k);
    // interface sigma_dot above and below (exact zeros at the top and the surface)
    V sd0 = zero, sd1 = zero;
    if (k > 0) sd0 = pe_sub(pe_mul(sg.s[k], total), S(5, k - 1));
    if (k + 1 < K) sd1 = pe_sub(pe_mul(sg.s[k + 1], total), S(5, k));
    auto vadv = [&](int a) {  // centred vertical advection of array a
      if (K == 1) return zero;
      V r = zero;
      if (k + 1 < K) r = pe_mul(sd1, pe_sub(S(a, k + 1), S(a, k)));
      if (k > 0) {
        const V up = pe_mul(sd0, pe_sub(S(a, k), S(a, k - 1)));
        r = k + 1 < K ? pe_add(r, up) : up;
      }
      return pe_mul(r, sg.h2[k]);
    };
    const V eta = pe_add(zeta, f);
    V wp = k == 0 ? A : pe_sub(A, pe_mul(sg.bd[k], S(5, k - 1)));
    wp = pe_sub(wp, pe_mul(sg.alpha[k], D));
    const V adv_t = pe_mul(pe_sub(pe_mul(u, t_lam), pe_mul(v, t_snt)), ic);
    G* o = P + (long)kPeProd * k * np;
    pe_st(o[0], pe_add(pe_sub(pe_neg(adv_t), vadv(2)), pe_mul(pe_mul(kap, T), wp)));
    pe_st(o[np], pe_neg(pe_add(pe_mul(pe_sub(pe_mul(u, e_lam), pe_mul(v, e_snt)), ic), pe_mul(eta, delta))));
    pe_st(o[2 * np], pe_add(pe_mul(eta, zeta), pe_mul(pe_add(pe_mul(v, e_lam), pe_mul(u, e_snt)), ic)));
    pe_st(o[3 * np], pe_half(pe_add(pe_mul(u, u), pe_mul(v, v))));
    const V rt = pe_mul(rd, T);
    pe_st(o[4 * np], pe_mul(pe_add(vadv(0), pe_mul(rt, gu)), ic));  // Z / cos
    pe_st(o[5 * np], pe_mul(pe_add(vadv(1), pe_mul(rt, gv)), ic));
  }
}

// What becomes of a tendency value: stored (stage 0) or one RK4 stage update
// (rk4_stage_kernel's operations and roundings).  ys may be the stage input:
// each CTA reads what it needs of it before it writes.
struct PeOut {
  int stage;
  double dt;
  double2 *tend, *y0, *ys, *acc;
  __device__ __forceinline__ double2 axpy(double2 y, double c, double2 k) const {
    return make_double2(__dadd_rn(y.x, __dmul_rn(c, k.x)), __dadd_rn(y.y, __dmul_rn(c, k.y)));
  }
  __device__ __forceinline__ void put(long i, double2 k) const {
    if (stage == 0) {
      tend[i] = k;
    } else if (stage == 1) {
      acc[i] = k;
      ys[i] = axpy(y0[i], 0.5 * dt, k);
    } else if (stage < 4) {
      acc[i] = axpy(acc[i], 2.0, k);
      ys[i] = axpy(y0[i], stage == 2 ? 0.5 * dt : dt, k);
    } else {
      const double2 a = acc[i];
      y0[i] = axpy(y0[i], dt / 6.0, make_double2(__dadd_rn(a.x, k.x), __dadd_rn(a.y, k.y)));
    }
  }
};

// Weak-form curl/div of Z, 2/3 cuts, Simmons-Burridge geopotential of the
// spectral T (scanned upward in shared memory), -lap(KE + Phi), pins: one
// warp per 32 (l, m) slots and every eighth level.
__global__ void __launch_bounds__(32 * kPeColWarps) pe_level_spectral_kernel(PeSigma sg, Spec s, double r_dry, int batch,
                                                                           const double2* st, const double2* an,
                                                                           const double2* __restrict__ phis, PeOut out) {
  extern __shared__ char smem_pe[];
  double2* below = reinterpret_cast<double2*>(smem_pe);  // [K][32] geopotential under level k, less Phi_s
  pdl_wait();
  const int K = sg.K, L = s.L, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long n2 = (long)(L + 1) * (L + 1);
  const long idx = (long)blockIdx.x * 32 + lane;
  const bool in = idx < n2 * batch;
  const long ii = in ? idx : 0;
  const int b = (int)(ii / n2);
  const long r = ii - b * n2;
  const int l = (int)(r / (L + 1)), m = (int)(r - (long)l * (L + 1));
  const long base = (long)b * (3 * K + 1) * n2 + r;
  const double2 zero = make_double2(0.0, 0.0);
  const double2* T = st + base + (long)2 * K * n2;
  const bool low = in && m <= l;
  if (low)
    for (int k = warp; k < K; k += kPeColWarps) below[k * 32 + lane] = T[(long)k * n2];
  __syncthreads();
  if (warp == 0 && low) {
    double2 acc = phis[r];
    for (int k = K - 1; k >= 0; --k) {
      const double2 Tk = below[k * 32 + lane];
      below[k * 32 + lane] = cadd(acc, cscale(r_dry * sg.alpha[k], Tk));  // Phi_k
      if (k > 0) acc = cadd(acc, cscale(r_dry * sg.beta[k], Tk));
    }
  }
  __syncthreads();
  if (!in) return;
  const int cut = (2 * L) / 3;
  const bool keep = low && l <= cut && m <= cut;
  const double lap = s.lap(l), mr = (double)m * s.ir;
  const double cp = keep && l < L ? s.ir * s.cplus[r] : 0.0, cm = keep && l > m ? s.ir * s.cminus[r] : 0.0;
  for (int k = warp; k <= K; k += kPeColWarps) {
    const double2* a = an + ((long)b * (K + 1) + k) * kPeProd * n2 + r;
    if (k == K) {
      out.put(base + (long)3 * K * n2, keep ? a[0] : zero);
      continue;
    }
    double2 zd = zero, dd = zero, ke = zero, td = zero;
    if (keep) {
      const double2 *A = a + 4 * n2, *B = a + 5 * n2;  // analysed Z_east / cos, Z_north / cos
      auto snt = [&](const double2* c) {               // (1/R) (C+_l c_{l+1} + C-_l c_{l-1})
        const double2 up = l < L ? c[L + 1] : zero, dn = l > m ? c[-(L + 1)] : zero;
        return make_double2(fma(cp, up.x, cm * dn.x), fma(cp, up.y, cm * dn.y));
      };
      const double2 sa = snt(A), sb = snt(B), al = A[0], bl = B[0];
      const double2 div = make_double2(fma(-mr, al.y, sb.x), fma(mr, al.x, sb.y));
      const double2 curl = make_double2(fma(-mr, bl.y, -sa.x), fma(mr, bl.x, -sa.y));
      td = a[0];
      zd = csub(a[n2], curl);
      dd = csub(a[2 * n2], div);
      ke = a[3 * n2];
    }
    out.put(base + (long)(2 * K + k) * n2, td);
    out.put(base + (long)k * n2, l == 0 ? zero : zd);
    const double2 phi = low ? below[k * 32 + lane] : zero;
    out.put(base + (long)(K + k) * n2, l == 0 || !low ? zero : csub(dd, cscale(lap, cadd(ke, phi))));
  }
}

size_t pe_grid_bytes(const aeolus_plan_impl* p, int nlev, int batch) {
  return align256((size_t)batch * (nlev + 1) * kPeGrid * p->npoints * 8);
}
size_t pe_prod_bytes(const aeolus_plan_impl* p, int nlev, int batch) {
  return align256((size_t)batch * (nlev + 1) * kPeProd * p->npoints * 8);
}
size_t pe_state_bytes(const aeolus_plan_impl* p, int nlev, int batch) {
  return align256((size_t)batch * (3 * nlev + 1) * (p->lmax + 1) * (p->lmax + 1) * sizeof(double2));
}
size_t pe_bytes(const aeolus_plan_impl* p, int nlev, int batch) {
  const int bk = batch * (nlev + 1);
  return pe_grid_bytes(p, nlev, batch) + pe_prod_bytes(p, nlev, batch) +
         align256((size_t)bk * kPeProd * (p->lmax + 1) * (p->lmax + 1) * sizeof(double2)) +
         std::max(synth_chain_bytes<kPeGrid, kPeGrid>(p, bk), anal_chain_bytes<kPeProd, kPeProd>(p, bk));
}

template <class V, class G>
int launch_pe_columns(const aeolus_plan_impl* p, const typename PeCol::Sigma<V>& sg, double f10, int batch, double r_dry,
                      double kappa, const void* grid, void* prod, cudaStream_t st) {
  auto kern = pe_level_columns_kernel<V, G>;
  const size_t sm = (size_t)6 * sg.K * 32 * sizeof(V);
  if (int s = allow_smem(kern, sm)) return s;
  const long ncol = p->npoints * (long)batch;
  ProfScope prof("pe_columns", st);
  launch_pdl(kern, dim3(blocks_for(ncol, 32)), dim3(32 * kPeColWarps), sm, st, sg, p->npoints,
             p->kind == kGauss ? p->nlon : 0, static_cast<const double*>(p->coslat),
             static_cast<const double*>(p->fgrid), f10, ncol, r_dry, kappa, static_cast<const G*>(grid),
             static_cast<G*>(prod));
  AE_LAUNCH("pe_level_columns_kernel");
  return AEOLUS_OK;
}

int pe_chain(const aeolus_plan_impl* p, const aeolus_pe_params* prm, const PeSigma& sg, const double2* state,
             const double2* phi_s, const PeOut& out, int batch, void* work, cudaStream_t st) {
  const int K = sg.K, bk = batch * (K + 1);
  const long np = p->npoints;
  char* w = static_cast<char*>(work);
  double* grid = reinterpret_cast<double*>(w);
  w += pe_grid_bytes(p, K, batch);
  double* prod = reinterpret_cast<double*>(w);
  w += pe_prod_bytes(p, K, batch);
  double2* an = reinterpret_cast<double2*>(w);
  w += align256((size_t)bk * kPeProd * (p->lmax + 1) * (p->lmax + 1) * sizeof(double2));
  const Spec sp = make_spec(p, prm->radius);
  const double f10 = 2.0 * prm->omega * kSqrt4PiOver3, kappa = prm->r_dry / prm->cp_dry;
  const PeDerive d{sp, state, K, f10};
  const PeEpi e{an, p->lmax};
  int s;
  if (split_on(p)) {
    if ((s = run_synth_chain<PeDerive, PePw, kOutGridDf>(p, d, PePw{}, bk, grid, kPeGrid * np, np, w, nullptr, st)) ||
        (s = launch_pe_columns<df, df>(p, sigma_df(sg), f10, batch, prm->r_dry, kappa, grid, prod, st)) ||
        (s = run_anal_chain<PwCopyN<kPeProd>, PeEpi, kInGridDf>(p, PwCopyN<kPeProd>{}, e, bk, prod, kPeProd * np, np, w,
                                                                st)))
      return s;
  } else {
    if ((s = run_synth_chain(p, d, PePw{}, bk, grid, kPeGrid * np, np, w, nullptr, st)) ||
        (s = p->precision == AEOLUS_PREC_SPLIT_BF16
                 ? launch_pe_columns<df, double>(p, sigma_df(sg), f10, batch, prm->r_dry, kappa, grid, prod, st)
                 : launch_pe_columns<double, double>(p, sg, f10, batch, prm->r_dry, kappa, grid, prod, st)) ||
        (s = run_anal_chain(p, PwCopyN<kPeProd>{}, e, bk, prod, kPeProd * np, np, w, st)))
      return s;
  }
  const size_t sm = (size_t)K * 32 * sizeof(double2);
  const long n = (long)(p->lmax + 1) * (p->lmax + 1) * batch;
  ProfScope prof("pe_spectral", st);
  launch_pdl(pe_level_spectral_kernel, dim3(blocks_for(n, 32)), dim3(32 * kPeColWarps), sm, st, sg, sp, prm->r_dry, batch,
             state, static_cast<const double2*>(an), phi_s, out);
  AE_LAUNCH("pe_level_spectral_kernel");
  return AEOLUS_OK;
}

int pe_chain_check(aeolus_plan plan, const aeolus_pe_params* prm, int nlev, const double* interfaces, const void* state,
                   const void* phi_s, const void* out, int batch, const char* who, PeSigma* sg) {
  if (int s = check_common(plan, who, batch, state, out)) return s;
  if (int s = pe_check(prm)) return s;
  if (int s = make_sigma(interfaces, nlev, sg)) return s;
  if (batch > 0 && !phi_s) return fail(AEOLUS_ERR_ARG, std::string(who) + ": NULL phi_s");
  // a Gauss plan's kernels take a level of a member per grid row
  if (plan->kind == kGauss && (long)batch * (nlev + 1) > 65535)
    return fail(AEOLUS_ERR_ARG, std::string(who) + ": batch (nlev + 1) above 65535");
  return AEOLUS_OK;
}

// One classical RK4 stage update over n complex values, in the reference's
// order of operations (run/engine.py:406-431), with every FP64 product and
// sum rounded separately (no contraction into FMAs), as NumPy/torch do:
//   stage 1: acc = k;           ys = y0 + (dt/2) k
//   stage 2: acc = acc + 2 k;   ys = y0 + (dt/2) k
//   stage 3: acc = acc + 2 k;   ys = y0 + dt k
//   stage 4: out = y0 + (dt/6) (acc + k)
__global__ void rk4_stage_kernel(int stage, double dt, const double2* __restrict__ y0, const double2* __restrict__ k,
                                 double2* __restrict__ ys, double2* __restrict__ acc, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 kk = k[i], y = y0[i];
  if (stage == 4) {
    const double2 a = acc[i];
    const double c = dt / 6.0;
    const double sx = __dadd_rn(a.x, kk.x), sy = __dadd_rn(a.y, kk.y);
    ys[i] = make_double2(__dadd_rn(y.x, __dmul_rn(c, sx)), __dadd_rn(y.y, __dmul_rn(c, sy)));
    return;
  }
  if (stage == 1) {
    acc[i] = kk;
  } else {
    const double2 a = acc[i];
    acc[i] = make_double2(__dadd_rn(a.x, __dmul_rn(2.0, kk.x)), __dadd_rn(a.y, __dmul_rn(2.0, kk.y)));
  }
  const double c = stage == 3 ? dt : 0.5 * dt;
  ys[i] = make_double2(__dadd_rn(y.x, __dmul_rn(c, kk.x)), __dadd_rn(y.y, __dmul_rn(c, kk.y)));
}

}  // namespace
}  // namespace aeolus

using namespace aeolus;

extern "C" int aeolus_rk4_stage(int stage, double dt, const double* y0, const double* k, double* ystage, double* acc,
                                long n, void* stream) {
  if (stage < 1 || stage > 4 || n < 0 || !std::isfinite(dt))
    return fail(AEOLUS_ERR_ARG, "aeolus_rk4_stage: stage must be 1..4, n >= 0, dt finite");
  if (n == 0) return AEOLUS_OK;
  if (!y0 || !k || !ystage || !acc) return fail(AEOLUS_ERR_ARG, "aeolus_rk4_stage: NULL array");
  if (acc == ystage || acc == k) return fail(AEOLUS_ERR_ARG, "aeolus_rk4_stage: acc must not alias ystage or k");
  ProfScope prof("rk4_stage", static_cast<cudaStream_t>(stream));
  rk4_stage_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      stage, dt, reinterpret_cast<const double2*>(y0), reinterpret_cast<const double2*>(k),
      reinterpret_cast<double2*>(ystage), reinterpret_cast<double2*>(acc), n);
  AE_LAUNCH("rk4_stage_kernel");
  return AEOLUS_OK;
}

extern "C" int aeolus_pe_derive(aeolus_plan plan, const aeolus_pe_params* prm, int nlev, const double* state,
                                double* fields, int batch, void* stream) {
  if (int s = check_common(plan, "aeolus_pe_derive", batch, state, fields)) return s;
  if (int s = pe_check(prm)) return s;
  if (nlev < 1 || nlev > kPeMaxLevels) return fail(AEOLUS_ERR_ARG, "aeolus_pe_derive: bad nlev");
  if (batch == 0) return AEOLUS_OK;
  const long n2 = (long)(plan->lmax + 1) * (plan->lmax + 1);
  ProfScope prof("pe_derive", static_cast<cudaStream_t>(stream));
  const Spec sp = make_spec(plan, prm->radius);
  if (plan->precision == AEOLUS_PREC_SPLIT_BF16 && sp.dcoef_df) {
    pe_derive_df_kernel<<<blocks_for(n2 * (nlev + 1) * batch, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        sp, nlev, batch, 2.0 * prm->omega * kSqrt4PiOver3, reinterpret_cast<const double2*>(state),
        reinterpret_cast<double2*>(fields));
    AE_LAUNCH("pe_derive_df_kernel");
    return AEOLUS_OK;
  }
  pe_derive_kernel<<<blocks_for(n2 * batch, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      sp, nlev, batch, 2.0 * prm->omega * kSqrt4PiOver3, reinterpret_cast<const double2*>(state),
      reinterpret_cast<double2*>(fields));
  AE_LAUNCH("pe_derive_kernel");
  return AEOLUS_OK;
}

extern "C" int aeolus_pe_columns(aeolus_plan plan, const aeolus_pe_params* prm, int nlev, const double* interfaces,
                                 const double* grid, double* prod, double* f_en, int batch, void* stream) {
  if (int s = check_common(plan, "aeolus_pe_columns", batch, grid, prod)) return s;
  if (int s = pe_check(prm)) return s;
  PeSigma sg;
  if (int s = make_sigma(interfaces, nlev, &sg)) return s;
  if (batch > 0 && !f_en) return fail(AEOLUS_ERR_ARG, "aeolus_pe_columns: NULL f_en");
  if (batch == 0) return AEOLUS_OK;
  const long np = plan->npoints;
  const int nlon = plan->kind == kGauss ? plan->nlon : 0;
  ProfScope prof("pe_columns", static_cast<cudaStream_t>(stream));
  if (plan->precision == AEOLUS_PREC_SPLIT_BF16) {  // split plans: the double-float column
    pe_columns_df_kernel<<<blocks_for(np * batch, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        sigma_df(sg), np, nlon, plan->coslat, batch, host_df(prm->r_dry), host_df(prm->r_dry / prm->cp_dry), grid,
        prod, f_en);
    AE_LAUNCH("pe_columns_df_kernel");
    return AEOLUS_OK;
  }
  pe_columns_kernel<<<blocks_for(np * batch, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      sg, np, nlon, plan->coslat, batch, prm->r_dry, prm->r_dry / prm->cp_dry, grid, prod, f_en);
  AE_LAUNCH("pe_columns_kernel");
  return AEOLUS_OK;
}

extern "C" int aeolus_pe_spectral(int lmax, const aeolus_pe_params* prm, int nlev, const double* interfaces,
                                  const double* state, const double* analysed, const double* curl_z,
                                  const double* div_z, const double* phi_s, double* tendency, int batch,
                                  void* stream) {
  if (lmax < 0 || batch < 0) return fail(AEOLUS_ERR_ARG, "aeolus_pe_spectral: bad lmax/batch");
  if (int s = pe_check(prm)) return s;
  PeSigma sg;
  if (int s = make_sigma(interfaces, nlev, &sg)) return s;
  if (batch == 0) return AEOLUS_OK;
  if (!state || !analysed || !curl_z || !div_z || !phi_s || !tendency)
    return fail(AEOLUS_ERR_ARG, "aeolus_pe_spectral: NULL array");
  const long n2 = (long)(lmax + 1) * (lmax + 1);
  ProfScope prof("pe_spectral", static_cast<cudaStream_t>(stream));
  pe_spectral_kernel<<<blocks_for(n2 * batch, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      sg, lmax, prm->radius, prm->r_dry, batch, reinterpret_cast<const double2*>(state),
      reinterpret_cast<const double2*>(analysed), reinterpret_cast<const double2*>(curl_z),
      reinterpret_cast<const double2*>(div_z), reinterpret_cast<const double2*>(phi_s),
      reinterpret_cast<double2*>(tendency));
  AE_LAUNCH("pe_spectral_kernel");
  return AEOLUS_OK;
}

extern "C" int aeolus_pe_workspace_bytes(aeolus_plan plan, int nlev, int batch, size_t* tendency_bytes,
                                         size_t* rk4_bytes) {
  if (!plan_ok(plan) || nlev < 1 || nlev > kPeMaxLevels || batch < 0)
    return fail(AEOLUS_ERR_ARG, "aeolus_pe_workspace_bytes: bad arguments");
  const size_t n = pe_bytes(plan, nlev, std::max(batch, 1));
  if (tendency_bytes) *tendency_bytes = n;
  if (rk4_bytes) *rk4_bytes = n + 2 * pe_state_bytes(plan, nlev, std::max(batch, 1));
  return AEOLUS_OK;
}

extern "C" int aeolus_pe_tendency(aeolus_plan plan, const aeolus_pe_params* prm, int nlev, const double* interfaces,
                                  const double* state, const double* phi_s, double* tendency, int batch, void* work,
                                  size_t work_bytes, void* stream) {
  PeSigma sg;
  if (int s = pe_chain_check(plan, prm, nlev, interfaces, state, phi_s, tendency, batch, "aeolus_pe_tendency", &sg))
    return s;
  if (batch == 0) return AEOLUS_OK;
  if (!work || work_bytes < pe_bytes(plan, nlev, batch))
    return fail(AEOLUS_ERR_WORKSPACE, "aeolus_pe_tendency: workspace too small");
  const PeOut out{0, 0.0, reinterpret_cast<double2*>(tendency), nullptr, nullptr, nullptr};
  return pe_chain(plan, prm, sg, reinterpret_cast<const double2*>(state), reinterpret_cast<const double2*>(phi_s), out,
                  batch, work, static_cast<cudaStream_t>(stream));
}

extern "C" int aeolus_pe_rk4(aeolus_plan plan, const aeolus_pe_params* prm, int nlev, const double* interfaces,
                             double* state, const double* phi_s, int batch, double dt, int nsteps, void* work,
                             size_t work_bytes, void* stream) {
  PeSigma sg;
  if (int s = pe_chain_check(plan, prm, nlev, interfaces, state, phi_s, state, batch, "aeolus_pe_rk4", &sg)) return s;
  if (!std::isfinite(dt)) return fail(AEOLUS_ERR_ARG, "aeolus_pe_rk4: dt must be finite");
  if (batch == 0 || nsteps <= 0) return AEOLUS_OK;
  const size_t nb = pe_bytes(plan, nlev, batch), ns = pe_state_bytes(plan, nlev, batch);
  if (!work || work_bytes < nb + 2 * ns) return fail(AEOLUS_ERR_WORKSPACE, "aeolus_pe_rk4: workspace too small");
  char* w = static_cast<char*>(work);
  double2* y0 = reinterpret_cast<double2*>(state);
  double2* ys = reinterpret_cast<double2*>(w + nb);
  double2* acc = reinterpret_cast<double2*>(w + nb + ns);
  for (int it = 0; it < nsteps; ++it)
    for (int stage = 1; stage <= 4; ++stage) {
      const PeOut out{stage, dt, nullptr, y0, ys, acc};
      if (int s = pe_chain(plan, prm, sg, stage == 1 ? y0 : ys, reinterpret_cast<const double2*>(phi_s), out, batch,
                           work, static_cast<cudaStream_t>(stream)))
        return s;
    }
  return AEOLUS_OK;
}
