// Point-set plan: real basis built on the device (FP64 normalised
// recurrence, one thread per point) and the FP64 basis GEMMs.
#include "points.cuh"

namespace aeolus {

namespace {

constexpr double kInvSqrt4Pi = 0.28209479177387814347;

__global__ void points_basis_kernel(long n, int L, const double* __restrict__ lat, const double* __restrict__ lon,
                                    double* __restrict__ B) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double x = sin(lat[p]);   // cos(colatitude)
  const double s = cos(lat[p]);   // sin(colatitude) >= 0
  const double lam = lon[p];
  double pmm = kInvSqrt4Pi;
  for (int m = 0; m <= L; ++m) {
    if (m > 0) pmm = -sqrt((2.0 * m + 1.0) / (2.0 * m)) * s * pmm;
    double sm, cm;
    sincos(m * lam, &sm, &cm);
    const long cb = col_base(m, L);
    const long sb = cb + (L + 1 - m);
    double p2 = pmm, p1 = 0.0;
    B[(cb + 0) * n + p] = pmm * cm;
    if (m > 0) B[(sb + 0) * n + p] = pmm * sm;
    if (m < L) {
      p1 = sqrt(2.0 * m + 3.0) * x * pmm;
      B[(cb + 1) * n + p] = p1 * cm;
      if (m > 0) B[(sb + 1) * n + p] = p1 * sm;
    }
    for (int l = m + 2; l <= L; ++l) {
      const double a = sqrt((4.0 * l * l - 1.0) / ((double)l * l - (double)m * m));
      const double b = sqrt(((l - 1.0) * (l - 1.0) - (double)m * m) / (4.0 * (l - 1.0) * (l - 1.0) - 1.0));
      const double pl = a * (x * p1 - b * p2);
      B[(cb + (l - m)) * n + p] = pl * cm;
      if (m > 0) B[(sb + (l - m)) * n + p] = pl * sm;
      p2 = p1;
      p1 = pl;
    }
  }
}

}  // namespace

int build_points_basis(aeolus_plan_impl* p, const double* lat, const double* lon) {
  const long n = p->npoints;
  double *dlat = nullptr, *dlon = nullptr;
  AE_CUDA(cudaMalloc(&dlat, n * sizeof(double)));
  AE_CUDA(cudaMalloc(&dlon, n * sizeof(double)));
  int s = cuda_check(cudaMemcpy(dlat, lat, n * sizeof(double), cudaMemcpyHostToDevice), "lat");
  if (!s) s = cuda_check(cudaMemcpy(dlon, lon, n * sizeof(double), cudaMemcpyHostToDevice), "lon");
  if (!s) s = cuda_check(cudaMalloc(&p->basis, (size_t)n * p->ncol * sizeof(double)), "cudaMalloc basis");
  if (!s) {
    points_basis_kernel<<<(unsigned)((n + 127) / 128), 128>>>(n, p->lmax, dlat, dlon, p->basis);
    s = cuda_check(cudaGetLastError(), "points_basis_kernel");
  }
  if (!s) s = cuda_check(cudaDeviceSynchronize(), "points basis");
  cudaFree(dlat);
  cudaFree(dlon);
  p->ld_basis = (int)n;
  return s;
}

// Passes of equal width: ceil(N / 8) passes of NT = ceil(N / passes) columns
// each waste fewer than one column per pass.
namespace {

template <int NT>
void synth_pass(long M, int K, int N, const double* B, const double* V, double* out, cudaStream_t st) {
  const long grid = (M + kPtRows - 1) / kPtRows * ((N + NT - 1) / NT);
  launch_pdl(points_synth_kernel<NT>, dim3((unsigned)grid), dim3(kPtThreads), 0, st, M, K, N, B, V, out);
}

template <int NT>
void analysis_pass(int M, long K, int N, const double* B, const double* W, double* C, cudaStream_t st) {
  const long grid = M * (long)((N + NT - 1) / NT);
  launch_pdl(points_analysis_kernel<NT>, dim3((unsigned)grid), dim3(kPtThreads), 0, st, M, K, N, B, W, C);
}

inline int pass_columns(int N) {
  const int passes = (N + kPtCols - 1) / kPtCols;
  return (N + passes - 1) / passes;
}

}  // namespace

#define AE_PT_PASS(f, nt, ...)                 \
  switch (nt) {                                \
    case 1: f<1>(__VA_ARGS__); break;          \
    case 2: f<2>(__VA_ARGS__); break;          \
    case 3: f<3>(__VA_ARGS__); break;          \
    case 4: f<4>(__VA_ARGS__); break;          \
    case 5: f<5>(__VA_ARGS__); break;          \
    case 6: f<6>(__VA_ARGS__); break;          \
    case 7: f<7>(__VA_ARGS__); break;          \
    default: f<8>(__VA_ARGS__); break;         \
  }

int points_gemm_synth(const aeolus_plan_impl* p, const double* V, double* out, int ncols, cudaStream_t st) {
  ProfScope prof("points_synth_f64", st);
  AE_PT_PASS(synth_pass, pass_columns(ncols), p->npoints, p->ncol, ncols, p->basis, V, out, st)
  AE_LAUNCH("points_synth_kernel");
  return AEOLUS_OK;
}

int points_gemm_analysis(const aeolus_plan_impl* p, const double* W, double* C, int ncols, cudaStream_t st) {
  ProfScope prof("points_analysis_f64", st);
  AE_PT_PASS(analysis_pass, pass_columns(ncols), p->ncol, p->npoints, ncols, p->basis, W, C, st)
  AE_LAUNCH("points_analysis_kernel");
  return AEOLUS_OK;
}

}  // namespace aeolus
