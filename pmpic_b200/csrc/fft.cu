// fft.cu -- semi-spectral 2-D real transforms (y then x) on the B200.
//
// Restates perform_forward_3dfft / perform_backwards_3dfft
// (model_core/src/fft/pencilfft.F90:151-212) for one GPU: no pencil transposes
// (the whole field is in HBM), FFTE's conventions (ffte_mod.F90:66-124,
// ffte/vzfft1d.f:41-68): forward unscaled, inverse scaled by 1/N per 1-D pass,
// complex-to-real passes ignore the imaginary parts of the zero and Nyquist
// modes (the conjugate-symmetric fill of ffte_c2r).
//
// Layouts (x fastest):  phys (Nz+1) x Ny x Nx;  mid (Nz+1) x (Ny+2) x Nx after
// the y pass (Re/Im of y-mode a interleaved at rows 2a, 2a+1);  spec
// (Nz+1) x (Ny+2) x (Nx+2) after the x pass (the reference's four reals per
// (kx, ky) mode, pencilfft.F90:838-864).
//
// Rows of two register radices (fft_impl.cuh: the four-step kernels) or, for
// the other lengths, a radix-4/2/3/5 Stockham FFT over rows staged in shared
// memory.  Two real rows are packed into one complex row
// (re = row A, im = row B) and separated after the transform, which halves the
// arithmetic of the reference's zero-imaginary complex transforms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "fft_rows.h"

namespace pmpic {

namespace {

bool factor(int n, std::vector<int>& out) {
  out.clear();
  int m = n;
  while (m % 4 == 0) { out.push_back(4); m /= 4; }
  while (m % 2 == 0) { out.push_back(2); m /= 2; }
  while (m % 3 == 0) { out.push_back(3); m /= 3; }
  while (m % 5 == 0) { out.push_back(5); m /= 5; }
  return m == 1;
}

// The register split n = n1 n2 of a row length (0: none), n1 and n2 in 2 .. 16.
// Powers of two from 16 to 256 take the four-step split (st false: any
// factorisation, one twiddle table).  The other lengths take a prefix of the
// Stockham path's stages as n1 and the rest as n2 (st true), so that their
// rows keep that path's order of radices (fft_impl.cuh: fs_step1).  Of several
// the most even one.
void fs_split(FftPlan& p, bool st) {
  p.n1 = p.n2 = 0;
  p.st = st;
  if (!st) {
    for (int a = 4; a <= 16; a *= 2)
      for (int b = 4; b <= a; b *= 2)
        if (a * b == p.n && (!p.n1 || a < p.n1)) {
          p.n1 = a;
          p.n2 = b;
        }
    return;
  }
  int a = 1;
  for (int s = 0; s + 1 < p.nst; ++s) {
    a *= p.radix[s];
    const int b = p.n / a;
    if (a <= 16 && b <= 16 && (!p.n1 || std::max(a, b) < std::max(p.n1, p.n2))) {
      p.n1 = a;
      p.n2 = b;
    }
  }
}

// The split's twiddles, long double accuracy, the index n2 fastest.
// st false: W_n^(n2 k1).  st true, n1 = m1 m2 (m2 = 1: one stage): the first
// stage's W_n^((n2 + n2's range m) k), [m m1 + k], then the second stage's
// W_(n / m1)^(n2 k), [k].
void fs_twiddles(FftPlan& p, bool st, std::vector<double2>& tw) {
  fs_split(p, st);
  p.tw4_off = (int)tw.size();
  if (!p.n1) return;
  auto put = [&](long long num, int den) {
    const long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)num / (long double)den;
    tw.push_back(make_double2((double)cosl(ang), (double)sinl(ang)));
  };
  if (!p.st) {
    for (int k1 = 0; k1 < p.n1; ++k1)
      for (int n2 = 0; n2 < p.n2; ++n2) put((long long)n2 * k1, p.n);
    return;
  }
  const int m1 = p.radix[0], m2 = p.n1 / m1;
  for (int m = 0; m < m2; ++m)
    for (int k = 0; k < m1; ++k)
      for (int n2 = 0; n2 < p.n2; ++n2) put((long long)(n2 + p.n2 * m) * k, p.n);
  for (int k = 0; k < m2; ++k)
    for (int n2 = 0; n2 < p.n2; ++n2) put((long long)n2 * k, p.n / m1);
}

FftPlan make_plan(int n, std::vector<double2>& tw) {
  // twiddles w^(q r) = exp(-2 pi i q r / len) of each Stockham stage, long double accuracy
  FftPlan p{};
  std::vector<int> rad;
  if (!factor(n, rad) || (int)rad.size() > FFT_MAX_STAGES) return p;
  p.n = n;
  p.nst = (int)rad.size();
  int len = n;
  for (int s = 0; s < p.nst; ++s) {
    int R = rad[s], m = len / R;
    p.radix[s] = R;
    p.tw_off[s] = (int)tw.size();
    for (int q = 0; q < m; ++q)
      for (int r = 0; r < R; ++r) {
        long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)((long long)q * r) /
                          (long double)len;
        tw.push_back(make_double2((double)cosl(ang), (double)sinl(ang)));
      }
    len = m;
  }
  return p;
}

}  // namespace

// the transform kernels of the FP64 path (fft32.cu: the FP32 form's)
namespace f64 {
using real = double;
using real2 = double2;
__host__ __device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
#include "fft_impl.cuh"
}  // namespace f64
cudaError_t fft_attributes32(const FftPlan& px, const FftPlan& py);

int fft_init(pmpic_ctx* ctx) {
  std::vector<int> tmp;
  if (!factor(ctx->g.Nx, tmp) || !factor(ctx->g.Ny, tmp))
    return set_error(ctx, PMPIC_ERR_CONFIG, "nx and ny must have only the prime factors 2, 3 and 5");
  std::vector<double2> tw;
  FftPlan px = make_plan(ctx->g.Nx, tw);
  auto pow2 = [](int n) { return n >= 16 && n <= 256 && (n & (n - 1)) == 0; };
  fs_twiddles(px, !pow2(px.n), tw);
  ctx->ftw_off_y = (int)tw.size();
  ctx->ftw_off_x = 0;
  FftPlan py = make_plan(ctx->g.Ny, tw);
  fs_twiddles(py, !(pow2(py.n) && ctx->g.Nx % 16 == 0), tw);
  for (int s = 0; s < py.nst; ++s) py.tw_off[s] -= ctx->ftw_off_y;
  py.tw4_off -= ctx->ftw_off_y;
  PMPIC_CUDA(cudaMalloc(&ctx->ftw, sizeof(double2) * tw.size()));
  PMPIC_CUDA(cudaMemcpy(ctx->ftw, tw.data(), sizeof(double2) * tw.size(), cudaMemcpyHostToDevice));
  // the FP32 table: the same twiddles rounded once to single precision
  std::vector<float2> tw32(tw.size());
  for (size_t i = 0; i < tw.size(); ++i) tw32[i] = make_float2((float)tw[i].x, (float)tw[i].y);
  PMPIC_CUDA(cudaMalloc(&ctx->ftw32, sizeof(float2) * tw32.size()));
  PMPIC_CUDA(cudaMemcpy(ctx->ftw32, tw32.data(), sizeof(float2) * tw32.size(), cudaMemcpyHostToDevice));
  ctx->plan_x = px;
  ctx->plan_y = py;
  // per device (the attribute is a property of the function on the current device)
  PMPIC_CUDA(ctx->mixed ? fft_attributes32(px, py) : f64::fft_attributes(px, py));
  return 0;
}

int fft_forward(pmpic_ctx* ctx, int nb, const double* const* phys, double* const* spec, double* const* mids) {
  return f64::fft_forward_impl(ctx, nb, phys, spec, mids, (const double2*)ctx->ftw);
}
int fft_inverse(pmpic_ctx* ctx, int nb, const SpecIn<double>& S, double* const* phys, double* const* mids) {
  return f64::fft_inverse_impl(ctx, nb, S, phys, mids, (const double2*)ctx->ftw);
}
int fft_tendency(pmpic_ctx* ctx, const SpecIn<double>& S, const double* const* pqr, double* const* dpqr,
                 double* const* mids, double* const* work) {
  return f64::fft_tendency_impl(ctx, S, pqr, dpqr, mids, work, (const double2*)ctx->ftw);
}
int fft_forward(pmpic_ctx* ctx, const double* phys, double* spec) {
  return fft_forward(ctx, 1, &phys, &spec, &ctx->fftmid);
}
int fft_backward(pmpic_ctx* ctx, const double* spec, double* phys) {
  SpecIn<double> S;
  S.x[0] = spec;
  return fft_inverse(ctx, 1, S, &phys, &ctx->fftmid);
}

}  // namespace pmpic
