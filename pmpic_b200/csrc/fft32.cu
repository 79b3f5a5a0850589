// fft32.cu -- the transforms of the mixed-precision form: the kernels of
// fft_impl.cuh in FP32 (fft.cu: the FP64 path, the plans and the tables).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "fft_rows.h"

namespace pmpic {

namespace f32 {
using real = float;
using real2 = float2;
__host__ __device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
#include "fft_impl.cuh"
}  // namespace f32

cudaError_t fft_attributes32(const FftPlan& px, const FftPlan& py) { return f32::fft_attributes(px, py); }
int fft_forward(pmpic_ctx* ctx, int nb, const float* const* phys, float* const* spec, float* const* mids) {
  return f32::fft_forward_impl(ctx, nb, phys, spec, mids, (const float2*)ctx->ftw32);
}
int fft_inverse(pmpic_ctx* ctx, int nb, const SpecIn<float>& S, float* const* phys, float* const* mids) {
  return f32::fft_inverse_impl(ctx, nb, S, phys, mids, (const float2*)ctx->ftw32);
}
int fft_tendency(pmpic_ctx* ctx, const SpecIn<float>& S, const float* const* pqr, float* const* dpqr,
                 float* const* mids, float* const* work) {
  return f32::fft_tendency_impl(ctx, S, pqr, dpqr, mids, work, (const float2*)ctx->ftw32);
}

}  // namespace pmpic
