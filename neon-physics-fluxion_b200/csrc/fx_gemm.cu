// fx_gemm.cu -- NT GEMM dispatch for the DCT stage's reduced-precision
// settings (the kernels live in fx_gemm_tc.cu) and the placing of half products.
#include "fx_internal.h"
#include "fx_gemm.cuh"

namespace fx {

int gemm_nt_tc(fx_ctx *ctx, int precision, int G, const GemmOperands &A,
               const GemmOperands &B, const float *S, const GemmOperands &D,
               cudaStream_t s);
int gemm_half_tc(fx_ctx *ctx, int precision, int G, const GemmOperands &Ah,
                 const GemmOperands &Bh, float *part, cudaStream_t s);

// Places the two half products of a pair:
// kHalfRows: even and odd output rows (2r, 2r + 1) of a C-type product;
// kHalfPair: rows r and G-1-r as E + O and sign (E - O) of a C^T-type one.
__global__ void half_place_kernel(const float *__restrict__ part, int G, int mode, float sign,
                                  const float *__restrict__ S, float *__restrict__ D) {
  const int h = G >> 1;
  const size_t half = (size_t)h * G;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < half;
       o += (size_t)gridDim.x * blockDim.x) {
    const float e = part[o], q = part[half + o];
    const size_t r = o / (size_t)G, c = o - r * (size_t)G;
    size_t o0, o1;
    float v0, v1;
    if (mode == kHalfRows) {
      o0 = (2 * r) * G + c;
      o1 = (2 * r + 1) * G + c;
      v0 = e;
      v1 = q;
    } else {
      o0 = r * G + c;
      o1 = ((size_t)G - 1 - r) * G + c;
      v0 = e + q;
      v1 = sign * (e - q);
    }
    if (S) {
      v0 *= S[o0];
      v1 *= S[o1];
    }
    D[o0] = v0;
    D[o1] = v1;
  }
}

int gemm_half(fx_ctx *ctx, int precision, int G, const GemmOperands &Ah,
              const GemmOperands &Bh, int mode, float sign, const float *S, float *D,
              float *part, cudaStream_t s) {
  if (G % 256 != 0) {
    set_error("gemm_half: G=%d is not a multiple of 256", G);
    return FX_EINVAL;
  }
  FX_TRY(gemm_half_tc(ctx, precision, G, Ah, Bh, part, s));
  half_place_kernel<<<ctx->num_sms * 8, 256, 0, s>>>(part, G, mode, sign, S, D);
  FX_CHECK_LAUNCH();
  ctx->launches += 1;
  return FX_OK;
}

int gemm_nt(fx_ctx *ctx, int precision, int G, const GemmOperands &A,
            const GemmOperands &B, const float *S, const GemmOperands &D,
            cudaStream_t s) {
  if (G % 128 != 0) {
    set_error("gemm_nt: G=%d is not a multiple of 128", G);
    return FX_EINVAL;
  }
  return gemm_nt_tc(ctx, precision, G, A, B, S, D, s);
}

}  // namespace fx
