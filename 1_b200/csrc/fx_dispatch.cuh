// Launches of the compiled (fixed-length) pass kernels by line length.  The
// kernels of one family and epilogue are instantiated in one translation
// unit each (fx_conv.cu, fx_zinv.cu, fx_batch.cu), so that they compile side by side.
#pragma once
#include "fft_fixed_kernels.cuh"

// fused convolution pass: X axis of a 3D grid (fx_conv_0), Y axis of a film (fx_conv_1)
cudaError_t fx_conv_0(int L, const ConvArgs& a, cudaStream_t st);
cudaError_t fx_conv_1(int L, const ConvArgs& a, cudaStream_t st);
// the same for other line lengths
namespace mix { struct Conv; }
cudaError_t mx_conv_0(const mix::Conv& a, cudaStream_t st);
cudaError_t mx_conv_1(const mix::Conv& a, cudaStream_t st);
// the compiled passes over a batch's instances (half: every instance's data fill half the line)
struct BatchLaunch {
  int L, nseg, blocks, half, variant, flag;
  const void* args;
  const int* starts;
};
cudaError_t bx_conv_0(const BatchLaunch& l, cudaStream_t st);
cudaError_t bx_conv_1(const BatchLaunch& l, cudaStream_t st);
cudaError_t bx_col(const BatchLaunch& l, cudaStream_t st);    // flag: inverse
cudaError_t bx_zr2c(const BatchLaunch& l, cudaStream_t st);   // flag: with the stage combination
// inverse Z with an epilogue (EPI_*), any line length for a single grid;
// fuse: followed by the next evaluation's forward Z
#define FX_ZINV_DECL(MODE)                                                                \
  cudaError_t fx_zinv_##MODE(int M, const ZinvArgs& za, bool fuse, cudaStream_t st);      \
  cudaError_t bx_zinv_##MODE(const BatchLaunch& l, bool fuse, cudaStream_t st);
FX_ZINV_DECL(0)
FX_ZINV_DECL(1)
FX_ZINV_DECL(2)
FX_ZINV_DECL(3)
FX_ZINV_DECL(4)
FX_ZINV_DECL(5)
#undef FX_ZINV_DECL
static inline cudaError_t fx_zinv(int mode, int M, const ZinvArgs& za, bool fuse, cudaStream_t st) {
  switch (mode) {
    case EPI_FIELD: return fx_zinv_0(M, za, fuse, st);
    case EPI_HEUN1: return fx_zinv_1(M, za, fuse, st);
    case EPI_HEUN2: return fx_zinv_2(M, za, fuse, st);
    case EPI_TORQUE: return fx_zinv_3(M, za, fuse, st);
    case EPI_RK: return fx_zinv_4(M, za, fuse, st);
    default: return fx_zinv_5(M, za, fuse, st);
  }
}
static inline cudaError_t bx_zinv(int mode, const BatchLaunch& l, bool fuse, cudaStream_t st) {
  switch (mode) {
    case EPI_HEUN1: return bx_zinv_1(l, fuse, st);
    case EPI_HEUN2: return bx_zinv_2(l, fuse, st);
    case EPI_TORQUE: return bx_zinv_3(l, fuse, st);
    default: return bx_zinv_4(l, fuse, st);
  }
}

__device__ __forceinline__ int find_seg(const int* __restrict__ starts, int nseg, int b) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(&starts[mid]) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// per-instance arguments of a batch launch
struct BCol {
  const float2* src;
  float2* dst;
  ColPass cp;
};
struct BZr2c {
  const float* src;
  float2* dst;
  ZPass z;
  ZComb cb;
  int vec2;
};

// The batch autotuner's alternative column-tile width: half the default where
// that leaves >= 8 columns (more, smaller blocks), else double (fewer,
// larger blocks).
__host__ __device__ constexpr int col_tk_alt(int L) { return fx_col_tk(L) >= 16 ? fx_col_tk(L) / 2 : 2 * fx_col_tk(L); }
__host__ __device__ constexpr int col_tk_variant(int L, int v) { return v ? col_tk_alt(L) : fx_col_tk(L); }
