// The fused convolution passes, compiled for one axis each: FX_D2 = 0 the X
// axis of a 3D grid, FX_D2 = 1 the Y axis of a film (single grid and batch).
#include "fx_dispatch.cuh"
#include "fft_mixed.cuh"

template <int L, int TK, int T, bool D2, bool HALF>
// at least 768 resident threads per SM (6 blocks of 128 for L = 64):
// measured faster than the unconstrained 96-register build (5 blocks) and
// than 7 or 8 blocks (register spills)
__global__ void __launch_bounds__(T, (768 / T) > 0 ? (768 / T) : 1) k_conv_fx(ConvArgs a) {
  conv_body<L, TK, T, D2, HALF, !D2>(a, blockIdx.x);
}

template <int L, int TK, int T, bool D2, bool HALF>
__global__ void __launch_bounds__(T) kb_conv(const ConvArgs* __restrict__ a, const int* __restrict__ starts,
                                             int nseg) {
  int s = find_seg(starts, nseg, blockIdx.x);
  conv_body<L, TK, T, D2, HALF>(a[s], blockIdx.x - starts[s]);
}
template <int L, bool D2>
cudaError_t fx_launch_conv(const ConvArgs& a, cudaStream_t st) {
  constexpr int TKP = conv_tkp(L);
  // one thread per (column, radix-8 butterfly): it owns the three components
  constexpr int NBF = TKP * (L / fwd_radix(L, n_stages(L) - 1));
  constexpr int T = NBF < 64 ? 64 : (NBF > 512 ? 512 : ((NBF + 31) / 32) * 32);
  size_t smem = conv_smem(L);
  if (2 * a.n_data == L) {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(k_conv_fx<L, TKP, T, D2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_conv_fx<L, TKP, T, D2, true><<<div_up(a.ncols, TKP), T, smem, st>>>(a);
  } else {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(k_conv_fx<L, TKP, T, D2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_conv_fx<L, TKP, T, D2, false><<<div_up(a.ncols, TKP), T, smem, st>>>(a);
  }
  return cudaGetLastError();
}

// batch: narrow tiles (conv_tkp_narrow)
template <int L, bool D2, bool HALF>
static cudaError_t run_conv(const BatchLaunch& l, cudaStream_t st) {
  constexpr int TKP = conv_tkp_narrow(L);
  constexpr int NBF = TKP * (L / fwd_radix(L, n_stages(L) - 1));
  constexpr int T = NBF < 64 ? 64 : (NBF > 512 ? 512 : ((NBF + 31) / 32) * 32);
  size_t smem = conv_smem_tk(L, TKP);
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(kb_conv<L, TKP, T, D2, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  kb_conv<L, TKP, T, D2, HALF><<<l.blocks, T, smem, st>>>((const ConvArgs*)l.args, l.starts, l.nseg);
  return cudaGetLastError();
}

#define CAT2_(a, b) a##b
#define CAT_(a, b) CAT2_(a, b)
cudaError_t CAT_(fx_conv_, FX_D2)(int L, const ConvArgs& a, cudaStream_t st) {
  switch (L) {
#define C_(LL) \
  case LL: return fx_launch_conv<LL, FX_D2 != 0>(a, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
cudaError_t CAT_(bx_conv_, FX_D2)(const BatchLaunch& l, cudaStream_t st) {
  switch (l.L) {
#define C_(LL) \
  case LL: return l.half ? run_conv<LL, FX_D2 != 0, true>(l, st) : run_conv<LL, FX_D2 != 0, false>(l, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
cudaError_t CAT_(mx_conv_, FX_D2)(const mix::Conv& a, cudaStream_t st) {
  if (3 * a.f.L > 8192) return cudaErrorInvalidValue;
  size_t bytes;
  const int lg = mix::pick_columns(a.f.L, 3, a.f.conv_nst > 1 ? 2 : 0, a.ncols, &bytes);
  cudaError_t e = mix::allow(mix::k_conv_mix<FX_D2 != 0>, bytes);
  if (e != cudaSuccess) return e;
  mix::k_conv_mix<FX_D2 != 0><<<div_up(a.ncols, 1 << lg), mix::T_COL, bytes, st>>>(a, lg);
  return cudaGetLastError();
}
