// The fused convolution passes, compiled for one axis each: FX_D2 = 0 the X
// axis of a 3D grid, FX_D2 = 1 the Y axis of a film (single grid and batch).
#include "fx_dispatch.cuh"
#include "fft_mixed.cuh"

// A film's split blocks come in threes: components 1 and 2 of two tiles of TK
// columns, and component 0 of both, the same number of lines in each.
template <int L, int TK, int T, bool D2, bool HALF, bool STREAM>
__device__ __forceinline__ void conv_block(const ConvArgs& a, int bx) {
  __shared__ float2 tw[L];
  if constexpr (D2 && conv_split(L, TK)) {
    const int g = bx / 3, r = bx - 3 * g;
    if (r == 2) conv_body<L, 2 * TK, T, true, 0, 1, HALF, STREAM>(a, g, tw);
    else conv_body<L, TK, T, true, 1, 2, HALF, STREAM>(a, 2 * g + r, tw);
  } else {
    conv_body<L, TK, T, D2, 0, 3, HALF, STREAM>(a, bx, tw);
  }
}

// at least 768 resident threads per SM (6 blocks of 128 for L = 64):
// measured faster than the unconstrained 96-register build (5 blocks) and
// than 7 or 8 blocks (register spills).  Split blocks of a film: 1024, as far
// as the shared memory of a block allows.  A block that leaves no room for a
// second one has the registers to itself.
__host__ __device__ constexpr int conv_min_blocks(int L, int TK, int T, bool split) {
  const int want = (split ? 1024 : 768) / T;
  const int fit = (int)(220 * 1024 / (conv_smem(L, TK, split) + sizeof(float2) * L + 1024));
  return want < 1 || fit < 2 ? 1 : !split || want < fit ? want : fit;
}
template <int L, int TK, int T, bool D2, bool HALF>
__global__ void __launch_bounds__(T, conv_min_blocks(L, TK, T, D2 && conv_split(L, TK))) k_conv_fx(ConvArgs a) {
  conv_block<L, TK, T, D2, HALF, !D2>(a, blockIdx.x);
}
template <int L, int TK, int T, bool D2, bool HALF>
__global__ void __launch_bounds__(T) kb_conv(const ConvArgs* __restrict__ a, const int* __restrict__ starts,
                                             int nseg) {
  int s = find_seg(starts, nseg, blockIdx.x);
  int t = blockIdx.x - starts[s];
  conv_block<L, TK, T, D2, HALF, false>(a[s], t);
}

// Wide blocks (a thread per component) take 4 columns, a 32-byte
// sector of every row, and serve grids of at most one such block per SM, for the
// lines whose block then has 48 to 768 threads.
#define WIDE_TK 4
__host__ __device__ constexpr bool wide_ok(int L) {
  return n_stages(L) > 1 && 3 * WIDE_TK * conv_bf(L) >= 48 && 3 * WIDE_TK * conv_bf(L) <= 768;
}
// (A batch keeps its tiles: its launches run side by side and are bound by the
// work of all of them.  Wide blocks and Z tiles of fewer rows for its launches
// of few blocks made a step of 24 instances 393 -> 454 us.)
template <int L, int TK, int T, bool D2, bool HALF>
__global__ void __launch_bounds__(T) k_conv_wide(ConvArgs a) {
  __shared__ float2 tw[L];
  conv_wide_body<L, TK, T, D2, HALF>(a, blockIdx.x, tw);
}

template <int L, bool D2, bool HALF>
static cudaError_t launch_conv(const ConvArgs& a, cudaStream_t st) {
  if constexpr (wide_ok(L)) {
    constexpr int TK = WIDE_TK, T = 3 * TK * conv_bf(L);
    const int blocks = div_up(a.ncols, TK);
    if (blocks <= mmx_sm_count()) {
      constexpr size_t smem = conv_smem(L, TK, false);
      const cudaError_t e = smem_opt_in<smem, tw_smem(L)>(k_conv_wide<L, TK, T, D2, HALF>);
      if (e != cudaSuccess) return e;
      return launch_pass(k_conv_wide<L, TK, T, D2, HALF>, blocks, T, smem, st, a);
    }
  }
  constexpr int TK = conv_cols(L, D2), T = conv_threads(L, TK);
  constexpr bool split = D2 && conv_split(L, TK);
  constexpr size_t smem = conv_smem(L, TK, split);
  const cudaError_t e = smem_opt_in<smem, tw_smem(L)>(k_conv_fx<L, TK, T, D2, HALF>);
  if (e != cudaSuccess) return e;
  return launch_pass(k_conv_fx<L, TK, T, D2, HALF>, split ? 3 * div_up(a.ncols, 2 * TK) : div_up(a.ncols, TK), T, smem, st, a);
}
template <int L, bool D2>
static cudaError_t fx_launch_conv(const ConvArgs& a, cudaStream_t st) {
  return 2 * a.n_data == L ? launch_conv<L, D2, true>(a, st) : launch_conv<L, D2, false>(a, st);
}

// batch: narrow tiles (conv_tkp_narrow)
template <int L, bool D2, bool HALF>
static cudaError_t run_conv(const BatchLaunch& l, cudaStream_t st) {
  constexpr int TK = conv_tkp_narrow(L), T = conv_threads(L, TK);
  constexpr bool split = D2 && conv_split(L, TK);
  constexpr size_t smem = conv_smem(L, TK, split);
  const cudaError_t e = smem_opt_in<smem, tw_smem(L)>(kb_conv<L, TK, T, D2, HALF>);
  if (e != cudaSuccess) return e;
  kb_conv<L, TK, T, D2, HALF><<<l.blocks, T, smem, st>>>((const ConvArgs*)l.args, l.starts, l.nseg);
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
  // a stage's items are the butterflies of three components; the product's are of all three
  int items[8], radix[8];
  for (int s = 0; s < a.f.conv_nst; s++) {
    const int r = (int)((a.f.conv_code >> (8 * s)) & 255), last = s == a.f.conv_nst - 1;
    items[s] = ((last ? 1 : 3) * (a.f.L / r)) << lg;
    radix[s] = (last ? 3 : 1) * r;
  }
  const int blocks = div_up(a.ncols, 1 << lg);
  if (a.f.conv_small) {
    cudaError_t e = mix::allow(mix::k_conv_mix<FX_D2 != 0, true>, bytes);
    if (e != cudaSuccess) return e;
    const int t = mix::pick_threads(a.f.conv_nst, items, radix, 256);
    return launch_pass(mix::k_conv_mix<FX_D2 != 0, true>, blocks, t, bytes, st, a, lg);
  }
  cudaError_t e = mix::allow(mix::k_conv_mix<FX_D2 != 0, false>, bytes);
  if (e != cudaSuccess) return e;
  const int t = mix::pick_threads(a.f.conv_nst, items, radix, 128);
  return launch_pass(mix::k_conv_mix<FX_D2 != 0, false>, blocks, t, bytes, st, a, lg);
}
