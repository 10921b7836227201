// The inverse Z passes with one epilogue each (FX_MODE, an EPI_* value):
// plain and followed by the next evaluation's forward Z, single grid and batch.
#include "fx_dispatch.cuh"
#include "fft_mixed.cuh"

template <int M, int RT, int T, int MODE>
__global__ void __launch_bounds__(T) k_zinv_fx(ZinvArgs za) {
  zinv_body<M, RT, T, MODE, false, false>(za, blockIdx.x);
}
template <int M, int RT, int T, int MODE>
__global__ void __launch_bounds__(T) k_zinv_fwd_fx(ZinvArgs za) {
  zinv_body<M, RT, T, MODE, true, false>(za, blockIdx.x);
}

template <int M, int RT, int T, int MODE, bool FUSE>
__global__ void __launch_bounds__(T) kb_zinv(const ZinvArgs* __restrict__ a, const int* __restrict__ starts,
                                             int nseg) {
  int s = find_seg(starts, nseg, blockIdx.x);
  int t = blockIdx.x - starts[s];
  zinv_body<M, RT, T, MODE, FUSE, true>(a[s], t);
}

// epilogues that a step can follow with the next forward Z, and that a batch runs
static constexpr bool IN_STEP = FX_MODE >= EPI_HEUN1 && FX_MODE <= EPI_RK;

template <int M>
static cudaError_t launch(ZinvArgs za, bool fuse, cudaStream_t st) {
  constexpr int RT = fx_rows(M, 3);
  za.rt = rows_in_use(RT, za.nrows);
  constexpr int T = fx_threads(3 * RT * M);
  constexpr size_t smem = rows_smem(M, 3 * RT);
  auto go = [&](auto kern) {
    const cudaError_t e = smem_opt_in<smem, tw_smem(M) + 8 * RT>(kern);
    if (e != cudaSuccess) return e;
    return launch_pass(kern, div_up(za.nrows, za.rt), T, smem, st, za);
  };
  if (!fuse) return go(k_zinv_fx<M, RT, T, FX_MODE>);
  if constexpr (IN_STEP) return go(k_zinv_fwd_fx<M, RT, T, FX_MODE>);
  return cudaErrorInvalidValue;
}
template <int M>
static cudaError_t launch_batch(const BatchLaunch& l, bool fuse, cudaStream_t st) {
  constexpr int RT = fx_rows(M, 3);
  constexpr int T = fx_threads(3 * RT * M);
  constexpr size_t smem = rows_smem(M, 3 * RT);
  auto go = [&](auto kern) {
    const cudaError_t e = smem_opt_in<smem, tw_smem(M) + 8 * RT>(kern);
    if (e != cudaSuccess) return e;
    kern<<<l.blocks, T, smem, st>>>((const ZinvArgs*)l.args, l.starts, l.nseg);
    return cudaGetLastError();
  };
  if constexpr (IN_STEP) return fuse ? go(kb_zinv<M, RT, T, FX_MODE, true>) : go(kb_zinv<M, RT, T, FX_MODE, false>);
  return cudaErrorInvalidValue;
}

// line lengths without compiled kernels
template <int MODE>
static cudaError_t launch_mix(const ZinvArgs& za, bool fuse, cudaStream_t st) {
  const int M = za.fz.L;
  if (3 * (M + 1) > 8192) return cudaErrorInvalidValue;
  size_t bytes;
  const int rt = mix::pick_rows(M, 3, za.nrows, &bytes);
  auto go = [&](auto kern) {
    cudaError_t e = mix::allow(kern, bytes);
    if (e != cudaSuccess) return e;
    return launch_pass(kern, div_up(za.nrows, rt), mix::T_ROW, bytes, st, za.S, za.fz, za.twP, za.P1, za.HZ, za.CS,
                       za.nrows, za.ea, rt);
  };
  if constexpr (IN_STEP) {
    if (fuse) return go(mix::k_zinv_mix<MODE, true>);
  }
  return fuse ? cudaErrorInvalidValue : go(mix::k_zinv_mix<MODE, false>);
}

#define CAT2_(a, b) a##b
#define CAT_(a, b) CAT2_(a, b)
cudaError_t CAT_(fx_zinv_, FX_MODE)(int M, const ZinvArgs& za, bool fuse, cudaStream_t st) {
  if (!fx_ok(M)) return launch_mix<FX_MODE>(za, fuse, st);
  switch (M) {
#define C_(LL) \
  case LL: return launch<LL>(za, fuse, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
cudaError_t CAT_(bx_zinv_, FX_MODE)(const BatchLaunch& l, bool fuse, cudaStream_t st) {
  switch (l.L) {
#define C_(LL) \
  case LL: return launch_batch<LL>(l, fuse, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
