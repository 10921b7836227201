// The batch's column (Y) passes in both tile widths and its forward Z passes.
#include "fx_dispatch.cuh"

template <int L, int TK, int T, bool INV, bool HALF>
__global__ void __launch_bounds__(T) kb_col(const BCol* __restrict__ a, const int* __restrict__ starts,
                                             int nseg) {
  int s = find_seg(starts, nseg, blockIdx.x);
  int t = blockIdx.x - starts[s];
  const BCol& c = a[s];
  col_body<L, TK, T, INV, HALF>(c.src, c.dst, c.cp, t);
}
template <int M, int RT, int T, bool COMB>
__global__ void __launch_bounds__(T) kb_zr2c(const BZr2c* __restrict__ a, const int* __restrict__ starts,
                                             int nseg) {
  int s = find_seg(starts, nseg, blockIdx.x);
  int t = blockIdx.x - starts[s];
  const BZr2c& c = a[s];
  zr2c_body<M, RT, T, COMB, true>(c.src, c.dst, c.z, c.cb, c.vec2, RT, t);
}
template <int L, int TK>
static cudaError_t run_col_tk(const BatchLaunch& l, cudaStream_t st) {
  constexpr int T = fx_threads(TK * L);
  constexpr size_t smem = col_smem(L, TK);
  auto go = [&](auto kern) {
    const cudaError_t e = smem_opt_in<smem, tw_smem(L)>(kern);
    if (e != cudaSuccess) return e;
    kern<<<l.blocks, T, smem, st>>>((const BCol*)l.args, l.starts, l.nseg);
    return cudaGetLastError();
  };
  if (l.flag) return l.half ? go(kb_col<L, TK, T, true, true>) : go(kb_col<L, TK, T, true, false>);
  return l.half ? go(kb_col<L, TK, T, false, true>) : go(kb_col<L, TK, T, false, false>);
}
template <int L>
static cudaError_t run_col(const BatchLaunch& l, cudaStream_t st) {
  return l.variant ? run_col_tk<L, col_tk_alt(L)>(l, st) : run_col_tk<L, fx_col_tk(L)>(l, st);
}
template <int M>
static cudaError_t run_zr2c(const BatchLaunch& l, cudaStream_t st) {
  constexpr int RT = fx_rows(M, 1);
  constexpr int T = fx_threads(RT * M);
  constexpr size_t smem = rows_smem(M, RT);
  auto go = [&](auto kern) {
    const cudaError_t e = smem_opt_in<smem, tw_smem(M) + 16 * RT>(kern);
    if (e != cudaSuccess) return e;
    kern<<<l.blocks, T, smem, st>>>((const BZr2c*)l.args, l.starts, l.nseg);
    return cudaGetLastError();
  };
  return l.flag ? go(kb_zr2c<M, RT, T, true>) : go(kb_zr2c<M, RT, T, false>);
}

cudaError_t bx_col(const BatchLaunch& l, cudaStream_t st) {
  switch (l.L) {
#define C_(LL) \
  case LL: return run_col<LL>(l, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
cudaError_t bx_zr2c(const BatchLaunch& l, cudaStream_t st) {
  switch (l.L) {
#define C_(LL) \
  case LL: return run_zr2c<LL>(l, st);
    FX_SIZES(C_)
#undef C_
  }
  return cudaErrorInvalidValue;
}
