// The batch's column (Y) passes in both tile widths and its forward Z passes.
#include "fx_dispatch.cuh"

template <typename K>
static void set_smem(K kern, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

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
  size_t smem = sizeof(float2) * (size_t)odd_pitch(TK) * L;
#define KB_COL_(INV, HALF)                                                                        \
  set_smem(kb_col<L, TK, T, INV, HALF>, smem);                                                    \
  kb_col<L, TK, T, INV, HALF><<<l.blocks, T, smem, st>>>((const BCol*)l.args, l.starts, l.nseg);
  if (l.flag) {
    if (l.half) { KB_COL_(true, true) } else { KB_COL_(true, false) }
  } else {
    if (l.half) { KB_COL_(false, true) } else { KB_COL_(false, false) }
  }
#undef KB_COL_
  return cudaGetLastError();
}
template <int L>
static cudaError_t run_col(const BatchLaunch& l, cudaStream_t st) {
  return l.variant ? run_col_tk<L, col_tk_alt(L)>(l, st) : run_col_tk<L, fx_col_tk(L)>(l, st);
}
template <int M>
static cudaError_t run_zr2c(const BatchLaunch& l, cudaStream_t st) {
  constexpr int RT = fx_rows(M, 1);
  constexpr int T = fx_threads(RT * M);
  size_t smem = sizeof(float2) * (size_t)RT * row_pitch(M);
  if (l.flag) {
    set_smem(kb_zr2c<M, RT, T, true>, smem);
    kb_zr2c<M, RT, T, true><<<l.blocks, T, smem, st>>>((const BZr2c*)l.args, l.starts, l.nseg);
  } else {
    set_smem(kb_zr2c<M, RT, T, false>, smem);
    kb_zr2c<M, RT, T, false><<<l.blocks, T, smem, st>>>((const BZr2c*)l.args, l.starts, l.nseg);
  }
  return cudaGetLastError();
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
