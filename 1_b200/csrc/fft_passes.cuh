// Pass kernels of the zero-aware padded FFT (see fft_engine.cu).
#pragma once
#include "fft_engine.cuh"

// Rows along Z: real (ld_real floats apart, n_real valid values) <->
// half spectrum (HZ = M + 1 complex values, ld_spec apart).  Row r maps to
// component c, x plane, y row:  r = (c * planes_per_comp + x) *
// rows_per_plane + y.
struct ZPass {
  LineFFT f;               // complex FFT of length M = P2 / 2
  const float2* twP;       // exp(-2 pi i t / P2), t < P2
  int nrows;
  int rows_per_plane;
  int planes_per_comp;
  int ld_real;
  int n_real;              // data values per row (N2)
  int ld_spec;             // HZ
  int64_t plane_stride_spec;
  int64_t comp_stride_real;
  int64_t comp_stride_spec;
};

// Strided columns: line (plane p, column c) has element i at
// p * plane_stride + i * stride_i + c (complex units).  Elements i >= n_in
// are zero; only i < n_out are stored.
struct ColPass {
  LineFFT f;
  int nplanes;
  int64_t plane_stride;
  int ncols;
  int64_t stride_i;
  int n_in;
  int n_out;
  int inv;
};

struct BoxPlan {
  int N[3], P[3], HZ;
  LineFFT fz, fy, fx;
  const float2* twz;
};

__device__ __forceinline__ void zrow_offsets(const ZPass& z, int r, int64_t* roff, int64_t* soff) {
  int per_comp = z.planes_per_comp * z.rows_per_plane;
  int c = r / per_comp;
  int q = r - c * per_comp;
  int x = q / z.rows_per_plane;
  int y = q - x * z.rows_per_plane;
  *roff = c * z.comp_stride_real + (int64_t)q * z.ld_real;
  *soff = c * z.comp_stride_spec + x * z.plane_stride_spec + (int64_t)y * z.ld_spec;
}

// Optional stage combination applied while loading a row: the value
// transformed is  m0 + sum_j (dt a_j) k_j  over the nk stages with a non-zero
// weight (the Runge-Kutta stage input of src/go/sim/rk.go:316-322, same
// operation order), also stored to 'out'.
#define ZCOMB_MAXK 7
struct ZComb {
  const float* m0;
  const float* k[ZCOMB_MAXK];
  float a[ZCOMB_MAXK];
  int nk;
  const float* dt;   // device scalar
  float* out;
};

__device__ __forceinline__ float zcomb_value(const ZComb& cb, float dt, int64_t gi) {
  float q = cb.m0[gi];
#pragma unroll 1
  for (int j = 0; j < cb.nk; j++) q = __fadd_rn(q, __fmul_rn(__fmul_rn(dt, cb.a[j]), cb.k[j][gi]));
  return q;
}

cudaError_t launch_z_r2c(const float* src, float2* dst, const ZPass& zp, cudaStream_t st, const ZComb* cb = nullptr);
cudaError_t launch_z_c2r(const float2* src, float* dst, const ZPass& zp, cudaStream_t st);
cudaError_t launch_col(const float2* src, float2* dst, const ColPass& cp, cudaStream_t st);
int box_plan_init(BoxPlan* p, const int N[3], const int P[3]);
ZPass box_zpass(const BoxPlan* p, int ncomp, int n_x_planes, int64_t comp_stride_real, int64_t comp_stride_spec);
cudaError_t box_forward(const BoxPlan* p, const float* in, float2* spec, cudaStream_t st);
cudaError_t box_inverse(const BoxPlan* p, float2* spec, float* out, cudaStream_t st);
