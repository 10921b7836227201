// Kernel spectrum octant and the per-bin 3x3 kernel products.
#pragma once
#include "llg_ops.cuh"

struct KernOct {
  const float* kh;  // [6][O0][O1][HZ]
  int O0, O1, HZ, P0, P1;
  int64_t cs;       // component stride
};

__device__ __forceinline__ void kern_at(const KernOct& K, int kx, int ky, int kz, float& Kxx, float& Kyy,
                                        float& Kzz, float& Kyz, float& Kxz, float& Kxy) {
  int fx = kx <= K.P0 / 2 ? kx : K.P0 - kx;
  int fy = ky <= K.P1 / 2 ? ky : K.P1 - ky;
  bool nx = kx > K.P0 / 2, ny = ky > K.P1 / 2;
  int64_t o = ((int64_t)fx * K.O1 + fy) * K.HZ + kz;
  Kxx = __ldg(K.kh + o);
  Kyy = __ldg(K.kh + K.cs + o);
  Kzz = __ldg(K.kh + 2 * K.cs + o);
  Kyz = __ldg(K.kh + 3 * K.cs + o);
  Kxz = __ldg(K.kh + 4 * K.cs + o);
  Kxy = __ldg(K.kh + 5 * K.cs + o);
  if (ny) Kyz = -Kyz;
  if (nx) Kxz = -Kxz;
  if (nx != ny) Kxy = -Kxy;
}

// H = K M per bin with fused multiply-adds, for the fused convolution
// passes (their results are compared with the FP64 oracle within a
// tolerance; the drop-in gpu_kernelmul6/4 keep the rounding of gpu_kernmul.cu).
__device__ __forceinline__ void kmul6_fma(float2& mx, float2& my, float2& mz, float Kxx, float Kyy, float Kzz,
                                          float Kyz, float Kxz, float Kxy) {
  float2 hx, hy, hz;
  hx.x = fmaf(mz.x, Kxz, fmaf(my.x, Kxy, mx.x * Kxx));
  hx.y = fmaf(mz.y, Kxz, fmaf(my.y, Kxy, mx.y * Kxx));
  hy.x = fmaf(mz.x, Kyz, fmaf(my.x, Kyy, mx.x * Kxy));
  hy.y = fmaf(mz.y, Kyz, fmaf(my.y, Kyy, mx.y * Kxy));
  hz.x = fmaf(mz.x, Kzz, fmaf(my.x, Kyz, mx.x * Kxz));
  hz.y = fmaf(mz.y, Kzz, fmaf(my.y, Kyz, mx.y * Kxz));
  mx = hx;
  my = hy;
  mz = hz;
}
__device__ __forceinline__ void kmul2_fma(float2& my, float2& mz, float Kyy, float Kzz, float Kyz) {
  const float2 hy = make_float2(fmaf(mz.x, Kyz, my.x * Kyy), fmaf(mz.y, Kyz, my.y * Kyy));
  const float2 hz = make_float2(fmaf(mz.x, Kzz, my.x * Kyz), fmaf(mz.y, Kzz, my.y * Kyz));
  my = hy;
  mz = hz;
}
__device__ __forceinline__ void kmul4_fma(float2& mx, float2& my, float2& mz, float Kxx, float Kyy, float Kzz,
                                          float Kyz) {
  mx = make_float2(mx.x * Kxx, mx.y * Kxx);
  kmul2_fma(my, mz, Kyy, Kzz, Kyz);
}
