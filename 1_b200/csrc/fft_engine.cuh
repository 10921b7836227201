// Line transforms of the LLG engine: the run-time plan of a line and the
// butterflies the compiled passes (fft_fixed.cuh) use.
//
// Twiddles come from a per-length table tw[t] = exp(-2 pi i t / Lt) in
// float, computed in double on the host; a stage of radix R at span ns
// uses tw[(q * (j mod ns) * (L / (ns R))) * tws] with Lt = L * tws.
#pragma once
#include "mmx_common.cuh"

// A line length is any product of 2, 3, 5 and 7.  The radix of stage s is
// byte s of 'code'; the second plan, for the fused convolution, ends with a
// radix of at most 10 (5 where that takes no more stages).
struct LineFFT {
  int L;                       // complex length of the line
  int nst, conv_nst;           // number of stages
  int conv_small;              // the convolution plan's radices are at most 12, its last at most 5
  unsigned long long code, conv_code;
  const float2* tw;            // twiddle table, length L * tws
  int tws;                     // table stride (table built for a multiple of L)
};

// complex product with two fused multiply-adds (the transforms are
// compared with the FP64 oracle within a tolerance, never bit for bit)
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// multiply by -i (forward) or +i (inverse)
__device__ __forceinline__ float2 mul_mi(float2 a, bool inv) {
  return inv ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <int R>
struct Radix {
  // out = DFT_R(v), sign -1 (forward) or +1 (inverse)
  __device__ __forceinline__ static void dft(float2* v, bool inv);
};

template <>
__device__ __forceinline__ void Radix<2>::dft(float2* v, bool) {
  float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <>
__device__ __forceinline__ void Radix<4>::dft(float2* v, bool inv) {
  float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
  float2 t2 = cadd(v[1], v[3]), t3 = mul_mi(csub(v[1], v[3]), inv);
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  v[1] = cadd(t1, t3);
  v[3] = csub(t1, t3);
}

template <>
__device__ __forceinline__ void Radix<8>::dft(float2* v, bool inv) {
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  Radix<4>::dft(e, inv);
  Radix<4>::dft(o, inv);
  const float h = 0.70710678118654752440f;
  // W8^1, W8^2, W8^3 for the given direction
  float2 w1 = inv ? make_float2(h, h) : make_float2(h, -h);
  float2 w3 = inv ? make_float2(-h, h) : make_float2(-h, -h);
  float2 o1 = cmul(o[1], w1);
  float2 o2 = mul_mi(o[2], inv);
  float2 o3 = cmul(o[3], w3);
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  v[1] = cadd(e[1], o1);
  v[5] = csub(e[1], o1);
  v[2] = cadd(e[2], o2);
  v[6] = csub(e[2], o2);
  v[3] = cadd(e[3], o3);
  v[7] = csub(e[3], o3);
}

// Radix 16 (fixed-size transforms only): two radix-8 DFTs of the even and
// odd samples combined with the twiddles W16^k.
template <>
__device__ __forceinline__ void Radix<16>::dft(float2* v, bool inv) {
  float2 e[8], o[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  Radix<8>::dft(e, inv);
  Radix<8>::dft(o, inv);
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
  // W16^k = exp(-+ 2 pi i k / 16), k = 1..7 (conjugated for the inverse)
  const float wr[8] = {1.f, c1, h, s1, 0.f, -s1, -h, -c1};
  const float wi[8] = {0.f, s1, h, c1, 1.f, c1, h, s1};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    float2 t = k == 0 ? o[0] : k == 4 ? mul_mi(o[4], inv) : cmul(o[k], make_float2(wr[k], inv ? wi[k] : -wi[k]));
    v[k] = cadd(e[k], t);
    v[k + 8] = csub(e[k], t);
  }
}

// Radix-R DFTs whose upper half of inputs is zero (a zero-padded line's
// first stage): the zero terms are never added.
template <int R>
__device__ __forceinline__ void dft_half(float2* v, bool inv);
template <>
__device__ __forceinline__ void dft_half<8>(float2* v, bool inv) {
  // DFT4 of [a, b, 0, 0] = (a + b, a + W4 b, a - b, a - W4 b)
  float2 mb = mul_mi(v[2], inv), md = mul_mi(v[3], inv);
  float2 e[4] = {cadd(v[0], v[2]), cadd(v[0], mb), csub(v[0], v[2]), csub(v[0], mb)};
  float2 o[4] = {cadd(v[1], v[3]), cadd(v[1], md), csub(v[1], v[3]), csub(v[1], md)};
  const float h = 0.70710678118654752440f;
  float2 w1 = inv ? make_float2(h, h) : make_float2(h, -h);
  float2 w3 = inv ? make_float2(-h, h) : make_float2(-h, -h);
  float2 o1 = cmul(o[1], w1);
  float2 o2 = mul_mi(o[2], inv);
  float2 o3 = cmul(o[3], w3);
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  v[1] = cadd(e[1], o1);
  v[5] = csub(e[1], o1);
  v[2] = cadd(e[2], o2);
  v[6] = csub(e[2], o2);
  v[3] = cadd(e[3], o3);
  v[7] = csub(e[3], o3);
}
template <>
__device__ __forceinline__ void dft_half<16>(float2* v, bool inv) {
  float2 e[8], o[8];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  dft_half<8>(e, inv);
  dft_half<8>(o, inv);
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
  const float wr[8] = {1.f, c1, h, s1, 0.f, -s1, -h, -c1};
  const float wi[8] = {0.f, s1, h, c1, 1.f, c1, h, s1};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    float2 t = k == 0 ? o[0] : k == 4 ? mul_mi(o[4], inv) : cmul(o[k], make_float2(wr[k], inv ? wi[k] : -wi[k]));
    v[k] = cadd(e[k], t);
    v[k + 8] = csub(e[k], t);
  }
}

// ---------------------------------------------------------------------
// Host-side plan construction helpers (fft_engine.cu).
// ---------------------------------------------------------------------
// Splits L into as few stages as the radices of fft_mixed.cuh allow.
// Returns false if L has a prime factor above 7.
bool fft_factor(int L, LineFFT* f);
// Device twiddle table exp(-2 pi i t / Lt), t < Lt, cached per length for
// the lifetime of the process.
const float2* fft_twiddles(int Lt);
