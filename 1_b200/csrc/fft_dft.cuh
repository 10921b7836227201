// Butterflies of composite and odd radices in registers, with compile-time
// twiddles: radix A * B from A- and B-point transforms, odd primes with the
// products of the pairs (j, R - j) shared.
#pragma once
#include "fft_engine.cuh"

namespace mix {

// cos and sin of 2 pi k / n in float64 at compile time (Taylor series of an
// argument reduced to the first octant)
constexpr double pi = 3.14159265358979323846264338327950288;
constexpr double cos_small(double x) {
  double t = 1, s = 1;
  for (int i = 1; i < 14; i++) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return s;
}
constexpr double sin_small(double x) {
  double t = x, s = x;
  for (int i = 1; i < 14; i++) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return s;
}
constexpr double cos_of(int k, int n);
constexpr double sin_of(int k, int n) {
  k %= n;
  if (2 * k > n) return -sin_of(n - k, n);
  if (4 * k > n) {  // sin(pi - x)
    return 4 * k == n ? 1.0 : (8 * k < 3 * n ? cos_small(2 * pi * (4 * k - n) / (4.0 * n))
                                             : sin_small(2 * pi * (n - 2 * k) / (2.0 * n)));
  }
  return 8 * k <= n ? sin_small(2 * pi * k / n) : cos_small(2 * pi * (n - 4 * k) / (4.0 * n));
}
constexpr double cos_of(int k, int n) { return sin_of((4 * (k % n) + n) % (4 * n), 4 * n); }

// exp(-2 pi i k / n)
template <int K, int N>
struct W {
  static constexpr float c = (float)cos_of(K, N);
  static constexpr float s = (float)-sin_of(K, N);
};
template <int K, int N>
__device__ __forceinline__ float2 times_w(float2 a) {
  constexpr int k = K % N;
  if constexpr (k == 0) return a;
  else if constexpr (4 * k == N) return make_float2(a.y, -a.x);
  else if constexpr (2 * k == N) return make_float2(-a.x, -a.y);
  else if constexpr (4 * k == 3 * N) return make_float2(-a.y, a.x);
  else {
    constexpr float c = W<k, N>::c, s = W<k, N>::s;
    return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c));
  }
}

__host__ __device__ constexpr int split_of(int r) { return r == 4 ? 2 : r == 8 ? 4 : r == 16 ? 4 : r == 6 ? 2 : r == 9 ? 3 : r == 10 ? 2 : r == 12 ? 4 : r == 14 ? 2 : r == 15 ? 3 : r == 20 ? 4 : r == 25 ? 5 : 1; }

// forward DFT of R points in registers
template <int R>
struct Dft;

template <int A, int B, int I>
__device__ __forceinline__ void twiddle_row(float2 (&t)[A]) {
  // t[k1] *= W_(AB)^(I k1)
  if constexpr (A > 1) t[1] = times_w<I * 1, A * B>(t[1]);
  if constexpr (A > 2) t[2] = times_w<I * 2, A * B>(t[2]);
  if constexpr (A > 3) t[3] = times_w<I * 3, A * B>(t[3]);
  if constexpr (A > 4) t[4] = times_w<I * 4, A * B>(t[4]);
}
template <int A, int B, int I>
__device__ __forceinline__ void first_rows(float2 (&u)[B][A], const float2 (&v)[A * B]) {
  if constexpr (I < B) {
#pragma unroll
    for (int n1 = 0; n1 < A; n1++) u[I][n1] = v[n1 * B + I];
    Dft<A>::run(u[I]);
    twiddle_row<A, B, I>(u[I]);
    first_rows<A, B, I + 1>(u, v);
  }
}
// composite R = A B: n = n1 B + n2, k = k1 + A k2
template <int R>
struct Dft {
  __device__ __forceinline__ static void run(float2 (&v)[R]) {
    constexpr int A = split_of(R), B = R / A;
    float2 u[B][A];
    first_rows<A, B, 0>(u, v);
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      float2 w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; n2++) w[n2] = u[n2][k1];
      Dft<B>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = w[k2];
    }
  }
};
template <>
struct Dft<2> {
  __device__ __forceinline__ static void run(float2 (&v)[2]) {
    float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};
template <>
struct Dft<4> {
  __device__ __forceinline__ static void run(float2 (&v)[4]) { Radix<4>::dft(v, false); }
};
// odd primes: pairs (j, R - j) share their products,
// X_k = v0 + sum_j cos(2 pi jk/R) (v_j + v_-j) - i sum_j sin(2 pi jk/R) (v_j - v_-j)
template <int R>
struct DftOdd {
  template <int J, int K>
  __device__ __forceinline__ static void term(const float2 (&s)[R / 2 + 1], const float2 (&d)[R / 2 + 1], float2& a,
                                              float2& b) {
    if constexpr (J <= R / 2) {
      constexpr float c = W<(J * K) % R, R>::c, n = -W<(J * K) % R, R>::s;
      a = make_float2(fmaf(c, s[J].x, a.x), fmaf(c, s[J].y, a.y));
      b = make_float2(fmaf(n, d[J].x, b.x), fmaf(n, d[J].y, b.y));
      term<J + 1, K>(s, d, a, b);
    }
  }
  template <int K>
  __device__ __forceinline__ static void out(float2 (&v)[R], float2 v0, const float2 (&s)[R / 2 + 1],
                                             const float2 (&d)[R / 2 + 1]) {
    if constexpr (K <= R / 2) {
      float2 a = v0, b = make_float2(0.f, 0.f);
      term<1, K>(s, d, a, b);
      v[K] = make_float2(a.x + b.y, a.y - b.x);
      v[R - K] = make_float2(a.x - b.y, a.y + b.x);
      out<K + 1>(v, v0, s, d);
    }
  }
  __device__ __forceinline__ static void run(float2 (&v)[R]) {
    float2 s[R / 2 + 1], d[R / 2 + 1], v0 = v[0];
#pragma unroll
    for (int j = 1; j <= R / 2; j++) {
      s[j] = cadd(v[j], v[R - j]);
      d[j] = csub(v[j], v[R - j]);
      v[0] = cadd(v[0], s[j]);
    }
    out<1>(v, v0, s, d);
  }
};
template <> struct Dft<3> : DftOdd<3> {};
template <> struct Dft<5> : DftOdd<5> {};
template <> struct Dft<7> : DftOdd<7> {};

}  // namespace mix
