// Pass kernels for line lengths without compiled kernels (any product of 2,
// 3, 5 and 7), with the radix plan known at run time only.
//
// A line is split into as few stages as its factors allow, with radices up
// to 25 (fft_factor): 250 = 25 * 10, 200 = 20 * 10, 100 = 10 * 10.  A stage
// picks its radix in one switch, uniform over the block, whose cases are the
// unrolled butterflies of that radix; everything else a stage needs is one
// division by a constant and one by the span.  Stages read one tile in
// shared memory and write another (Stockham order), so a stage costs one
// barrier; the first stage of a column reads global memory and the last one
// writes it, so two-stage columns keep a single tile.  The inverse
// transform is the forward one with real and imaginary parts exchanged on
// the way in and out.  Blocks have 256 threads for rows, and for columns what
// pick_threads says.
//
// Several units include this header.  What is not a template by nature is one
// of a defaulted parameter (template <int = 0>): a unit then compiles only the
// kernels that it launches, and the units' copies are one function.
#pragma once
#include "epilogue.cuh"
#include "fft_dft.cuh"
#include "fft_passes.cuh"
#include "kernmul.cuh"

namespace mix {

// the radices a plan may hold; the last one of a convolution plan (whose three components share a
// thread's registers) is at most 10
#define MIX_CASE_(RR, ...)      \
  case RR: {                    \
    constexpr int R = RR;       \
    __VA_ARGS__;                \
    break;                      \
  }
#define MIX_SMALL(r, ...)                                                                                  \
  switch (r) {                                                                                             \
    MIX_CASE_(2, __VA_ARGS__) MIX_CASE_(3, __VA_ARGS__) MIX_CASE_(4, __VA_ARGS__) MIX_CASE_(5, __VA_ARGS__) \
    MIX_CASE_(6, __VA_ARGS__) MIX_CASE_(7, __VA_ARGS__) MIX_CASE_(8, __VA_ARGS__) MIX_CASE_(9, __VA_ARGS__) \
    MIX_CASE_(10, __VA_ARGS__)                                                                             \
    default: break;                                                                                        \
  }
#define MIX_LE5(r, ...)                                                                                    \
  switch (r) {                                                                                             \
    MIX_CASE_(2, __VA_ARGS__) MIX_CASE_(3, __VA_ARGS__) MIX_CASE_(4, __VA_ARGS__) MIX_CASE_(5, __VA_ARGS__) \
    default: break;                                                                                        \
  }
#define MIX_LE12(r, ...)                                                                                   \
  switch (r) {                                                                                             \
    MIX_CASE_(2, __VA_ARGS__) MIX_CASE_(3, __VA_ARGS__) MIX_CASE_(4, __VA_ARGS__) MIX_CASE_(5, __VA_ARGS__) \
    MIX_CASE_(6, __VA_ARGS__) MIX_CASE_(7, __VA_ARGS__) MIX_CASE_(8, __VA_ARGS__) MIX_CASE_(9, __VA_ARGS__) \
    MIX_CASE_(10, __VA_ARGS__) MIX_CASE_(12, __VA_ARGS__)                                                  \
    default: break;                                                                                        \
  }
#define MIX_RADIX(r, ...)                                                                                  \
  switch (r) {                                                                                             \
    MIX_CASE_(2, __VA_ARGS__) MIX_CASE_(3, __VA_ARGS__) MIX_CASE_(4, __VA_ARGS__) MIX_CASE_(5, __VA_ARGS__) \
    MIX_CASE_(6, __VA_ARGS__) MIX_CASE_(7, __VA_ARGS__) MIX_CASE_(8, __VA_ARGS__) MIX_CASE_(9, __VA_ARGS__) \
    MIX_CASE_(10, __VA_ARGS__) MIX_CASE_(12, __VA_ARGS__) MIX_CASE_(14, __VA_ARGS__)                        \
    MIX_CASE_(15, __VA_ARGS__) MIX_CASE_(16, __VA_ARGS__) MIX_CASE_(20, __VA_ARGS__)                        \
    MIX_CASE_(25, __VA_ARGS__)                                                                             \
    default: break;                                                                                        \
  }

#define MIX_UNROLL _Pragma("unroll")  // inside a macro argument

// n / d by a multiply-high; exact while n d < 2^32
struct Div {
  unsigned d, m;
  __device__ __forceinline__ explicit Div(unsigned d_) : d(d_), m(d_ > 1 ? 0xffffffffu / d_ + 1 : 0) {}
  __device__ __forceinline__ int operator()(int n) const { return d > 1 ? (int)__umulhi((unsigned)n, m) : n; }
};

__device__ __forceinline__ int radix_at(unsigned long long code, int st) { return (int)((code >> (8 * st)) & 255); }
__device__ __forceinline__ float2 swapped(float2 v, bool sw) { return sw ? make_float2(v.y, v.x) : v; }

// butterfly j of a stage of radix R at span ns: ld(i) reads element i of the
// line, st(i, v) writes it
template <int R, typename LD, typename ST>
__device__ __forceinline__ void butterfly(int j, const Div& dns, int ns, int L, const float2* __restrict__ tw, int tws,
                                          LD ld, ST st) {
  const int M = L / R;
  float2 v[R];
#pragma unroll
  for (int q = 0; q < R; q++) v[q] = ld(j + q * M);
  int k = 0;
  if (ns > 1) {
    k = j - dns(j) * ns;
    const int s = k * (L / R / ns) * tws;
#pragma unroll
    for (int q = 1; q < R; q++) v[q] = cmul(v[q], __ldg(tw + q * s));
  }
  Dft<R>::run(v);
  const int o = (j - k) * R + k;
#pragma unroll
  for (int q = 0; q < R; q++) st(o + q * ns, v[q]);
}

__host__ __device__ constexpr int odd_up(int n) { return n | 1; }

// ---------------------------------------------------------------------
// Columns: 2^lg adjacent columns, element i of column l at s[i * TKP + l].
// ---------------------------------------------------------------------
constexpr int T_COL = 256;  // at most

template <int = 0>
__global__ void __launch_bounds__(T_COL, 2) k_col_mix(const float2* src, float2* dst, ColPass cp, int lg) {
  extern __shared__ float2 sm[];
  pass_begin();
  const int TK = 1 << lg, TKP = odd_up(TK), L = cp.f.L, nst = cp.f.nst;
  const int l = threadIdx.x & (TK - 1), j0 = threadIdx.x >> lg, dj = blockDim.x >> lg;
  const int g = blockIdx.x * TK + l, pl = g / cp.ncols;
  const bool ok = g < cp.nplanes * cp.ncols, inv = cp.inv != 0;
  const int64_t base = (int64_t)pl * cp.plane_stride + (g - pl * cp.ncols), sti = cp.stride_i;
  const int n_in = cp.n_in, n_out = cp.n_out;
  auto load = [&](int i) { return ok && i < n_in ? swapped(src[base + i * sti], inv) : make_float2(0.f, 0.f); };
  auto store = [&](int i, float2 v) {
    if (ok && i < n_out) dst[base + i * sti] = swapped(v, inv);
  };
  float2 *x = sm + l, *y = sm + L * TKP + l;
  pass_wait();
  int ns = 1;
  for (int st = 0; st < nst; st++) {
    const int r = radix_at(cp.f.code, st);
    const Div dns(ns);
    auto from = [&](int i) { return x[i * TKP]; };
    auto to = [&](int i, float2 v) { y[i * TKP] = v; };
    auto to0 = [&](int i, float2 v) { x[i * TKP] = v; };
    if (st == 0 && nst == 1) {
      MIX_RADIX(r, for (int j = j0; j < L / R; j += dj) butterfly<R>(j, dns, 1, L, nullptr, 0, load, store))
    } else if (st == 0) {
      MIX_RADIX(r, for (int j = j0; j < L / R; j += dj) butterfly<R>(j, dns, 1, L, nullptr, 0, load, to0))
      __syncthreads();
    } else if (st == nst - 1) {
      MIX_RADIX(r, for (int j = j0; j < L / R; j += dj) butterfly<R>(j, dns, ns, L, cp.f.tw, cp.f.tws, from, store))
    } else {
      MIX_RADIX(r, for (int j = j0; j < L / R; j += dj) butterfly<R>(j, dns, ns, L, cp.f.tw, cp.f.tws, from, to))
      __syncthreads();
      float2* t = x;
      x = y;
      y = t;
    }
    ns *= r;
  }
}

// ---------------------------------------------------------------------
// Fused convolution (ConvArgs of the compiled passes): element i of column
// t, component c at s[i * NLP + c * TK + t].  The last forward stage, the
// kernel product and the first inverse stage (the same radix, so the same
// elements) stay in the registers of one thread.
// ---------------------------------------------------------------------
struct Conv {
  float2* S;
  KernOct K;
  LineFFT f;
  int n_data, ncols, HZ;
  int64_t stride, CS;
};

// SMALL: radices up to 12, the last up to 5 (f.conv_small), which takes 85 instead of
// 168 registers (X lines of 20 points: 47 us with the large ones, 250 x 100 x 10 grid)
#define MIX_ANY(r, ...)                    \
  if constexpr (SMALL) {                   \
    MIX_LE12(r, __VA_ARGS__)               \
  } else {                                 \
    MIX_RADIX(r, __VA_ARGS__)              \
  }
#define MIX_LAST(r, ...)                   \
  if constexpr (SMALL) {                   \
    MIX_LE5(r, __VA_ARGS__)                \
  } else {                                 \
    MIX_SMALL(r, __VA_ARGS__)              \
  }
template <bool D2, bool SMALL>
__global__ void __launch_bounds__(SMALL ? 256 : 128, 3) k_conv_mix(Conv a, int lg) {
  extern __shared__ float2 sm[];
  pass_begin();
  const int TK = 1 << lg, NLP = odd_up(3 * TK), L = a.f.L, nst = a.f.conv_nst;
  const int t = threadIdx.x & (TK - 1), j0 = threadIdx.x >> lg, dj = blockDim.x >> lg;
  const int col = blockIdx.x * TK + t;
  const bool ok = col < a.ncols;
  const int nd = a.n_data;
  int kyc = 0, kzc = col;
  if (!D2) {
    kyc = col / a.HZ;
    kzc = col - kyc * a.HZ;
  }
  float2* S = a.S + col;
  float2 *x = sm + t, *y = sm + L * NLP + t;
  const float2* tw = a.f.tw;
  const int tws = a.f.tws;
  int ns = 1;
  pass_wait();
  // forward stages but the last; a thread's butterflies of all components
  for (int st = 0; st < nst - 1; st++) {
    const int r = radix_at(a.f.conv_code, st);
    const Div dns(ns);
    MIX_ANY(r, {
      const int M = L / R;
      const Div dm(M);
      for (int b = j0; b < 3 * M; b += dj) {
        const int c = dm(b), j = b - c * M;
        if (st == 0)
          butterfly<R>(
              j, dns, 1, L, nullptr, 0,
              [&](int i) { return ok && i < nd ? S[c * a.CS + i * a.stride] : make_float2(0.f, 0.f); },
              [&](int i, float2 v) { x[i * NLP + c * TK] = v; });
        else
          butterfly<R>(
              j, dns, ns, L, tw, tws, [&](int i) { return x[i * NLP + c * TK]; },
              [&](int i, float2 v) { y[i * NLP + c * TK] = v; });
      }
    })
    __syncthreads();
    if (st > 0) {
      float2* s = x;
      x = y;
      y = s;
    }
    ns *= r;
  }
  // last forward stage, kernel product, first inverse stage
  const int rl = radix_at(a.f.conv_code, nst - 1);
  const Div dnl(ns);
  MIX_LAST(rl, {
    const int M = L / R;
    for (int j = j0; j < M; j += dj) {
      float2 v[3][R];
MIX_UNROLL
      for (int c = 0; c < 3; c++) {
MIX_UNROLL
        for (int q = 0; q < R; q++) {
          const int i = j + q * M;
          v[c][q] = nst > 1 ? x[i * NLP + c * TK]
                            : (ok && i < nd ? S[c * a.CS + i * a.stride] : make_float2(0.f, 0.f));
        }
        if (nst > 1) {
          // span L / R: butterfly j has twiddle index j
MIX_UNROLL
          for (int q = 1; q < R; q++) v[c][q] = cmul(v[c][q], __ldg(tw + q * j * tws));
        }
        Dft<R>::run(v[c]);
      }
      if (ok) {
MIX_UNROLL
        for (int q = 0; q < R; q++) {
          float Kxx, Kyy, Kzz, Kyz, Kxz, Kxy;
          kern_at(a.K, D2 ? 0 : j + q * M, D2 ? j + q * M : kyc, kzc, Kxx, Kyy, Kzz, Kyz, Kxz, Kxy);
          if (D2) kmul4_fma(v[0][q], v[1][q], v[2][q], Kxx, Kyy, Kzz, Kyz);
          else kmul6_fma(v[0][q], v[1][q], v[2][q], Kxx, Kyy, Kzz, Kyz, Kxz, Kxy);
        }
      }
MIX_UNROLL
      for (int c = 0; c < 3; c++) {
MIX_UNROLL
        for (int q = 0; q < R; q++) v[c][q] = swapped(v[c][q], true);
        Dft<R>::run(v[c]);
MIX_UNROLL
        for (int q = 0; q < R; q++) {
          if (nst > 1) {
            y[(j * R + q) * NLP + c * TK] = v[c][q];
          } else if (ok && q < nd) {
            S[c * a.CS + q * a.stride] = swapped(v[c][q], true);
          }
        }
      }
    }
  })
  if (nst == 1) return;
  __syncthreads();
  // the other inverse stages, radices in reverse order
  ns = rl;
  for (int st = nst - 2; st >= 0; st--) {
    float2* s = x;
    x = y;
    y = s;
    const int r = radix_at(a.f.conv_code, st);
    const Div dns(ns);
    MIX_ANY(r, {
      const int M = L / R;
      const Div dm(M);
      for (int b = j0; b < 3 * M; b += dj) {
        const int c = dm(b), j = b - c * M;
        if (st == 0)
          butterfly<R>(
              j, dns, ns, L, tw, tws, [&](int i) { return x[i * NLP + c * TK]; },
              [&](int i, float2 v) {
                if (ok && i < nd) S[c * a.CS + i * a.stride] = swapped(v, true);
              });
        else
          butterfly<R>(
              j, dns, ns, L, tw, tws, [&](int i) { return x[i * NLP + c * TK]; },
              [&](int i, float2 v) { y[i * NLP + c * TK] = v; });
      }
    })
    __syncthreads();
    ns *= r;
  }
}

// ---------------------------------------------------------------------
// Rows (the Z axis): RT rows, element i of line l at s[l * pitch + i + i / 16].
// ---------------------------------------------------------------------
constexpr int T_ROW = 256;
__host__ __device__ inline int row_tile_pitch(int M) { return odd_up(M + M / 16); }
__device__ __forceinline__ int at(int i) { return i + (i >> 4); }

// the stages of 'lines' rows from tile x, with tile y to alternate; elements
// from 'limit' on are zero in the first stage.  Returns the tile that holds
// the result.  Called with x complete, returns after a barrier.
template <int = 0>
__device__ __noinline__ float2* row_stages(float2* x, float2* y, const LineFFT& f, int lines, int pitch, int limit) {
  const int L = f.L, nst = f.nst;
  int ns = 1;
  for (int st = 0; st < nst; st++) {
    const int r = radix_at(f.code, st);
    const Div dns(ns);
    const int lim = st == 0 ? limit : L;
    MIX_RADIX(r, {
      const int M = L / R;
      const Div dm(M);
      for (int b = threadIdx.x; b < lines * M; b += T_ROW) {
        const int l = dm(b), j = b - l * M;
        const float2* xs = x + l * pitch;
        float2* ys = y + l * pitch;
        butterfly<R>(
            j, dns, ns, L, f.tw, f.tws, [&](int i) { return i < lim ? xs[at(i)] : make_float2(0.f, 0.f); },
            [&](int i, float2 v) { ys[at(i)] = v; });
      }
    })
    __syncthreads();
    float2* t = x;
    x = y;
    y = t;
    ns *= r;
  }
  return x;
}

// X_k and X_(M-k), k <= M/2, of the real line whose pair transform is z
__device__ __forceinline__ void split_pair(const float2* z, int k, int M, const float2* __restrict__ twP, float2& a,
                                           float2& b) {
  const float2 Zk = z[at(k)], Zm = z[at(k == 0 ? 0 : M - k)];
  const float2 E = make_float2(0.5f * (Zk.x + Zm.x), 0.5f * (Zk.y - Zm.y));
  const float2 O = make_float2(0.5f * (Zk.y + Zm.y), -0.5f * (Zk.x - Zm.x));
  const float2 wo = cmul(__ldg(&twP[k]), O);
  a = make_float2(E.x + wo.x, E.y + wo.y);
  b = make_float2(E.x - wo.x, wo.y - E.y);
}
// Z'_k = (X_k + conj X_(M-k)) + i (X_k - conj X_(M-k)) w^-k, X_0 and X_M real
__device__ __forceinline__ float2 merge_pair(float2 Xk, float2 Xm, int k, const float2* __restrict__ twP) {
  if (k == 0) Xk.y = Xm.y = 0.f;
  const float2 A = make_float2(Xk.x + Xm.x, Xk.y - Xm.y), B = make_float2(Xk.x - Xm.x, Xk.y + Xm.y);
  float2 w = __ldg(&twP[k]);
  w.y = -w.y;
  const float2 C = cmul(B, w);
  return make_float2(A.x - C.y, A.y + C.x);
}

constexpr int MAX_ROWS = 32;

template <bool COMB>
__global__ void __launch_bounds__(T_ROW) k_zr2c_mix(const float* src, float2* dst, ZPass z,
                                                    ZComb cb, int vec2, int RT) {
  extern __shared__ float2 sm[];
  __shared__ int64_t roff_s[MAX_ROWS], soff_s[MAX_ROWS];
  const int M = z.f.L, pitch = row_tile_pitch(M), nreal = z.n_real;
  const int r0 = blockIdx.x * RT, nl = min(RT, z.nrows - r0);
  if ((int)threadIdx.x < nl) zrow_offsets(z, r0 + threadIdx.x, &roff_s[threadIdx.x], &soff_s[threadIdx.x]);
  pass_begin();
  pass_wait();
  __syncthreads();
  // the rows' (x_2n, x_2n+1) pairs, four in flight a thread
  const int np = (nreal + 1) / 2;
  const Div dn(np);
  const float dt = COMB ? *cb.dt : 0.f;
  constexpr int U = 4;
  for (int e0 = threadIdx.x; e0 < nl * np; e0 += U * T_ROW) {
    float2 v[U];
    int64_t gi[U];
    int to[U];
    bool two[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = e0 + u * T_ROW;
      to[u] = -1;
      if (e >= nl * np) continue;
      const int l = dn(e), n = e - l * np;
      to[u] = l * pitch + at(n);
      gi[u] = roff_s[l] + 2 * n;
      two[u] = 2 * n + 1 < nreal;
      const float* s = COMB ? cb.m0 : src;
      if (vec2 && two[u]) v[u] = *reinterpret_cast<const float2*>(s + gi[u]);
      else v[u] = make_float2(s[gi[u]], two[u] ? s[gi[u] + 1] : 0.f);
    }
    if (COMB) {
#pragma unroll 1
      for (int t = 0; t < cb.nk; t++) {
        const float* kt = cb.k[t];
        const float f = __fmul_rn(dt, cb.a[t]);
        float2 w[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (to[u] < 0) continue;
          if (vec2 && two[u]) w[u] = *reinterpret_cast<const float2*>(kt + gi[u]);
          else w[u] = make_float2(kt[gi[u]], two[u] ? kt[gi[u] + 1] : 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (to[u] < 0) continue;
          v[u].x = __fadd_rn(v[u].x, __fmul_rn(f, w[u].x));
          v[u].y = __fadd_rn(v[u].y, __fmul_rn(f, w[u].y));
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (to[u] < 0) continue;
        cb.out[gi[u]] = v[u].x;
        if (two[u]) cb.out[gi[u] + 1] = v[u].y;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (to[u] >= 0) sm[to[u]] = v[u];
  }
  __syncthreads();
  // a line of one pair has no stage to clear what lies past the data: np = M = 1 there
  const float2* x = row_stages(sm, sm + RT * pitch, z.f, nl, pitch, np);
  const int HP = M / 2 + 1;
  const Div dh(HP);
  for (int e = threadIdx.x; e < nl * HP; e += T_ROW) {
    const int l = dh(e), k = e - l * HP;
    float2 a, b;
    split_pair(x + l * pitch, k, M, z.twP, a, b);
    float2* row = dst + soff_s[l];
    row[k] = a;
    if (2 * k < M) row[M - k] = b;
  }
}

// spectrum rows -> merged (and real/imaginary exchanged) tile lines: each
// pair (X_k, X_(M-k)) is read once.  row(l): the line's spectrum.
template <typename ROW>
__device__ __forceinline__ void load_merged(float2* x, int lines, int M, int pitch, const float2* __restrict__ twP,
                                            ROW row) {
  const int HP = M / 2 + 1;
  const Div dh(HP);
  constexpr int U = 4;
  for (int e0 = threadIdx.x; e0 < lines * HP; e0 += U * T_ROW) {
    float2 a[U], b[U];
    int l[U], k[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = e0 + u * T_ROW;
      l[u] = -1;
      if (e >= lines * HP) continue;
      l[u] = dh(e);
      k[u] = e - l[u] * HP;
      const float2* s = row(l[u]);
      a[u] = s[k[u]];
      b[u] = s[M - k[u]];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (l[u] < 0) continue;
      x[l[u] * pitch + at(k[u])] = swapped(merge_pair(a[u], b[u], k[u], twP), true);
      if (k[u] > 0 && 2 * k[u] < M)
        x[l[u] * pitch + at(M - k[u])] = swapped(merge_pair(b[u], a[u], M - k[u], twP), true);
    }
  }
}

template <int = 0>
__global__ void __launch_bounds__(T_ROW) k_zc2r_mix(const float2* src, float* dst, ZPass z,
                                                    int RT) {
  extern __shared__ float2 sm[];
  __shared__ int64_t roff_s[MAX_ROWS], soff_s[MAX_ROWS];
  const int M = z.f.L, pitch = row_tile_pitch(M);
  const int r0 = blockIdx.x * RT, nl = min(RT, z.nrows - r0);
  if ((int)threadIdx.x < nl) zrow_offsets(z, r0 + threadIdx.x, &roff_s[threadIdx.x], &soff_s[threadIdx.x]);
  pass_begin();
  pass_wait();
  __syncthreads();
  load_merged(sm, nl, M, pitch, z.twP, [&](int l) { return src + soff_s[l]; });
  __syncthreads();
  const float2* x = row_stages(sm, sm + RT * pitch, z.f, nl, pitch, M);
  const Div dn(z.n_real);
  for (int e = threadIdx.x; e < nl * z.n_real; e += T_ROW) {
    const int l = dn(e), i = e - l * z.n_real;
    dst[roff_s[l] + i] = reinterpret_cast<const float*>(x + l * pitch + at(i >> 1))[1 - (i & 1)];
  }
}

// Inverse Z of the three components of RT spatial rows, the solver epilogue
// and, with FUSE (open Z boundary, N2 == M), the next forward Z.
template <int MODE, bool FUSE>
__global__ void __launch_bounds__(T_ROW, 2) k_zinv_mix(float2* S, LineFFT fz, const float2* __restrict__ twP, int P1,
                                                       int HZ, int64_t CS, int nrows, EpiArgs ea, int RT) {
  extern __shared__ float2 sm[];
  __shared__ int64_t rbase_s[MAX_ROWS];
  const int M = fz.L, pitch = row_tile_pitch(M);
  const int r0 = blockIdx.x * RT, nr = min(RT, nrows - r0), N1 = ea.N1, N2 = ea.N2;
  if ((int)threadIdx.x < nr) {
    const int gr = r0 + threadIdx.x, xp = gr / N1, yr = gr - xp * N1;
    rbase_s[threadIdx.x] = ((int64_t)xp * P1 + yr) * HZ;
  }
  pass_begin();
  pass_wait();
  __syncthreads();
  float2 *A = sm, *B = sm + 3 * RT * pitch;
  auto spec_row = [&](int l) {
    const int r = l / 3;
    return S + (l - 3 * r) * CS + rbase_s[r];
  };
  load_merged(A, 3 * nr, M, pitch, twP, spec_row);
  __syncthreads();
  float2* x = row_stages(A, B, fz, 3 * nr, pitch, M);
  float2* y = x == A ? B : A;
  float lmax = 0.f;
  double eacc = 0.0;
  const Div dn(N2);
  constexpr int C = 4;
  for (int e0 = threadIdx.x; e0 < nr * N2; e0 += C * T_ROW) {
    EpiIn<MODE, FUSE> in[C];
    int64_t g[C];
    float h[C][3];
    int to[C];
#pragma unroll
    for (int i = 0; i < C; i++) {
      const int e = e0 + i * T_ROW;
      g[i] = e < nr * N2 ? (int64_t)r0 * N2 + e : -1;
      if (g[i] < 0) continue;
      epi_load<MODE, FUSE>(ea, g[i], in[i]);
      const int r = dn(e), zz = e - r * N2;
      to[i] = 2 * (3 * r * pitch + at(zz >> 1)) + (zz & 1);
      // real and imaginary parts are still exchanged
#pragma unroll
      for (int c = 0; c < 3; c++) h[i][c] = reinterpret_cast<const float*>(x + c * pitch)[to[i] ^ 1];
    }
    epi_cells<MODE, FUSE, C>(ea, g, h, in, lmax, eacc);
    if constexpr (FUSE) {
#pragma unroll
      for (int i = 0; i < C; i++) {
        if (g[i] < 0) continue;
        // the new m, natural order; an odd row's last pair ends with a zero
#pragma unroll
        for (int c = 0; c < 3; c++) {
          float* w = reinterpret_cast<float*>(y + c * pitch) + to[i];
          w[0] = h[i][c];
          if ((N2 & 1) && (e0 + i * T_ROW) % N2 == N2 - 1) w[1] = 0.f;
        }
      }
    }
  }
  epi_flush_max<MODE>(ea, lmax, eacc);
  if constexpr (FUSE) {
    __syncthreads();
    const float2* f = row_stages(y, x, fz, 3 * nr, pitch, (N2 + 1) / 2);
    const int HP = M / 2 + 1;
    const Div dh(HP);
    for (int e = threadIdx.x; e < 3 * nr * HP; e += T_ROW) {
      const int l = dh(e), k = e - l * HP;
      float2 a, b;
      split_pair(f + l * pitch, k, M, twP, a, b);
      float2* row = spec_row(l);
      row[k] = a;
      if (2 * k < M) row[M - k] = b;
    }
  }
}

// ---------------------------------------------------------------------
// launch shapes
// ---------------------------------------------------------------------
// A kernel's opt-in is one value for the process, and launches of different
// tiles may come from several threads: it is always the largest tile's.
constexpr int TILE_MOST = 200 * 1024;
template <typename K>
static cudaError_t allow(K kern, size_t bytes) {
  if (bytes > TILE_MOST) return cudaErrorInvalidValue;
  return bytes > 40 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_MOST)
                           : cudaSuccess;
}
// widest tile (2^lg columns, at most 16 and no more than there are, fewer
// where an SM would have no tile) whose shared memory stays below a third of an SM's, but 4 columns (a 32-byte
// sector of every row) where they fit at all
static inline int pick_columns(int L, int comps, int tiles, int64_t ncols, size_t* bytes) {
  int lg = 4;
  auto need = [&](int g) { return sizeof(float2) * (size_t)tiles * L * odd_up(comps << g); };
  while (lg > 0 && (1ll << (lg - 1)) >= ncols) lg--;
  while (lg > 2 && (ncols >> lg) < mmx_sm_count()) lg--;
  while (lg > 2 && need(lg) > 72 * 1024) lg--;
  while (lg > 0 && need(lg) > TILE_MOST) lg--;
  *bytes = need(lg);
  return lg;
}
// threads of a block whose stage s has items[s] butterflies of radix[s]: the
// multiple of 32 from 128 on that leaves the fewest idle slots over all
// stages (smaller blocks waste fewer still, but the tiles then limit an SM to
// few threads: 210 x 140 x 8 grid, 280-point columns, 242 us a Heun step pair
// with 128 threads, 270 us with 64)
static inline int pick_threads(int nst, const int* items, const int* radix, int most) {
  int best = 128;
  long best_cost = -1;
  for (int t = 128; t <= most; t += 32) {
    long cost = 0;
    for (int s = 0; s < nst; s++) cost += (long)div_up(items[s], t) * t * radix[s];
    // more threads at the same cost: fewer rounds
    if (best_cost < 0 || cost <= best_cost) {
      best_cost = cost;
      best = t;
    }
  }
  return best;
}
// rows of a Z tile: about 1024 elements a component, fewer where an SM would
// have no tile, and shared memory below half an SM's
static inline int pick_rows(int M, int lines_per_row, int nrows, size_t* bytes) {
  int rt = 1024 / M < 1 ? 1 : 1024 / M > MAX_ROWS ? MAX_ROWS : 1024 / M;
  if (rt > div_up(nrows, mmx_sm_count())) rt = div_up(nrows, mmx_sm_count());
  auto need = [&](int r) { return sizeof(float2) * 2 * (size_t)r * lines_per_row * row_tile_pitch(M); };
  while (rt > 1 && need(rt) > 100 * 1024) rt--;
  *bytes = need(rt);
  return rt;
}

template <int = 0>
cudaError_t launch_col_mix(const float2* src, float2* dst, const ColPass& cp, cudaStream_t st) {
  size_t bytes;
  const int lg = pick_columns(cp.f.L, 1, cp.f.nst > 2 ? 2 : 1, (int64_t)cp.ncols * cp.nplanes, &bytes);
  cudaError_t e = allow(k_col_mix<>, bytes);
  if (e != cudaSuccess) return e;
  int items[8], radix[8];
  for (int s = 0; s < cp.f.nst; s++) {
    radix[s] = (int)((cp.f.code >> (8 * s)) & 255);
    items[s] = (cp.f.L / radix[s]) << lg;
  }
  const int t = pick_threads(cp.f.nst, items, radix, T_COL);
  return launch_pass(k_col_mix<>, div_up((int64_t)cp.ncols * cp.nplanes, 1 << lg), t, bytes, st, src, dst, cp, lg);
}
template <bool COMB>
static cudaError_t launch_zr2c_mix(const float* src, float2* dst, const ZPass& z, const ZComb& cb, cudaStream_t st) {
  size_t bytes;
  const int rt = pick_rows(z.f.L, 1, z.nrows, &bytes);
  cudaError_t e = allow(k_zr2c_mix<COMB>, bytes);
  if (e != cudaSuccess) return e;
  // 8-byte accesses when every row starts at an even float offset
  const int vec2 = z.ld_real % 2 == 0 && z.comp_stride_real % 2 == 0 && ((uintptr_t)src & 7) == 0;
  return launch_pass(k_zr2c_mix<COMB>, div_up(z.nrows, rt), T_ROW, bytes, st, src, dst, z, cb, vec2, rt);
}
template <int = 0>
cudaError_t launch_zc2r_mix(const float2* src, float* dst, const ZPass& z, cudaStream_t st) {
  size_t bytes;
  const int rt = pick_rows(z.f.L, 1, z.nrows, &bytes);
  cudaError_t e = allow(k_zc2r_mix<>, bytes);
  if (e != cudaSuccess) return e;
  return launch_pass(k_zc2r_mix<>, div_up(z.nrows, rt), T_ROW, bytes, st, src, dst, z, rt);
}

}  // namespace mix

