// Demagnetising kernel generation on the GPU.
//
// Restates FaceKernel6 / faceIntegral (src/go/sim/demag.go:26-84,
// 142-183) and Exch6NgbrKernel (src/go/sim/exchange.go:44-71) with the
// same float32 operations in the same order, so the real-space kernel is
// bit-identical to the one the reference's Go subprocess computes
// (mumaxkern-go, src/go/kernel-main/main.go:43): every product, sum,
// quotient and square root is an explicitly rounded IEEE float32
// operation (no contraction into fused multiply-adds).  The square root
// of the Go code is taken in float64 and rounded, which equals the
// correctly rounded float32 square root.
#pragma once
#include "mmx_common.cuh"

// Field at R of the two charged faces, n x n point charges each, of a cell
// magnetised along S; only the components d >= S that the symmetric kernel
// keeps.  Bound by the square roots and divisions of its 2 n^2 charges a
// point.  With the axis a template parameter the displacements stay in
// registers (a run-time axis indexed local memory), differences and squares
// that a row of charges shares are formed once, 1/r is one rounded
// reciprocal, and sc = +-(charge / den).  Every value is rounded as in the Go
// code: differences, products, the sum of squares in the order x, y, z,
// then the quotients, products and sums.
template <int S>
__device__ __forceinline__ void fk_face_integral(float (&B)[3], const float R[3], const float cs[3], int n) {
  constexpr int U = S, V = (S + 1) % 3, W = (S + 2) % 3;
  const float charge = __fmul_rn(cs[V], cs[W]);
  const float pu1 = __fdiv_rn(cs[U], 2.f);
  const float four_pi = 12.566370614359172f;
  const float tv0 = __fadd_rn(-__fdiv_rn(cs[V], 2.f), __fdiv_rn(cs[V], (float)(2 * n)));
  const float tv1 = __fdiv_rn(cs[V], (float)n);
  const float tw0 = __fadd_rn(-__fdiv_rn(cs[W], 2.f), __fdiv_rn(cs[W], (float)(2 * n)));
  const float tw1 = __fdiv_rn(cs[W], (float)n);
  const float du[2] = {__fsub_rn(R[U], pu1), __fsub_rn(R[U], -pu1)};
  const float qu[2] = {__fmul_rn(du[0], du[0]), __fmul_rn(du[1], du[1])};
  B[0] = B[1] = B[2] = 0.f;
  for (int i = 0; i < n; i++) {
    const float dv = __fsub_rn(R[V], __fadd_rn(tv0, __fmul_rn((float)i, tv1)));
    const float qv = __fmul_rn(dv, dv);
#pragma unroll 4
    for (int j = 0; j < n; j++) {
      const float dw = __fsub_rn(R[W], __fadd_rn(tw0, __fmul_rn((float)j, tw1)));
      const float qw = __fmul_rn(dw, dw);
#pragma unroll
      for (int side = 0; side < 2; side++) {
        // squares in the order of the axes 0, 1, 2
        float q[3], R2[3];
        q[U] = qu[side];
        q[V] = qv;
        q[W] = qw;
        R2[U] = du[side];
        R2[V] = dv;
        R2[W] = dw;
        const float r = __fsqrt_rn(__fadd_rn(__fadd_rn(q[0], q[1]), q[2]));
        const float inv = __frcp_rn(r);
        const float quot = __fdiv_rn(charge, __fmul_rn(__fmul_rn(four_pi, r), r));
        const float sc = side == 0 ? quot : -quot;
#pragma unroll
        for (int d = S; d < 3; d++) B[d] = __fadd_rn(B[d], __fmul_rn(__fmul_rn(R2[d], inv), sc));
      }
    }
  }
  const float fin = __fdiv_rn(1.f, (float)(n * n));
#pragma unroll
  for (int d = S; d < 3; d++) B[d] = __fmul_rn(B[d], fin);
}

struct FaceKernelArgs {
  int P[3];
  int periodic[3];
  float cs[3];
  int accuracy;
  int lo[3], hi[3];  // loop bounds of demag.go:136-154 (after periodic scaling)
};

// One thread per wrapped output cell; images are accumulated in the Go
// loop order (x, then y, then z, ascending).
__global__ void k_face_kernel6(float* __restrict__ k6, FaceKernelArgs a) {
  const int64_t n3 = (int64_t)a.P[0] * a.P[1] * a.P[2];
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n3;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int zw = (int)(idx % a.P[2]);
    int yw = (int)((idx / a.P[2]) % a.P[1]);
    int xw = (int)(idx / ((int64_t)a.P[2] * a.P[1]));
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // smallest image >= lo in each dimension
    int x0 = xw;
    while (x0 - a.P[0] >= a.lo[0]) x0 -= a.P[0];
    while (x0 < a.lo[0]) x0 += a.P[0];
    int y0 = yw;
    while (y0 - a.P[1] >= a.lo[1]) y0 -= a.P[1];
    while (y0 < a.lo[1]) y0 += a.P[1];
    int z0 = zw;
    while (z0 - a.P[2] >= a.lo[2]) z0 -= a.P[2];
    while (z0 < a.lo[2]) z0 += a.P[2];
    // one component of magnetisation after the other, each over all images
    auto images = [&](auto add) {
      for (int x = x0; x <= a.hi[0]; x += a.P[0])
        for (int y = y0; y <= a.hi[1]; y += a.P[1])
          for (int z = z0; z <= a.hi[2]; z += a.P[2]) {
            const float R[3] = {__fmul_rn((float)x, a.cs[0]), __fmul_rn((float)y, a.cs[1]),
                                __fmul_rn((float)z, a.cs[2])};
            add(R);
          }
    };
    // KernIdx (kernel.go:95-98): order XX,YY,ZZ,YZ,XZ,XY
    images([&](const float* R) {
      float B[3];
      fk_face_integral<0>(B, R, a.cs, a.accuracy);
      acc[0] = __fadd_rn(acc[0], B[0]);
      acc[5] = __fadd_rn(acc[5], B[1]);
      acc[4] = __fadd_rn(acc[4], B[2]);
    });
    images([&](const float* R) {
      float B[3];
      fk_face_integral<1>(B, R, a.cs, a.accuracy);
      acc[1] = __fadd_rn(acc[1], B[1]);
      acc[3] = __fadd_rn(acc[3], B[2]);
    });
    images([&](const float* R) {
      float B[3];
      fk_face_integral<2>(B, R, a.cs, a.accuracy);
      acc[2] = __fadd_rn(acc[2], B[2]);
    });
#pragma unroll
    for (int c = 0; c < 6; c++) k6[c * n3 + idx] = acc[c];
  }
}

// Exch6NgbrKernel folded into the diagonal components (init.go:256-267).
// The seven stencil cells are written in Go's order so that, when two
// wrap onto the same cell (a dimension of size 1 or 2), the last write
// wins, as in exchange.go:58-65; the tensor is then added.
__global__ void k_add_exch6(float* __restrict__ k6, int P0, int P1, int P2, float c0, float c1, float c2) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int64_t n3 = (int64_t)P0 * P1 * P2;
  float hx = __fmul_rn(c0, c0), hy = __fmul_rn(c1, c1), hz = __fmul_rn(c2, c2);
  float cc = __fsub_rn(__fsub_rn(__fdiv_rn(-2.f, hx), __fdiv_rn(2.f, hy)), __fdiv_rn(2.f, hz));
  const int cell[7][3] = {{0, 0, 0}, {1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
  float val[7] = {cc, __fdiv_rn(1.f, hx), __fdiv_rn(1.f, hx), __fdiv_rn(1.f, hy), __fdiv_rn(1.f, hy),
                  __fdiv_rn(1.f, hz), __fdiv_rn(1.f, hz)};
  const int P[3] = {P0, P1, P2};
  int64_t idx[7];
  float ev[7];
  int ne = 0;
  for (int c = 0; c < 7; c++) {
    int w[3];
    for (int d = 0; d < 3; d++) {
      int t = cell[c][d];
      while (t < 0) t += P[d];
      while (t >= P[d]) t -= P[d];
      w[d] = t;
    }
    int64_t id = ((int64_t)w[0] * P1 + w[1]) * P2 + w[2];
    int f = -1;
    for (int q = 0; q < ne; q++)
      if (idx[q] == id) f = q;
    if (f >= 0) ev[f] = val[c];
    else { idx[ne] = id; ev[ne] = val[c]; ne++; }
  }
  for (int comp = 0; comp < 3; comp++)
    for (int q = 0; q < ne; q++) k6[comp * n3 + idx[q]] = __fadd_rn(k6[comp * n3 + idx[q]], ev[q]);
}
