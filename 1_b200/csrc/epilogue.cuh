// Per-cell epilogues of the inverse-Z pass: local fields, LLG torque and
// the solver stage update, shared by the generic and the fixed-size
// kernels.  Every operation is an explicitly rounded float32 operation in
// the reference's order (see llg_ops.cuh).
#pragma once
#include "llg_ops.cuh"

// EPI_RK64: EPI_RK with the adaptive solvers' embedded error vector formed
// and normed in float64 (the precision form)
enum { EPI_FIELD = 0, EPI_HEUN1 = 1, EPI_HEUN2 = 2, EPI_TORQUE = 3, EPI_RK = 4, EPI_RK64 = 5 };
__host__ __device__ constexpr bool epi_rk(int mode) { return mode == EPI_RK || mode == EPI_RK64; }

#define RK_MAXS 7
// The combination a Runge-Kutta epilogue forms from the stage torques:
// m0 + sum_j (dt a_j) k_j over the np earlier stages with a non-zero weight
// (in stage order), then this stage's own torque (weight a_own).  Weights
// are zero where only the other combination of a pair uses the stage.
struct RKCoef {
  const float* kp[RK_MAXS - 1];  // earlier stage torques
  float a[RK_MAXS - 1];          // next stage's row of the tableau, or b for the final stage
  float b2[RK_MAXS - 1];         // lower-order weights (final stage, adaptive)
  float a_own, b2_own;
  int np;
  int adaptive;  // final stage: form the error as well and leave m_high to the controller
  int norm;      // final stage of a fixed step: out1 takes normalize(m_high)
};

struct EpiArgs {
  int N1, N2;
  int64_t n;            // cells per component
  LocalField lf;
  float alpha, dtg;
  const float* m_in;    // magnetisation at which the field was evaluated
  float* out0;
  float* out1;
  const float* aux0;
  const float* aux1;
  float* err;           // device scalar (maxabs target), may be null
  double* energy;       // RK stages: device accumulator of the total energy
                        // density sum (Relax's energy, relax.go:14-23), may be null
  const float* dt_dev;  // RK: device dt
  RKCoef rk;
};


// Per-cell inputs an epilogue reads besides the field: m at which the field
// was evaluated, and for Heun's corrector t0 and m (aux0, aux1), for an RK
// stage that forms a combination the step-start m (aux0, or m itself where
// aux0 is null).  Loaded ahead of their use so that the latencies overlap.
template <int MODE, bool NEXT>
struct EpiIn {
  static constexpr bool A0 = MODE == EPI_HEUN2 || epi_rk(MODE) || (MODE == EPI_TORQUE && NEXT);
  float m[3];
  float a0[A0 ? 3 : 1];
  float a1[MODE == EPI_HEUN2 ? 3 : 1];
};

template <int MODE, bool NEXT>
__device__ __forceinline__ void epi_load(const EpiArgs& ea, int64_t g, EpiIn<MODE, NEXT>& in) {
  const int64_t n = ea.n;
  in.m[0] = ea.m_in[g];
  in.m[1] = ea.m_in[n + g];
  in.m[2] = ea.m_in[2 * n + g];
  if constexpr (EpiIn<MODE, NEXT>::A0) {
    const float* a0 = ea.aux0;
    if (MODE == EPI_HEUN2 || a0) {
      in.a0[0] = a0[g];
      in.a0[1] = a0[n + g];
      in.a0[2] = a0[2 * n + g];
    } else {
      in.a0[0] = in.m[0];
      in.a0[1] = in.m[1];
      in.a0[2] = in.m[2];
    }
  }
  if (MODE == EPI_HEUN2) {
    in.a1[0] = ea.aux1[g];
    in.a1[1] = ea.aux1[n + g];
    in.a1[2] = ea.aux1[2 * n + g];
  }
}

// The local fields of one cell and, except for EPI_FIELD, the torque:
// (hx,hy,hz) comes in as the convolution's field and leaves as the torque.
template <int MODE>
__device__ __forceinline__ void epi_torque(const EpiArgs& ea, int64_t g, float mx, float my, float mz, float& hx,
                                           float& hy, float& hz, double& eacc) {
  llg_local(ea.lf, mx, my, mz, hx, hy, hz);
  if constexpr (epi_rk(MODE) || MODE == EPI_TORQUE) {
    // energy density of the stage's m: -1/2 m.h_conv - m.Hext - 1/2 K (m.u)^2
    // = -1/2 m.(h + Hext) with h the full field (the anisotropy terms
    // cancel), summed in float64
    if (ea.energy) {
      float s = FA(FA(FM(mx, FA(hx, ea.lf.hext[0])), FM(my, FA(hy, ea.lf.hext[1]))), FM(mz, FA(hz, ea.lf.hext[2])));
      eacc += (double)FM(-0.5f, s);
    }
    // the thermal field, added after the energy density (field.go:64-80)
    if (ea.lf.sigma != 0.f) {
      float nrm[3];
      thermal_normals(ea.lf, g, nrm);
      hx = FA(hx, FM(ea.lf.sigma, nrm[0]));
      hy = FA(hy, FM(ea.lf.sigma, nrm[1]));
      hz = FA(hz, FM(ea.lf.sigma, nrm[2]));
    }
  }
  if constexpr (MODE != EPI_FIELD) llg_delta_m(mx, my, mz, hx, hy, hz, ea.alpha, ea.dtg);
}

// The solver update of C cells of one thread: cell indices g (into one
// component), h the convolution's field, in the other inputs; cells with
// g < 0 are skipped.  With NEXT, h receives the next stage's input (Heun:
// the predicted and the corrected m; RK: the combination).
//
// An RK combination reads up to six earlier torques.  They are read stage
// by stage, all 3C values of a stage in flight together: one cell after the
// other with the stages inside, as this loop was first written, each load
// waited for the one before it (three-stage RK23 on a 512 x 512 film: final
// stage 27.7 us against 9.5 us for a stage without a combination).
template <int MODE, bool NEXT, int C>
__device__ __forceinline__ void epi_cells(const EpiArgs& ea, const int64_t (&g)[C], float (&h)[C][3],
                                          const EpiIn<MODE, NEXT> (&in)[C], float& lmax, double& eacc) {
  const int64_t n = ea.n;
#pragma unroll
  for (int i = 0; i < C; i++) {
    if (g[i] < 0) continue;
    const float mx = in[i].m[0], my = in[i].m[1], mz = in[i].m[2];
    epi_torque<MODE>(ea, g[i], mx, my, mz, h[i][0], h[i][1], h[i][2], eacc);
    if constexpr (MODE == EPI_HEUN1) {
      // t0 = torque*dt; m1est = normalize(m + t0)   (adaptive_heun.go:39-44)
      float ex = FA(mx, h[i][0]), ey = FA(my, h[i][1]), ez = FA(mz, h[i][2]);
      llg_normalize(ex, ey, ez);
#pragma unroll
      for (int c = 0; c < 3; c++) ea.out0[c * n + g[i]] = h[i][c];
      h[i][0] = ex;
      h[i][1] = ey;
      h[i][2] = ez;
#pragma unroll
      for (int c = 0; c < 3; c++) ea.out1[c * n + g[i]] = h[i][c];
    } else if constexpr (MODE == EPI_HEUN2) {
      // t = 0.5 t1 + 0.5 t0; m = normalize(m + t)   (adaptive_heun.go:46-52)
#pragma unroll
      for (int c = 0; c < 3; c++) h[i][c] = FA(in[i].a1[c], FA(FM(0.5f, h[i][c]), FM(0.5f, in[i].a0[c])));
      llg_normalize(h[i][0], h[i][1], h[i][2]);
#pragma unroll
      for (int c = 0; c < 3; c++) ea.out0[c * n + g[i]] = h[i][c];
      if (ea.err) {
        // error = maxabs(m1est - m)   (adaptive_heun.go:56-59)
#pragma unroll
        for (int c = 0; c < 3; c++) lmax = fmaxf(lmax, fabsf(FA(in[i].m[c], FM(-1.f, h[i][c]))));
      }
    } else {
      // the field (EPI_FIELD) or the stage torque
      if (ea.out0) {
#pragma unroll
        for (int c = 0; c < 3; c++) ea.out0[c * n + g[i]] = h[i][c];
      }
      if (MODE == EPI_TORQUE && ea.err) {
#pragma unroll
        for (int c = 0; c < 3; c++) lmax = fmaxf(lmax, fabsf(h[i][c]));
      }
    }
  }
  if constexpr (epi_rk(MODE) || (MODE == EPI_TORQUE && NEXT)) {
    const float dt = *ea.dt_dev;
    const bool low = MODE == EPI_RK && ea.rk.adaptive;
    const bool low64 = MODE == EPI_RK64 && ea.rk.adaptive;
    float q[C][3], lo[MODE == EPI_RK ? C : 1][3];
    double e64[MODE == EPI_RK64 ? C : 1][3];
#pragma unroll
    for (int i = 0; i < C; i++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        q[i][c] = in[i].a0[c];
        if constexpr (MODE == EPI_RK) lo[i][c] = in[i].a0[c];
        if constexpr (MODE == EPI_RK64) e64[i][c] = 0.0;
      }
    }
    auto add = [&](int i, int c, float a, float b, float k) {
      if (a != 0.f) q[i][c] = FA(q[i][c], FM(FM(dt, a), k));
      if constexpr (MODE == EPI_RK) {
        if (low && b != 0.f) lo[i][c] = FA(lo[i][c], FM(FM(b, dt), k));
      }
      if constexpr (MODE == EPI_RK64) {
        // the embedded error vector sum_j (b_j - b*_j) dt k_j formed and
        // normed in float64 from the float32 stage torques
        const double w = ((double)a - (double)b) * (double)dt;
        if (low64 && w != 0.0) e64[i][c] = fma(w, (double)k, e64[i][c]);
      }
    };
    const int np = ea.rk.np;
#pragma unroll 1
    for (int j = 0; j < np; j++) {
      const float* kj = ea.rk.kp[j];
      const float a = ea.rk.a[j], b = ea.rk.b2[j];
      float v[C][3];
#pragma unroll
      for (int i = 0; i < C; i++)
#pragma unroll
        for (int c = 0; c < 3; c++) v[i][c] = g[i] >= 0 ? kj[c * n + g[i]] : 0.f;
#pragma unroll
      for (int i = 0; i < C; i++)
#pragma unroll
        for (int c = 0; c < 3; c++) add(i, c, a, b, v[i][c]);
    }
#pragma unroll
    for (int i = 0; i < C; i++) {
      if (g[i] < 0) continue;
#pragma unroll
      for (int c = 0; c < 3; c++) add(i, c, ea.rk.a_own, ea.rk.b2_own, h[i][c]);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if constexpr (MODE == EPI_RK) {
          if (low) lmax = fmaxf(lmax, fabsf(FA(lo[i][c], FM(-1.f, q[i][c]))));
        }
        if constexpr (MODE == EPI_RK64) {
          if (low64) lmax = fmaxf(lmax, (float)fabs(e64[i][c]));
        }
      }
      if (epi_rk(MODE) && ea.rk.norm) llg_normalize(q[i][0], q[i][1], q[i][2]);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ea.out1[c * n + g[i]] = q[i][c];
        h[i][c] = q[i][c];
      }
    }
  }
}

// block-wide maximum of lmax into *ea.err (non-negative float atomics) and,
// for RK stages, the warp sums of the energy density into *ea.energy
template <int MODE>
__device__ __forceinline__ void epi_flush_max(const EpiArgs& ea, float lmax, double eacc = 0.0) {
  if ((MODE == EPI_HEUN2 || epi_rk(MODE) || MODE == EPI_TORQUE) && ea.err) {
    for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(ea.err, lmax);
  }
  if constexpr (epi_rk(MODE) || MODE == EPI_TORQUE) {
    if (ea.energy) {
      for (int o = 16; o > 0; o >>= 1) eacc += __shfl_xor_sync(0xffffffffu, eacc, o);
      if ((threadIdx.x & 31) == 0) atomicAdd(ea.energy, eacc);
    }
  }
}
