// Common definitions for the B200 LLG engine (libgpukern drop-in + mmx_*).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

// Error handling of the drop-in ABI follows the reference's convention:
// print and abort on any CUDA failure (src/gpukern/gpu_safe.h:36-57).
#define MMX_ABORT_ON(cond, ...)                                 \
  do {                                                          \
    if (cond) {                                                 \
      fprintf(stderr, "libgpukern(b200): " __VA_ARGS__);        \
      fprintf(stderr, "\n");                                    \
      abort();                                                  \
    }                                                           \
  } while (0)

#define GK_CHECK(call)                                                                  \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    MMX_ABORT_ON(e_ != cudaSuccess, "CUDA error %s at %s:%d", cudaGetErrorString(e_),  \
                 __FILE__, __LINE__);                                                   \
  } while (0)

// The ABI is synchronous: every entry point waits for its work
// (gpu_safe.h:41 gpu_sync after each launch).
// The reference synchronises the device after every primitive (gpu_sync,
// gpu_safe.h:40-44).  Here a drop-in primitive returns once its work is
// queued on the legacy default stream, which orders it before every later
// primitive and every cudaMemcpy of the caller; a failure surfaces, and
// aborts, at the next synchronising call (a host copy, a reduction, a free).
// MMX_GPUKERN_SYNC=1 in the environment restores a device synchronisation
// after every primitive.
bool gk_sync_each_call();
#define GK_SYNC()                                                    \
  do {                                                               \
    if (gk_sync_each_call()) GK_CHECK(cudaDeviceSynchronize());      \
  } while (0)
#define GK_LAUNCHED() GK_CHECK(cudaGetLastError())

// Status codes of the extended (mmx_*) ABI; it never aborts.
enum {
  MMX_OK = 0,
  MMX_ERR_ARG = 1,
  MMX_ERR_CUDA = 2,
  MMX_ERR_SIZE = 3,
  MMX_ERR_NAN = 4,
  MMX_ERR_MEM = 5,
  MMX_ERR_STATE = 6,
};

#define MMX_TRY(call)                          \
  do {                                         \
    cudaError_t e_ = (call);                   \
    if (e_ != cudaSuccess) {                   \
      mmx_set_error(cudaGetErrorString(e_));   \
      return MMX_ERR_CUDA;                     \
    }                                          \
  } while (0)

// Propagates a non-zero MMX_* status of an mmx_* call.
#define MMX_CHECK_RC(call)       \
  do {                           \
    int rc_ = (call);            \
    if (rc_ != 0) return rc_;    \
  } while (0)

void mmx_set_error(const char* msg);

static inline int div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Number of SMs of the current device (cached per process).
int mmx_sm_count();

// Shared memory of a block, static and dynamic together, that needs no
// opt-in, and the most that a block can have (sm_100).
constexpr size_t SMEM_FREE = 48 * 1024, SMEM_MOST = 227 * 1024;
// Opts a kernel in for a launch with DYN dynamic bytes next to its STAT static
// ones.  (The limit without opt-in is on the sum: a test of the dynamic bytes
// alone refused columns of 2048 points, 48 KB of tile + 16 KB of twiddles.)
template <size_t DYN, size_t STAT, typename K>
static cudaError_t smem_opt_in(K kern) {
  static_assert(DYN + STAT <= SMEM_MOST, "the tile does not fit an SM");
  if (DYN + STAT <= SMEM_FREE) return cudaSuccess;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DYN);
}

// ---------------------------------------------------------------------
// Programmatic dependent launch of passes that are queued one by one.  A pass
// lets its successor start at once (pass_begin) and waits for its
// predecessor's memory (pass_wait) before its first access; where the launch
// did not ask for the overlap both are no-ops.  (Waiting only after the
// twiddles are in shared memory would hide their latency too, but keeps the
// compiler from issuing the first spectrum loads before they arrive: 2% of a
// 256 x 256 x 32 Heun step.)  Every pass ends after it has waited, so a pass
// that has waited for its predecessor has waited for all before it.
// What other kernels write a pass reads by plain loads: it is resident while
// they still write, and the read-only path (__ldg, const __restrict__) is for
// data that does not change in a kernel's lifetime (twiddles, the kernel octant).
// ---------------------------------------------------------------------
__device__ __forceinline__ void pass_begin() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pass_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a pass.  On the default stream, whose launches are never part of a
// captured graph, grids that leave SMs free ask for the overlap: their time is
// launch latency and prologue (the drop-in call sequence on a 128 x 128 x 16
// grid: 328 -> 296 us a step).  Larger grids do not: the next pass's early
// blocks would take the slots of this one's last blocks.  Captured steps do
// not either: as programmatic edges of a graph the same overlap was slower
// (224 x 16 film, RKDP: 5.57 -> 6.25 ms for 45 trials).
template <typename... P, typename... A>
cudaError_t launch_pass(void (*kern)(P...), int grid, int block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = st == nullptr && grid <= mmx_sm_count() ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P(args)...);
  return e != cudaSuccess ? e : cudaGetLastError();
}
