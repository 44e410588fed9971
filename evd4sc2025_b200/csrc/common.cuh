// Shared device/host helpers for the B200 two-stage symmetric eigensolver.
//
// All matrices are FP64, column-major, with 64-bit leading dimensions, as in the
// reference (inc/myBase.h, api/inc/*.h).  Unlike the reference, which prints
// and exit()s on errors (inc/myBase.h:4-30), every entry point here returns an
// int status (EVD_* codes in include/evd_b200.h) and never terminates the host.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <stdio.h>

#include "../../include/evd_b200.h"

#define EVD_CUDA_TRY(call)                                                        \
  do {                                                                            \
    cudaError_t evd_err__ = (call);                                               \
    if (evd_err__ != cudaSuccess) {                                               \
      fprintf(stderr, "evd_b200: CUDA error %s at %s:%d: %s\n",                  \
              cudaGetErrorName(evd_err__), __FILE__, __LINE__,                    \
              cudaGetErrorString(evd_err__));                                     \
      return EVD_ERR_CUDA;                                                        \
    }                                                                             \
  } while (0)

// Every kernel launch site ends with EVD_LAUNCHED(): counts the launch (see
// evd_launch_count) and surfaces launch errors.
#define EVD_LAUNCHED()                          \
  do {                                          \
    ::evd::note_launch();                       \
    EVD_CUDA_TRY(cudaGetLastError());           \
  } while (0)

#define EVD_TRY(call)                          \
  do {                                         \
    int evd_st__ = (call);                     \
    if (evd_st__ != EVD_SUCCESS) return evd_st__; \
  } while (0)

namespace evd {

constexpr int kWarp = 32;

// Device-side error word written by kernels that wait on other CTAs.  A wait
// that runs out of its iteration budget records where it gave up and returns,
// so no kernel can spin forever on a shared GPU.
enum DeviceError : int {
  kDevOk = 0,
  kDevTimeoutChase = 1,
  kDevTimeoutTree = 2,
  kDevBadShape = 3,
  kDevNoConvergence = 4,
  kDevTimeoutStrips = 5,
};

// Which kernel runs a chase: the pipeline where it fits, or (for the tests, at
// orders where the pipeline would run) always the kernel with ticketed sweeps,
// or the pipeline with the gate of a cooperative launch shut from the start.
enum ChaseForm : int { kChaseAuto = 0, kChaseTicketed = 1, kChaseShut = 2 };

// The gate of a cooperative chase launch: its CTAs count themselves in, and the
// word turns to kGateShut if they do not all come in time.  Then none of them
// has touched the band, and the ticketed kernel, which every such launch is
// followed by and which else returns at once, runs the sweeps.
constexpr int kGateShut = 1 << 30;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, m));
  return v;
}

// Reductions on the tensor pipe, where the DMMA unit is otherwise idle.
// mma.m8n8k4.f64 fragments: lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4)], D[l/4][2(l%4)+1].
__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%5};\n"
      : "=d"(d0), "=d"(d1)
      : "d"(a), "d"(b), "d"(0.0), "d"(0.0));
}
// Sum over the warp, returned to every lane: quad sums s_i (A = values,
// B = ones); then B2[0][j] = s_j gives D = s_j per column, so lane l holds
// s_{2(l%4)} and s_{2(l%4)+1}; their sum u_{l%4} as A3[i][k] = u_k against
// ones adds the four u_k.
__device__ __forceinline__ double warp_sum_tc(double v) {
  const int lane = threadIdx.x & 31;
  double d0, d1;
  dmma884(d0, d1, v, 1.0);
  dmma884(d0, d1, 1.0, (lane & 3) == 0 ? d0 : 0.0);
  const double u = d0 + d1;
  dmma884(d0, d1, u, 1.0);
  return d0;
}

// Acquire/release helpers for flag-based progress between CTAs (gpu scope).
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Programmatic dependent launch: a kernel launched with launch_pdl() whose first
// statement is pdl_entry() may be brought onto the SMs while its predecessor in
// the stream drains, and starts its work when the predecessor has finished and
// its writes are visible.  The chains of short kernels (16 per panel of the
// full-to-band reduction, 11 per merge level) save about half of the launch gap.
// `trigger` false: the successor is not brought in early (kernels that fill the
// SMs, which would share them with waiting CTAs).
__device__ __forceinline__ void pdl_entry(bool trigger = true) {
  if (trigger) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

inline int ceil_div_i(long a, long b) { return (int)((a + b - 1) / b); }

// SM count of the current device (cached per device; thread-safe).
int device_sm_count();
void note_launch();

template <typename... P, typename... A>
int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
               A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  EVD_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  EVD_LAUNCHED();
  return EVD_SUCCESS;
}

// Raises `func`'s dynamic shared-memory limit to `bytes` once per (device,
// kernel); thread-safe, so host threads driving several devices or streams
// (the batched solver) may launch the same kernel concurrently.
int smem_attr_once(const void* func, int bytes);

// Reads a device error word written by a kernel (synchronises `st`) and maps
// it to an EVD_* status.
int read_device_error(const int* err_word, cudaStream_t st);

}  // namespace evd
