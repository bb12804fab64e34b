// Shared host/device helpers of the ICTC B200 library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include "../../include/ictc_b200.h"

namespace ictc {

void set_error(const char* fmt, ...);

// Device address of the status word that kernels with bounded waits report through (ictc_kernel_status).
int* kernel_status_word();

// Records a CUDA launch error (if any) and maps it to the C-ABI return code.
inline int finish_launch(const char* what) {
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("%s: %s", what, cudaGetErrorString(err));
    return ICTC_ERR_LAUNCH;
  }
  return ICTC_OK;
}

// Programmatic dependent launch.  The kernels of a force sweep follow each other with a few microseconds of work each for small
// systems, so that launch latency and the ramp of the next kernel are a good part of a step.  A kernel launched with
// launch_after() may start while the previous kernel of the stream is still running; pdl_enter() then lets the next one
// start and waits until the previous one has finished and its writes are visible.  energy_and_forces
// of 216 atoms 298 -> 261 us, 10 recorded MD steps of 1,000 atoms 4.09 -> 4.02 ms (a graph's own gaps are short already).
// Rules: every thread calls pdl_enter() before its first access to global memory that an earlier launch may have written or
// still reads; a kernel that allocates tensor memory calls it behind the allocation (a later kernel's block must
// not take the columns first and then wait for this one); an ordinary load cannot be moved above the wait (the clobber), a
// non-coherent one (ldg) could be, as its memory counts as constant: its address depends on the returned zero, also in loops
// and for weights and device scalars.
__device__ __forceinline__ int pdl_enter() {
  int zero;
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero) : : "memory");
  return zero;
}
// Only for launches of about one wave: blocks that wait early take room from the running kernel's own, and a long kernel gains
// nothing (2 steps of 131,072 atoms: 51.5 ms with ordinary launches, 53.1 with every launch early).  Where the line lies
// matters little: recorded MD step with half, this and twice the limit 216 atoms 262 / 262 / 262 us, 1,000 397 / 394 / 395, 2,744
// 771 / 774 / 775, 8,000 1,817 / 1,816 / 1,813, 10,164 2,312 / 2,277 / 2,295, larger systems within the runs' spread of 1 %.
constexpr int64_t kEarlyBlocks = 148 * 8;
template <class... P, class... A>
inline void launch_if(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  if (!early) {
    kernel<<<grid, block, smem, st>>>(P(args)...);
    return;
  }
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  launch_if(int64_t(grid.x) * grid.y <= kEarlyBlocks, kernel, grid, block, smem, st, args...);
}

constexpr int kWarp = 32;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums N per-lane values over the warp with recursive halving: at every level a lane keeps half of the values and
// hands the other half to its partner, so 9 values cost 5 + 3 + 2 + 1 + 1 = 12 shuffles instead of 9 x 5.  On return
// the lane holds the total of value `idx` in `out` when `size >= 1` (exactly N lanes do); the order of the additions is
// fixed, so the result is reproducible.
template <int N, int OFF> struct WarpReduceScatter {
  static __device__ __forceinline__ void run(const float (&v)[N], int lane, int& idx, int& size, float& out) {
    constexpr int H = (N + 1) / 2;
    float w[H];
    const bool upper = (lane & OFF) != 0;
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const float hi = (H + t < N) ? v[H + t < N ? H + t : 0] : 0.f;
      const float recv = __shfl_xor_sync(0xffffffffu, upper ? v[t] : hi, OFF);
      w[t] = (upper ? hi : v[t]) + recv;
    }
    idx += upper ? H : 0;
    size = upper ? (size > H ? size - H : 0) : (size < H ? size : H);
    WarpReduceScatter<H, OFF / 2>::run(w, lane, idx, size, out);
  }
};
template <int N> struct WarpReduceScatter<N, 0> {
  static __device__ __forceinline__ void run(const float (&v)[N], int, int&, int&, float& out) { out = v[0]; }
};
template <int N> __device__ __forceinline__ float warp_reduce_scatter(const float (&v)[N], int lane, int& idx, bool& valid) {
  int size = N;
  float out;
  idx = 0;
  WarpReduceScatter<N, 16>::run(v, lane, idx, size, out);
  valid = size >= 1;
  return out;
}

// Read-only loads that go through the non-coherent path.
__device__ __forceinline__ float ldg(const float* p) { return __ldg(p); }
__device__ __forceinline__ int64_t ldg(const int64_t* p) { return __ldg(reinterpret_cast<const long long*>(p)); }

}  // namespace ictc
