// First layer of the radial MLP in training: a bias-free linear map from 8 radial functions to 64 hidden units over the
// rows of an edge list, its input gradient and its weight gradient (reference: F.linear in the `fc` stack,
// mace_ictc/models/mace/layers.py:825-835, and its autograd).
//
// With 8 columns on one side there is nothing for a matrix unit or a tiled GEMM to hold on to: the maps are bound by the
// 64-wide rows, 256 bytes each way.  16 threads share a row, four units each (16-byte accesses, whole lines per warp), and keep
// their part of the weights or of the weight gradient in registers.  The weight gradient adds its rows per thread,
// per block and over the blocks in a fixed order.  Training step of 32,768 atoms, with the
// library's GEMMs before: 51.4 -> 49.5 ms.
#include "ictc_common.cuh"

namespace ictc {
namespace narrow {

constexpr int kIn = 8, kOut = 64, kThreads = 256, kRowsPerBlock = kThreads / 16;
constexpr int64_t kMaxBlocks = 148 * 8, kGradBlocks = 148 * 4;
constexpr int kSlices = 16, kColumns = 32;      // threads of the second stage

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// y[r, n] = sum_k x[r, k] w[n, k]
__global__ void __launch_bounds__(kThreads) forward_kernel(int64_t R, const float* __restrict__ x, const float* __restrict__ w, float* y) {
  const int q = threadIdx.x & 15;
  float m[4][kIn];
#pragma unroll
  for (int j = 0; j < 4; ++j) load8(w + (4 * q + j) * kIn, m[j]);
  for (int64_t r = int64_t(blockIdx.x) * kRowsPerBlock + (threadIdx.x >> 4); r < R; r += int64_t(gridDim.x) * kRowsPerBlock) {
    float v[kIn], s[4];
    load8(x + r * kIn, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = v[0] * m[j][0];
#pragma unroll
      for (int k = 1; k < kIn; ++k) s[j] = fmaf(v[k], m[j][k], s[j]);
    }
    reinterpret_cast<float4*>(y + r * kOut)[q] = make_float4(s[0], s[1], s[2], s[3]);
  }
}

// dx[r, k] = sum_n g[r, n] w[n, k]; the loop runs to the block's last row for every thread (shuffles)
__global__ void __launch_bounds__(kThreads) input_grad_kernel(int64_t R, const float* __restrict__ g, const float* __restrict__ w, float* dx) {
  const int lane = threadIdx.x & 31, q = lane & 15;
  float m[4][kIn];
#pragma unroll
  for (int j = 0; j < 4; ++j) load8(w + (4 * q + j) * kIn, m[j]);
  for (int64_t r0 = int64_t(blockIdx.x) * kRowsPerBlock; r0 < R; r0 += int64_t(gridDim.x) * kRowsPerBlock) {
    const int64_t r = r0 + (threadIdx.x >> 4);
    const float4 v = r < R ? __ldg(reinterpret_cast<const float4*>(g + r * kOut) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    float s[kIn];
#pragma unroll
    for (int k = 0; k < kIn; ++k) s[k] = fmaf(v.w, m[3][k], fmaf(v.z, m[2][k], fmaf(v.y, m[1][k], v.x * m[0][k])));
    // sums over the row's 16 threads: every step halves the values a thread is responsible for
#pragma unroll
    for (int half = 4, bit = 8; half > 0; half >>= 1, bit >>= 1) {
      const bool upper = (lane & bit) != 0;
#pragma unroll
      for (int k = 0; k < half; ++k) {
        const float other = __shfl_xor_sync(0xffffffffu, upper ? s[k] : s[half + k], bit);
        s[k] = (upper ? s[half + k] : s[k]) + other;
      }
    }
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
    if (r < R && (lane & 1) == 0) dx[r * kIn + ((lane >> 1) & 7)] = s[0];
  }
}

// dw[n, k] = sum_r g[r, n] x[r, k], first stage: one partial sum per block
__global__ void __launch_bounds__(kThreads) weight_grad_kernel(int64_t R, const float* __restrict__ g, const float* __restrict__ x, float* partial) {
  __shared__ float sums[kRowsPerBlock][kOut * kIn];
  const int q = threadIdx.x & 15, group = threadIdx.x >> 4;
  float acc[4][kIn];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < kIn; ++k) acc[j][k] = 0.f;
#pragma unroll 2
  for (int64_t r = int64_t(blockIdx.x) * kRowsPerBlock + group; r < R; r += int64_t(gridDim.x) * kRowsPerBlock) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(g + r * kOut) + q);
    float u[kIn];
    load8(x + r * kIn, u);
#pragma unroll
    for (int k = 0; k < kIn; ++k) {
      acc[0][k] = fmaf(v.x, u[k], acc[0][k]);
      acc[1][k] = fmaf(v.y, u[k], acc[1][k]);
      acc[2][k] = fmaf(v.z, u[k], acc[2][k]);
      acc[3][k] = fmaf(v.w, u[k], acc[3][k]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < kIn; ++k) sums[group][(4 * q + j) * kIn + k] = acc[j][k];
  __syncthreads();
  for (int i = threadIdx.x; i < kOut * kIn; i += kThreads) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kRowsPerBlock; ++k) s += sums[k][i];
    partial[int64_t(blockIdx.x) * (kOut * kIn) + i] = s;
  }
}

__global__ void __launch_bounds__(kSlices * kColumns) weight_sum_kernel(const float* __restrict__ partial, int blocks, float* dw) {
  __shared__ float sums[kSlices][kColumns];
  const int c = threadIdx.x % kColumns, slice = threadIdx.x / kColumns, i = blockIdx.x * kColumns + c;
  float s = 0.f;
#pragma unroll 4
  for (int b = slice; b < blocks; b += kSlices) s += __ldg(partial + int64_t(b) * (kOut * kIn) + i);
  sums[slice][c] = s;
  __syncthreads();
  if (slice) return;
  s = 0.f;
#pragma unroll
  for (int k = 0; k < kSlices; ++k) s += sums[k][c];
  dw[i] = s;
}

static int64_t grad_blocks(int64_t R) {
  const int64_t b = (R + 8 * kRowsPerBlock - 1) / (8 * kRowsPerBlock);       // at least eight rows to a thread
  return b < 1 ? 1 : (b < kGradBlocks ? b : kGradBlocks);
}

static int check(int64_t R, const void* a, const void* b, const void* c) {
  if (R < 0 || !a || !b || !c) { set_error("narrow linear: invalid arguments"); return ICTC_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) {
    set_error("narrow linear: buffers must be 16-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  return ICTC_OK;
}
static unsigned row_blocks(int64_t R) {
  const int64_t b = (R + kRowsPerBlock - 1) / kRowsPerBlock;
  return unsigned(b < kMaxBlocks ? b : kMaxBlocks);
}

}  // namespace narrow
}  // namespace ictc

using namespace ictc;

extern "C" {

int ictc_narrow_linear_forward(int64_t rows, const float* x, const float* w, float* y, void* stream) {
  if (rows == 0) return ICTC_OK;
  if (int rc = narrow::check(rows, x, w, y)) return rc;
  narrow::forward_kernel<<<narrow::row_blocks(rows), narrow::kThreads, 0, (cudaStream_t)stream>>>(rows, x, w, y);
  return finish_launch("narrow_linear_forward");
}

int ictc_narrow_linear_input_grad(int64_t rows, const float* g, const float* w, float* dx, void* stream) {
  if (rows == 0) return ICTC_OK;
  if (int rc = narrow::check(rows, g, w, dx)) return rc;
  narrow::input_grad_kernel<<<narrow::row_blocks(rows), narrow::kThreads, 0, (cudaStream_t)stream>>>(rows, g, w, dx);
  return finish_launch("narrow_linear_input_grad");
}

int64_t ictc_narrow_linear_workspace(int64_t rows) { return 4 * narrow::grad_blocks(rows) * narrow::kOut * narrow::kIn; }

int ictc_narrow_linear_weight_grad(int64_t rows, const float* g, const float* x, float* dw, float* workspace, void* stream) {
  if (int rc = narrow::check(rows, g, x, dw)) return rc;
  if (!workspace) { set_error("narrow linear: NULL workspace"); return ICTC_ERR_BAD_ARG; }
  const int blocks = int(narrow::grad_blocks(rows));
  narrow::weight_grad_kernel<<<blocks, narrow::kThreads, 0, (cudaStream_t)stream>>>(rows, g, x, workspace);
  narrow::weight_sum_kernel<<<narrow::kOut * narrow::kIn / narrow::kColumns, narrow::kSlices * narrow::kColumns, 0,
                              (cudaStream_t)stream>>>(workspace, blocks, dw);
  return finish_launch("narrow_linear_weight_grad");
}

}  // extern "C"
