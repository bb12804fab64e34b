// Prefix sums in one launch.
//
// A block owns a tile of kPrefixTile values and first adds up everything before its tile by itself, instead of waiting
// for the other blocks' totals: the values are 4 or 8 bytes and come from L2, so up to kPrefixDirect tiles this costs
// less than the two or three launches of a tiled scan.  Longer inputs get their tile totals from a first pass.
#pragma once
#include "ictc_common.cuh"

namespace ictc {

constexpr int kPrefixThreads = 512;
constexpr int kPrefixItems = 4;
constexpr int kPrefixTile = kPrefixThreads * kPrefixItems;   // 2048 values per block
constexpr int kPrefixDirect = 8;

template <class T> __device__ __forceinline__ T block_sum(T v, T* warp_tot) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = v;
  __syncthreads();
  T s = 0;
#pragma unroll
  for (int w = 0; w < kPrefixThreads / 32; ++w) s += warp_tot[w];
  __syncthreads();
  return s;
}

template <class T, class LOAD>
__global__ void __launch_bounds__(kPrefixThreads) tile_sum_kernel(int64_t n, LOAD load, T* sums) {
  __shared__ T warp_tot[kPrefixThreads / 32];
  const int64_t base = int64_t(blockIdx.x) * kPrefixTile + pdl_enter();
  T v = 0;
#pragma unroll
  for (int k = 0; k < kPrefixItems; ++k) {
    const int64_t i = base + k * kPrefixThreads + threadIdx.x;
    if (i < n) v += load(i);
  }
  v = block_sum(v, warp_tot);
  if (threadIdx.x == 0) sums[blockIdx.y * gridDim.x + blockIdx.x] = v;
}

// blockIdx.y numbers independent inputs of the same length; the functors look it up themselves.
// store(i, sum of the values before i, value i) for every i < n.  `sums`: totals of the tiles, or null: the values
// before the tile are read again (then `load` must not read what `store` writes).
template <class T, class LOAD, class STORE>
__global__ void __launch_bounds__(kPrefixThreads) prefix_kernel(int64_t n, LOAD load, STORE store, const T* sums) {
  __shared__ T warp_tot[kPrefixThreads / 32];
  const int64_t base = int64_t(blockIdx.x) * kPrefixTile + pdl_enter();
  T before = 0;
  if (sums) {
    for (int64_t i = threadIdx.x; i < blockIdx.x; i += kPrefixThreads) before += sums[blockIdx.y * gridDim.x + i];
  } else {
    for (int64_t i = threadIdx.x; i < base; i += kPrefixThreads) before += load(i);
  }
  before = block_sum(before, warp_tot);
  T v[kPrefixItems], run = 0;
#pragma unroll
  for (int k = 0; k < kPrefixItems; ++k) {
    const int64_t i = base + int64_t(threadIdx.x) * kPrefixItems + k;
    v[k] = i < n ? load(i) : T(0);
    run += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T up = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += up;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  T at = before + inc - run;
  for (int w = 0; w < warp; ++w) at += warp_tot[w];
#pragma unroll
  for (int k = 0; k < kPrefixItems; ++k) {
    const int64_t i = base + int64_t(threadIdx.x) * kPrefixItems + k;
    if (i < n) store(i, at, v[k]);
    at += v[k];
  }
}

inline int64_t prefix_tiles(int64_t n) { return n > 0 ? (n + kPrefixTile - 1) / kPrefixTile : 0; }

// `in_place`: store() writes where load() reads; `sums`: inputs * prefix_tiles(n) values of scratch.
template <class T, class LOAD, class STORE>
void prefix_sum(int64_t n, LOAD load, STORE store, T* sums, bool in_place, cudaStream_t st, int inputs = 1) {
  const int64_t tiles = prefix_tiles(n);
  if (tiles == 0) return;
  const bool two = tiles > kPrefixDirect || (in_place && tiles > 1);
  const dim3 grid((unsigned)tiles, (unsigned)inputs);
  if (two) launch_after(tile_sum_kernel<T, LOAD>, grid, kPrefixThreads, 0, st, n, load, sums);
  launch_after(prefix_kernel<T, LOAD, STORE>, grid, kPrefixThreads, 0, st, n, load, store, two ? (const T*)sums : (const T*)nullptr);
}

}  // namespace ictc
