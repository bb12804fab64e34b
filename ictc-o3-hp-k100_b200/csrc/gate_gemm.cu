// Wide last layer of the radial gate MLP on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   forward :  gates[r, :] = act(z3[r, :]) @ W3^T            K = 64,    N = P*C (192 or 704)
//   backward:  da3[r, :]   = (dG[a(r), :] + dG[b(r), :]) @ W3   K = P*C,  N = 64
//
// Reference: last `F.linear` of the interaction block's radial stack (mace_ictc/models/mace/layers.py:825-835),
// tiled per edge chunk by ictc_o3/ops/streamed_gate_message.py:112-116, and its input gradient
// (streamed_gate_message.py:224-260).  The reference forbids TF32 (ictc_o3/backends/k100/fp32_policy.py:6-11),
// so every operand is split into two TF32-representable parts, x = x_big + x_small, and a product is the sum of
// the three tcgen05.mma passes big*big + big*small + small*big into one fp32 TMEM accumulator.
//
// One persistent CTA per SM works on tiles of 128 rows.
// A launch covers up to three matrices (segments): the three degree blocks of a channel linear, one launch instead of
// three.  Warp roles:
//   warp 0      streams pre-packed 64-unit weight chunks (32 KB: big and small part) into a 4-stage ring
//               with cp.async.bulk, completing on mbarriers; a segment with a single chunk keeps it;
//   warp 1      allocates TMEM and issues the MMAs (one thread), committing to mbarriers;
//   warps 2-9   (backward: 2-5) epilogue, in the forward kernel two groups taking alternate blocks:
//               tcgen05.ld (thread = row), then coalesced row stores;
//   last eight  A-operand producers: global rows -> (activation | pair sum) -> split -> tcgen05.st into TMEM
//               (the A operand is read from TMEM: lane = row, column = k; no shared memory for A at all).
// Shared-memory layout of the B operand: element (n, k) of a [64 x 64] part lives at byte
// (k / 4) * 1024 + n * 16 + (k % 4) * 4, i.e. 16-byte K chunks, each chunk row-contiguous (canonical K-major
// no-swizzle layout).  In descriptor terms: 8-row core matrices of 128 contiguous bytes, stride between core
// matrices along n (SBO) 128 B, stride between the two K chunks of one K = 8 MMA (LBO) 1024 B.
// Every mbarrier wait is bounded; a wait that runs out raises the library's status word and the CTA leaves
// through the common exit (TMEM is always released).
#include "gate_gemm.cuh"

namespace ictc {
namespace gg {

using namespace tc;

constexpr int kFwdThreads = 18 * 32, kBwdThreads = 14 * 32;      // up to 16 warps leave 128 registers to a thread, 18 leave 96
constexpr int kProducerWarps = 8, kFwdProducer0 = 10, kBwdProducer0 = 6;
constexpr int kStagePitch = 272;                    // bytes per staged output row (256 + 16: conflict-free)

__device__ __forceinline__ int64_t row_offset(int64_t g, int mm, int64_t ld) {
  if (mm == 1) return g * ld;
  const int64_t node = g / mm;
  return node * ld + (g - node * mm) * kK;
}

constexpr int kWStages = 4;      // weight ring
constexpr int kAStagesBwd = 3;   // A ring of the backward kernel

struct Barriers {
  unsigned long long w_full[kWStages], w_empty[kWStages], a_full[4], a_empty[4], d_full[4], d_empty[4];
  unsigned tmem_base;
  volatile int failed;   // polled inside wait loops by other warps: every read must go to shared memory
};

// The tiles of a launch, segment after segment, dealt out round robin over the CTAs.  Every warp role walks the same tiles
// in the same order.
struct Work {
  int64_t base, live;        // first list entry, bound of the live rows
  int end0, end1, end2;      // running totals of tiles

  __device__ Work(const Args& a, int zero) {
    base = a.begin ? ldg(a.begin + zero) : zero;
    live = a.limit ? ldg(a.limit + zero) - base : a.seg[0].rows + a.seg[1].rows + a.seg[2].rows;
    if (live < 0) live = 0;
    end0 = int((rows(a, 0) + kRows - 1) / kRows);
    end1 = end0 + (a.segments > 1 ? int((rows(a, 1) + kRows - 1) / kRows) : 0);
    end2 = end1 + (a.segments > 2 ? int((rows(a, 2) + kRows - 1) / kRows) : 0);
  }
  __device__ int64_t rows(const Args& a, int s) const { return live < a.seg[s].rows ? live : a.seg[s].rows; }
  __device__ int segment(int tile) const { return (tile >= end0) + (tile >= end1); }
  __device__ int tiles() const { return end2; }
  __device__ int64_t first_row(int tile, int s) const {
    return int64_t(tile - (s == 0 ? 0 : s == 1 ? end0 : end1)) * kRows;
  }
};

__device__ __forceinline__ void give_up(Barriers* b, int* status, int code) {
  b->failed = 1;
  if (status) atomicExch(status, code);
}

// The weight stream of both kernels: chunk after chunk for every tile.  A segment with one chunk keeps it.  When the block has given
// up, the copies in flight are waited for (again with a limit) before the lane leaves.
__device__ __forceinline__ void stream_weights(const Args& a, const Work& work, Barriers* bar, unsigned char* w_buf, int code) {
  int64_t it = 0;
  int kept = -1;
  for (int tile = blockIdx.x; tile < work.tiles() && !bar->failed; tile += gridDim.x) {
    const int s = work.segment(tile);
    const Segment& seg = a.seg[s];
    if (s == kept) continue;
    for (int c = 0; c < seg.chunks && !bar->failed; ++c) {
      const int slot = int(it % kWStages);
      if (!mbar_wait(saddr(&bar->w_empty[slot]), unsigned((it / kWStages) & 1) ^ 1u)) { give_up(bar, a.status, code); break; }
      mbar_expect_tx(saddr(&bar->w_full[slot]), kWStageBytes);
      bulk_g2s(saddr(w_buf + slot * kWStageBytes), seg.w + int64_t(c) * (kWStageBytes / 4), kWStageBytes,
               saddr(&bar->w_full[slot]));
      ++it;
    }
    kept = seg.chunks == 1 ? s : -1;
  }
  if (bar->failed)
    for (int64_t k = it > kWStages ? it - kWStages : 0; k < it; ++k)
      mbar_wait(saddr(&bar->w_full[k % kWStages]), unsigned((k / kWStages) & 1));
}

// Barriers and all 512 TMEM columns; returns the TMEM base.
__device__ __forceinline__ unsigned enter(Barriers* bar, int a_stages, int accumulators) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < kWStages; ++i) {
      mbar_init(saddr(&bar->w_full[i]), 1);
      mbar_init(saddr(&bar->w_empty[i]), 1);
    }
    for (int i = 0; i < a_stages; ++i) {
      mbar_init(saddr(&bar->a_full[i]), kProducerWarps * 32);
      mbar_init(saddr(&bar->a_empty[i]), 1);
    }
    for (int i = 0; i < accumulators; ++i) {
      mbar_init(saddr(&bar->d_full[i]), 1);
      mbar_init(saddr(&bar->d_empty[i]), 128);
    }
    bar->failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if ((threadIdx.x >> 5) == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&bar->tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return __shfl_sync(0xffffffffu, bar->tmem_base, 0);
}

__device__ __forceinline__ void leave(unsigned tmem) {
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------
// forward.  Shared memory: W ring (4 x 32 KB) | output staging (2 x 34 KB) | row offsets (2 x 1 KB) | barriers.
// TMEM (512 columns): accumulator ring 4 x 64 | A operand of two tiles, each big (64) + small (64).
// Two tiles per weight chunk (half the weight traffic from L2, two accumulators in the ring) was measured slower: 1 M rows
// of 704 in 0.73 against 0.53 ms; the writes leave at 5.8 TB/s now (0.62 ms before the MMAs were issued by an elected lane).
constexpr int kFwdSmem = kWStages * kWStageBytes + 2 * kRows * (kStagePitch + 8) + 256;

__global__ void __launch_bounds__(kFwdThreads, 1) gate_gemm_forward_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(128) unsigned char gg_smem[];
  unsigned char* w_buf = gg_smem;
  unsigned char* stage = w_buf + kWStages * kWStageBytes;
  int64_t* offsets = reinterpret_cast<int64_t*>(stage + 2 * kRows * kStagePitch);
  Barriers* bar = reinterpret_cast<Barriers*>(offsets + 2 * kRows);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned tmem = enter(bar, 2, 4);
  const int zero = pdl_enter();
  const Work work(a, zero);
  const unsigned tmem_a = tmem + 4 * kChunk;       // A operands start after the accumulator ring

  if (warp == 0) {
    if (lane == 0) stream_weights(a, work, bar, w_buf, 21);
  } else if (warp == 1) {
    if (elect_one()) {           // ---- MMA issue: the role of one lane, its waits included
      int64_t it = 0, wit = 0;
      int t = 0, kept = -1;
      bool ok = true;
      for (int tile = blockIdx.x; tile < work.tiles() && ok && !bar->failed; tile += gridDim.x, ++t) {
        const int s = work.segment(tile), chunks = a.seg[s].chunks;
        const bool keep = chunks == 1 && tile + int(gridDim.x) < work.tiles() && work.segment(tile + gridDim.x) == s;
        const int ab = t & 1;
        if (!mbar_wait(saddr(&bar->a_full[ab]), unsigned((t >> 1) & 1))) { give_up(bar, a.status, 22); break; }
        for (int c = 0; c < chunks; ++c, ++it) {
          const int slot = int(wit % kWStages), d = int(it & 3);
          if ((kept != s && !mbar_wait(saddr(&bar->w_full[slot]), unsigned((wit / kWStages) & 1))) ||
              !mbar_wait(saddr(&bar->d_empty[d]), unsigned((it >> 2) & 1) ^ 1u)) {
            give_up(bar, a.status, 23);
            ok = false;
            break;
          }
          tc_fence_after();
          const unsigned w_big = saddr(w_buf + slot * kWStageBytes), w_small = w_big + kWPartBytes;
          issue_block(tmem + d * kChunk, tmem_a + ab * 2 * kK, w_big, w_small, true);
          if (!keep) umma_commit(saddr(&bar->w_empty[slot]));
          umma_commit(saddr(&bar->d_full[d]));
          if (c == chunks - 1) umma_commit(saddr(&bar->a_empty[ab]));
          wit += !keep;
        }
        kept = keep ? s : -1;
      }
    }
  } else if (warp < kFwdProducer0) {
    // ---- epilogue, two groups of four warps that take alternate chunks: tcgen05.ld gives thread = row; the
    // warp's 32 rows go through a padded staging buffer and leave as coalesced 256-byte row segments (two rows
    // per store instruction)
    const int q = warp & 3;                         // TMEM lane quarter this warp may read
    const int group = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    unsigned char* mine = stage + (group * kRows + row) * kStagePitch;
    // rows 2i + (lane >> 4) of this warp are stored by this lane, the 16 bytes lane & 15 of each
    const unsigned char* from = stage + (group * kRows + q * 32 + (lane >> 4)) * kStagePitch + (lane & 15) * 16;
    int64_t* my_offset = offsets + group * kRows + row;
    const int64_t* offset = offsets + group * kRows + q * 32 + (lane >> 4);
    int64_t it = 0;
    for (int tile = blockIdx.x; tile < work.tiles(); tile += gridDim.x) {
      const int s = work.segment(tile);
      const Segment& seg = a.seg[s];
      const int chunks = seg.chunks;
      const int64_t g = work.first_row(tile, s) + row;
      const bool valid = g < work.rows(a, s);
      __syncwarp();
      *my_offset = valid ? row_offset(g, seg.out_mm, seg.out_ld) : -1;
      float* out = seg.out + (lane & 15) * 4;
      const int64_t step = int64_t(seg.out_cs) * kChunk;
      const float* add = (a.bias && s == 0 && valid && g < a.bias_nodes)
                             ? a.bias + (a.bias_index ? ldg(a.bias_index + g + zero) : g + zero) * kK : nullptr;
      for (int c = 0; c < chunks; ++c, ++it, out += step) {
        if (int(it & 1) != group) continue;
        const int d = int(it & 3);
        if (!bar->failed && !mbar_wait(saddr(&bar->d_full[d]), unsigned((it >> 2) & 1))) give_up(bar, a.status, 24);
        tc_fence_after();
        float v0[32], v1[32];
        const unsigned taddr = tmem + (unsigned(q * 32) << 16) + d * kChunk;
        tmem_ld32(taddr, v0);
        tmem_ld32(taddr + 32, v1);
        tc_fence_before();
        mbar_arrive(saddr(&bar->d_empty[d]));
        if (add && c == 0) {
#pragma unroll
          for (int i = 0; i < 32; ++i) { v0[i] += __ldg(add + i); v1[i] += __ldg(add + 32 + i); }
        }
        __syncwarp();                                // the previous chunk's read-back is complete
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          *reinterpret_cast<float4*>(mine + j * 16) = make_float4(v0[4 * j], v0[4 * j + 1], v0[4 * j + 2], v0[4 * j + 3]);
          *reinterpret_cast<float4*>(mine + 128 + j * 16) =
              make_float4(v1[4 * j], v1[4 * j + 1], v1[4 * j + 2], v1[4 * j + 3]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int64_t off = offset[2 * i];
          const float4 v = *reinterpret_cast<const float4*>(from + 2 * i * kStagePitch);
          if (off >= 0) __stcs(reinterpret_cast<float4*>(out + off), v);
        }
      }
    }
  } else {
    // ---- A producers: thread = (row, half of the 64 columns); z3 -> activation -> split -> TMEM
    const int q = warp & 3, half = (warp - kFwdProducer0) >> 2;
    const int row = q * 32 + lane;
    int t = 0;
    for (int tile = blockIdx.x; tile < work.tiles(); tile += gridDim.x, ++t) {
      const int s = work.segment(tile), ab = t & 1;
      const Segment& seg = a.seg[s];
      const int64_t g = work.first_row(tile, s) + row;
      float x[32];
      if (g < work.rows(a, s)) {
        const int64_t srow = a.in_index ? ldg(a.in_index + work.base + g) : work.base + g;
        const float* p = seg.in + row_offset(srow, seg.in_mm, seg.in_ld) + half * 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) ldg256(p + j * 8, x + j * 8);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = 0.f;
      }
      if (a.act) {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = silu_s(x[i]);
      }
      if (!bar->failed && !mbar_wait(saddr(&bar->a_empty[ab]), unsigned((t >> 1) & 1) ^ 1u)) give_up(bar, a.status, 25);
      tc_fence_after();
      const unsigned t_big = tmem_a + (unsigned(q * 32) << 16) + ab * 2 * kK + half * 32;
      store_split_tmem(t_big, t_big + kK, x);
      tc_fence_before();
      mbar_arrive(saddr(&bar->a_full[ab]));
    }
  }
  leave(tmem);
}

// ------------------------------------------------------------------------------------------------
// backward.  Shared memory: W ring (4 x 32 KB) | raw input ring (3 x 32 KB) | barriers.  TMEM: two accumulators [128 x 64]
// that alternate between tiles | A ring of three stages (big + small, 128 columns each); K runs over the chunks.
// A producer warp fetches its 32 rows x 128 bytes of a stage with cp.async (whole lines, four rows per instruction) into a
// private, swizzled buffer two stages ahead, so that neither the latency of the rows nor 32 different lines per load
// instruction are on the path of a stage.  1 M rows of 704: 0.77 ms before (MMA issue 0.11, conversions 0.05, loads 0.06),
// 0.56 now (5.5 TB/s).
constexpr int kRawStages = 3;
constexpr int kRawWarpBytes = 32 * 128;
constexpr int kRawBytes = kRawStages * kProducerWarps * kRawWarpBytes;
constexpr int kBwdSmem = kWStages * kWStageBytes + kRawBytes + 256;

__global__ void __launch_bounds__(kBwdThreads, 1) gate_gemm_backward_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(128) unsigned char gg_smem[];
  unsigned char* w_buf = gg_smem;
  unsigned char* raw = w_buf + kWStages * kWStageBytes;
  Barriers* bar = reinterpret_cast<Barriers*>(raw + kRawBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned tmem = enter(bar, kAStagesBwd, 2);
  const Work work(a, pdl_enter());
  const unsigned tmem_a = tmem + 2 * kChunk;

  if (warp == 0) {
    if (lane == 0) stream_weights(a, work, bar, w_buf, 31);
  } else if (warp == 1) {
    if (elect_one()) {           // ---- MMA issue
      int64_t it = 0, wit = 0;
      int t = 0, kept = -1;
      bool ok = true;
      for (int tile = blockIdx.x; tile < work.tiles() && ok && !bar->failed; tile += gridDim.x, ++t) {
        const int s = work.segment(tile), chunks = a.seg[s].chunks;
        const bool keep = chunks == 1 && tile + int(gridDim.x) < work.tiles() && work.segment(tile + gridDim.x) == s;
        const int d = t & 1;
        if (!mbar_wait(saddr(&bar->d_empty[d]), unsigned((t >> 1) & 1) ^ 1u)) { give_up(bar, a.status, 32); break; }
        for (int c = 0; c < chunks; ++c, ++it) {
          const int slot = int(wit % kWStages), sa = int(it % kAStagesBwd);
          if ((kept != s && !mbar_wait(saddr(&bar->w_full[slot]), unsigned((wit / kWStages) & 1))) ||
              !mbar_wait(saddr(&bar->a_full[sa]), unsigned((it / kAStagesBwd) & 1))) {
            give_up(bar, a.status, 33);
            ok = false;
            break;
          }
          tc_fence_after();
          const unsigned w_big = saddr(w_buf + slot * kWStageBytes), w_small = w_big + kWPartBytes;
          issue_block(tmem + d * kChunk, tmem_a + sa * 2 * kK, w_big, w_small, c == 0);
          if (!keep) umma_commit(saddr(&bar->w_empty[slot]));
          umma_commit(saddr(&bar->a_empty[sa]));
          if (c == chunks - 1) umma_commit(saddr(&bar->d_full[d]));
          wit += !keep;
        }
        kept = keep ? s : -1;
      }
    }
  } else if (warp < kBwdProducer0) {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    int t = 0;
    for (int tile = blockIdx.x; tile < work.tiles(); tile += gridDim.x, ++t) {
      const int s = work.segment(tile), d = t & 1;
      const Segment& seg = a.seg[s];
      const int64_t g = work.first_row(tile, s) + row;
      if (!bar->failed && !mbar_wait(saddr(&bar->d_full[d]), unsigned((t >> 1) & 1))) give_up(bar, a.status, 34);
      tc_fence_after();
      float v0[32], v1[32];
      const unsigned taddr = tmem + (unsigned(q * 32) << 16) + d * kChunk;
      tmem_ld32(taddr, v0);
      tmem_ld32(taddr + 32, v1);
      tc_fence_before();
      mbar_arrive(saddr(&bar->d_empty[d]));
      if (g < work.rows(a, s)) {
        const int64_t orow = a.out_index ? ldg(a.out_index + work.base + g) : work.base + g;
        float4* o = reinterpret_cast<float4*>(seg.out + row_offset(orow, seg.out_mm, seg.out_ld));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j] = make_float4(v0[4 * j], v0[4 * j + 1], v0[4 * j + 2], v0[4 * j + 3]);
          o[8 + j] = make_float4(v1[4 * j], v1[4 * j + 1], v1[4 * j + 2], v1[4 * j + 3]);
        }
      }
    }
  } else {
    // ---- A producers: thread = (row, half of a 64-column chunk); (dG[a] + dG[b]) -> split -> TMEM ring.
    // `fetch` walks the stages (chunks of a tile, tile after tile) ahead of the loop that consumes them.  Lane l of the warp
    // copies the 16-byte piece l & 7 of rows 4j + (l >> 3), j = 0..7; row r's piece p sits at position p ^ (r & 7).
    const int pw = warp - kBwdProducer0, q = warp & 3, half = pw >> 2;
    unsigned char* mine = raw + pw * kRawWarpBytes;
    int f_tile = blockIdx.x, f_c = 0, f_chunks = 0, f_slot = 0;
    int64_t f_step = 0;
    const float* f_row[8];
    auto enter_tile = [&]() {
      if (f_tile >= work.tiles()) return;
      const int s = work.segment(f_tile);
      const Segment& seg = a.seg[s];
      f_chunks = seg.chunks;
      f_step = int64_t(seg.in_cs) * kChunk;
      const int64_t nrows = work.rows(a, s), first = work.first_row(f_tile, s) + q * 32;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int64_t g = first + 4 * j + (lane >> 3);
        const int64_t r = g < nrows ? (a.pair_a ? ldg(a.pair_a + work.base + g) : g) : -1;
        f_row[j] = r < 0 ? nullptr : seg.in + row_offset(r, seg.in_mm, seg.in_ld) + half * 32 + (lane & 7) * 4;
      }
    };
    auto fetch = [&]() {
      if (f_tile < work.tiles()) {
        unsigned char* slot = mine + f_slot * (kProducerWarps * kRawWarpBytes);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = 4 * j + (lane >> 3);
          const unsigned dst = saddr(slot + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
          const float* src = f_row[j] ? f_row[j] + f_c * f_step : a.seg[0].in;
          cp_async16(dst, src, f_row[j] ? 16u : 0u);          // rows beyond the end are zeros
        }
        if (++f_slot == kRawStages) f_slot = 0;
        if (++f_c == f_chunks) {
          f_c = 0;
          f_tile += gridDim.x;
          enter_tile();
        }
      }
      cp_async_commit();
    };
    enter_tile();
#pragma unroll
    for (int k = 0; k < kRawStages - 1; ++k) fetch();
    int64_t it = 0;
    int slot = 0;
    for (int tile = blockIdx.x; tile < work.tiles(); tile += gridDim.x) {
      const int s = work.segment(tile), chunks = a.seg[s].chunks;
      const Segment& seg = a.seg[s];
      const int64_t g = work.first_row(tile, s) + q * 32 + lane;
      const int64_t rb = (a.pair_b && g < work.rows(a, s)) ? ldg(a.pair_b + work.base + g) : -1;
      for (int c = 0; c < chunks; ++c, ++it) {
        const int sa = int(it % kAStagesBwd);
        fetch();
        cp_async_wait<kRawStages - 1>();
        __syncwarp();
        float x[32];
        const unsigned char* rows = mine + slot * (kProducerWarps * kRawWarpBytes) + lane * 128;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const float4 v = *reinterpret_cast<const float4*>(rows + ((p ^ (lane & 7)) << 4));
          x[4 * p] = v.x; x[4 * p + 1] = v.y; x[4 * p + 2] = v.z; x[4 * p + 3] = v.w;
        }
        __syncwarp();                          // the slot may be filled again
        if (++slot == kRawStages) slot = 0;
        if (rb >= 0) {
          const float* pb = seg.in + row_offset(rb, seg.in_mm, seg.in_ld) + half * 32 + c * (int64_t(seg.in_cs) * kChunk);
          float y[32];
#pragma unroll
          for (int j = 0; j < 4; ++j) ldg256(pb + j * 8, y + j * 8);
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] += y[i];
        }
        if (!bar->failed && !mbar_wait(saddr(&bar->a_empty[sa]), unsigned((it / kAStagesBwd) & 1) ^ 1u)) give_up(bar, a.status, 35);
        tc_fence_after();
        const unsigned t_big = tmem_a + (unsigned(q * 32) << 16) + sa * 2 * kK + half * 32;
        store_split_tmem(t_big, t_big + kK, x);
        tc_fence_before();
        mbar_arrive(saddr(&bar->a_full[sa]));
      }
    }
    cp_async_wait<0>();          // no copy may be in flight when the block leaves
  }
  leave(tmem);
}

// Packs W3 [nout, 64] into 64-unit chunks in the shared-memory operand layout, big part then small part.
// transpose = 0 (forward B operand):  block(n, k) = W3[c*64 + n][k]
// transpose = 1 (backward B operand): block(n, k) = W3[c*64 + k][n]
__global__ void gate_pack_kernel(int nout, const float* __restrict__ w, int transpose, float* out) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nout * kK) return;
  const int c = idx / (kChunk * kK), rem = idx % (kChunk * kK), n = rem / kK, k = rem % kK;
  const float v = transpose ? w[(c * kChunk + k) * kK + n] : w[(c * kChunk + n) * kK + k];
  const float big = to_tf32(v), small = to_tf32(v - big);
  const int off = (k / 4) * (kChunk * 4) + n * 4 + (k % 4);
  out[c * (2 * kChunk * kK) + off] = big;
  out[c * (2 * kChunk * kK) + kChunk * kK + off] = small;
}

// One persistent CTA per SM
static int prepare(Args& a, bool& one_wave) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int64_t tiles = 0;
  for (int s = 0; s < a.segments; ++s) tiles += (a.seg[s].rows + kRows - 1) / kRows;
  a.status = kernel_status_word();
  one_wave = tiles <= sms;
  return int(tiles < sms ? tiles : sms);
}

int launch_forward(Args a, cudaStream_t st) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(gate_gemm_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  if (attr != cudaSuccess) { set_error("gate gemm smem: %s", cudaGetErrorString(attr)); return ICTC_ERR_LAUNCH; }
  bool one_wave;
  const int grid = prepare(a, one_wave);
  if (grid == 0) return ICTC_OK;          // no rows
  launch_if(one_wave, gate_gemm_forward_kernel, grid, kFwdThreads, kFwdSmem, st, a);
  return finish_launch("gate_gemm_forward");
}

int launch_backward(Args a, cudaStream_t st) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(gate_gemm_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem);
  if (attr != cudaSuccess) { set_error("gate gemm smem: %s", cudaGetErrorString(attr)); return ICTC_ERR_LAUNCH; }
  bool one_wave;
  const int grid = prepare(a, one_wave);
  if (grid == 0) return ICTC_OK;          // no rows
  launch_if(one_wave, gate_gemm_backward_kernel, grid, kBwdThreads, kBwdSmem, st, a);
  return finish_launch("gate_gemm_backward");
}

static int check_common(int64_t rows, int nout) {
  if (rows < 0 || nout < kChunk || nout % kChunk) {
    set_error("gate gemm: the gate width must be a positive multiple of 64 (got %d)", nout);
    return ICTC_ERR_BAD_SPEC;
  }
  return ICTC_OK;
}

}  // namespace gg
}  // namespace ictc

using namespace ictc;

extern "C" {

int ictc_gate_pack_weights(int num_out, const float* w3, int transpose, float* packed, void* stream) {
  if (int rc = gg::check_common(0, num_out)) return rc;
  if (!w3 || !packed) { set_error("gate pack: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  const int n = num_out * gg::kK;
  gg::gate_pack_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(num_out, w3, transpose ? 1 : 0, packed);
  return finish_launch("gate_pack");
}

int ictc_gate_gemm_forward(int64_t num_rows, int num_out, const float* z3, const float* w_packed, float* gates,
                           int apply_silu, const int64_t* row_limit, void* stream) {
  if (int rc = gg::check_common(num_rows, num_out)) return rc;
  if (num_rows == 0) return ICTC_OK;
  if (!z3 || !w_packed || !gates) { set_error("gate gemm forward: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(z3) | reinterpret_cast<uintptr_t>(w_packed) | reinterpret_cast<uintptr_t>(gates)) & 31) {
    set_error("gate gemm forward: buffers must be 32-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  gg::Args a{};
  a.segments = 1;
  a.seg[0] = gg::segment(z3, w_packed, gates, num_rows, num_out / gg::kChunk, 1, gg::kK, 1, num_out);
  a.limit = row_limit; a.act = apply_silu ? 1 : 0;
  return gg::launch_forward(a, (cudaStream_t)stream);
}

int ictc_gate_gemm_backward(int64_t num_rows, int num_out, const float* dgates, const int64_t* pair_a,
                            const int64_t* pair_b, const float* w_packed_t, float* da3, const int64_t* row_limit,
                            void* stream) {
  if (int rc = gg::check_common(num_rows, num_out)) return rc;
  if (num_rows == 0) return ICTC_OK;
  if (!dgates || !w_packed_t || !da3) { set_error("gate gemm backward: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(dgates) | reinterpret_cast<uintptr_t>(w_packed_t) | reinterpret_cast<uintptr_t>(da3)) & 31) {
    set_error("gate gemm backward: buffers must be 32-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  gg::Args a{};
  a.segments = 1;
  a.seg[0] = gg::segment(dgates, w_packed_t, da3, num_rows, num_out / gg::kChunk, 1, num_out, 1, gg::kK);
  a.pair_a = pair_a; a.pair_b = pair_b; a.limit = row_limit;
  return gg::launch_backward(a, (cudaStream_t)stream);
}


int ictc_gate_gemm_forward_rows(int64_t capacity, int num_out, const float* z3, const int64_t* row_index,
                                const int64_t* row_begin, const int64_t* row_end, const float* w_packed, float* gates,
                                int apply_silu, void* stream) {
  if (int rc = gg::check_common(capacity, num_out)) return rc;
  if (capacity == 0) return ICTC_OK;
  if (!z3 || !w_packed || !gates || !row_begin || !row_end) { set_error("gate gemm forward rows: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(z3) | reinterpret_cast<uintptr_t>(w_packed) | reinterpret_cast<uintptr_t>(gates)) & 31) {
    set_error("gate gemm forward rows: buffers must be 32-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  gg::Args a{};
  a.segments = 1;
  a.seg[0] = gg::segment(z3, w_packed, gates, capacity, num_out / gg::kChunk, 1, gg::kK, 1, num_out);
  a.limit = row_end; a.begin = row_begin; a.in_index = row_index; a.act = apply_silu ? 1 : 0;
  return gg::launch_forward(a, (cudaStream_t)stream);
}

int ictc_gate_gemm_backward_rows(int64_t capacity, int num_out, const float* dgates, const int64_t* row_begin,
                                 const int64_t* row_end, const int64_t* out_index, const float* w_packed_t, float* da3,
                                 void* stream) {
  if (int rc = gg::check_common(capacity, num_out)) return rc;
  if (capacity == 0) return ICTC_OK;
  if (!dgates || !w_packed_t || !da3 || !row_begin || !row_end) { set_error("gate gemm backward rows: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(dgates) | reinterpret_cast<uintptr_t>(w_packed_t) | reinterpret_cast<uintptr_t>(da3)) & 31) {
    set_error("gate gemm backward rows: buffers must be 32-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  gg::Args a{};
  a.segments = 1;
  a.seg[0] = gg::segment(dgates, w_packed_t, da3, capacity, num_out / gg::kChunk, 1, num_out, 1, gg::kK);
  a.limit = row_end; a.begin = row_begin; a.out_index = out_index;
  return gg::launch_backward(a, (cudaStream_t)stream);
}


int ictc_channel_linear_tc(int64_t num_rows, int k_chunks, int n_chunks, const float* in, int in_mm, int64_t in_ld,
                           const float* w_packed, float* out, int out_mm, int64_t out_ld, void* stream) {
  if (num_rows < 0 || k_chunks < 1 || n_chunks < 1 || (k_chunks > 1 && n_chunks > 1) || in_mm < 1 || out_mm < 1 ||
      in_ld < 0 || out_ld < 0) {
    set_error("channel linear: one side must be 64 wide, the other a multiple of 64 (got %d x %d chunks)", k_chunks,
              n_chunks);
    return ICTC_ERR_BAD_SPEC;
  }
  if (num_rows == 0) return ICTC_OK;
  if (!in || !w_packed || !out) { set_error("channel linear: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  if (((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(w_packed) | reinterpret_cast<uintptr_t>(out)) & 31) ||
      (in_ld & 7) || (out_ld & 7)) {
    set_error("channel linear: buffers must be 32-byte aligned and strides multiples of 8 floats");
    return ICTC_ERR_BAD_ARG;
  }
  gg::Args a{};
  a.segments = 1;
  a.seg[0] = gg::segment(in, w_packed, out, num_rows, k_chunks * n_chunks, in_mm, in_ld, out_mm, out_ld);
  return k_chunks == 1 ? gg::launch_forward(a, (cudaStream_t)stream) : gg::launch_backward(a, (cudaStream_t)stream);
}

}  // extern "C"
