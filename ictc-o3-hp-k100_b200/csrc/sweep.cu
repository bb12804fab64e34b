// Force sweep: energy and position gradient of the two-interaction model as one native launch sequence.
//
// The reverse sweep is the hand-written adjoint of the forward sweep; no tape, no host read-back, every intermediate in one
// workspace of the caller (reference: mace_ictc/hp/runtime.py:82-111 over mace_ictc/models/mace/backbone.py:860-1246).
// What used to be about 100 launches per evaluation, driven from Python, is about 30:
//   * the element-wise ends (species lookup, geometry, readouts with their adjoint, position gradient) are the kernels of
//     this file, one each;
//   * a channel linear is one launch for its three degree blocks (gate_gemm.cu);
//   * the hidden radial layers of both interactions share a launch in each direction (mlp_chain.cu);
//   * products of weight matrices that no input depends on (embedding x linear_up, embedding x self connection,
//     readout x product linear) are formed when the weights are laid out, not per atom.
#include <exception>
#include <vector>
#include "csr.cuh"
#include "gate_gemm.cuh"
#include "geometry.cuh"
#include "mlp_chain.cuh"
#include "scan.cuh"
#include "tp_chunk.cuh"

namespace ictc {
namespace sweep {

constexpr int kC = 64;
constexpr float kSilu = 1.6791767923989418f;

// ------------------------------------------------------------------------------------------------ species, embedding
struct EmbedArgs {
  const int64_t* numbers;      // atomic numbers, or null: `species` is the input
  const int64_t* table;        // species index of an atomic number, -1 = not in the model
  int64_t table_size;
  int64_t* species;
  const float* up;             // [S, 64] embedding times linear_up
  float* u0;                   // [n, 64]
  double* energy;              // [graphs], cleared here (several graphs)
  int64_t graphs, n;
  const int64_t* batch;        // or null
  int* status;                 // bit 0: an atomic number outside the model, bit 1: a graph index outside [0, graphs)
};

__global__ void embed_kernel(EmbedArgs a) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i < a.graphs) a.energy[i] = 0.0;
  const int64_t row = i >> 4;
  if (row >= a.n) return;
  int64_t s;
  if (a.numbers) {
    int64_t z = ldg(a.numbers + row);
    if (z < 0) z += a.table_size;            // as an index of the table counts from its end in the model's forward
    s = z >= 0 && z < a.table_size ? ldg(a.table + z) : -1;
    if ((i & 15) == 0) {
      if (s < 0) atomicOr(a.status, 1);
      a.species[row] = s < 0 ? 0 : s;
    }
    if (s < 0) s = 0;
  } else {
    s = a.species[row];
  }
  if (a.batch && (i & 15) == 1) {
    const int64_t b = ldg(a.batch + row);
    if (b < 0 || b >= a.graphs) atomicOr(a.status, 2);
  }
  reinterpret_cast<float4*>(a.u0)[i] = __ldg(reinterpret_cast<const float4*>(a.up + s * kC) + (i & 15));
}

// Are the parameters still what the weights were laid out from?  A version counter does not see a write through
// `parameter.data`, so every word is compared (0.25 M words: 3 us, hidden behind the host's next launches).
constexpr int kWatchWords = 2048, kWatchThreads = 256;

__global__ void __launch_bounds__(kWatchThreads) watch_kernel(const int64_t* __restrict__ tiles, const int* __restrict__ copy,
                                                              int* status) {
  const int64_t t = blockIdx.x + pdl_enter();
  const int* now = reinterpret_cast<const int*>(ldg(tiles + 2 * t));
  const int words = int(ldg(tiles + 2 * t + 1));
  bool differ = false;
#pragma unroll
  for (int k = 0; k < kWatchWords / kWatchThreads; ++k) {
    const int i = threadIdx.x + k * kWatchThreads;
    if (i < words) differ |= now[i] != copy[t * kWatchWords + i];
  }
  if (__syncthreads_or(differ) && threadIdx.x == 0) atomicOr(status, 4);
}

// Graph of an atom; an index outside the batch is flagged by embed_kernel and read as graph 0.
__device__ __forceinline__ int64_t graph_of(const int64_t* batch, int64_t atom, int64_t graphs) {
  const int64_t b = ldg(batch + atom);
  return b >= 0 && b < graphs ? b : 0;
}

// ------------------------------------------------------------------------------------------------ geometry
struct GeoArgs {
  const float* pos;
  const int64_t* src;
  const int64_t* dst;
  const float* shifts;         // lattice units, or null
  float box[3];
  const float* cells;          // [graphs, 3, 3] or null: `box`
  const int64_t* batch;        // graph of an atom (null: graph 0)
  int64_t graphs;
  float r_max;
  int num_basis, p;
  int64_t E;
  const int64_t* gate_row;     // pair row of an edge (null: the edge itself)
  const int64_t* rep;          // edge that represents a pair row
  float* sh;                   // [E, 9]
  float4* geo;                 // unit vector, length
  int64_t* safe_src;           // edge ends with indices outside [0, N) replaced, or null: the indices are trusted
  int64_t* safe_dst;
  int64_t N;
  float* rb;                   // [rows, num_basis], one row per pair
  const float* dsh[2];         // backward: gradients of the harmonics and of the radial basis, per interaction
  const float* drb[2];
  float4* dvec;
};

constexpr int kGeoThreads = 256;

// Copies the block's part of a [E, 9] array between shared memory and global memory in 16-byte pieces: with a thread
// per edge the nine floats of an edge are 36 bytes apart (4.3 M edges: 344 -> 150 us forward).
template <bool STORE> __device__ __forceinline__ void block_rows9(float* global, float* shared, int64_t first, int64_t E) {
  const int n = 9 * int(min(int64_t(kGeoThreads), E - first));
  float* g = global + 9 * first;
  for (int i = threadIdx.x * 4; i < n; i += kGeoThreads * 4) {
    if (i + 4 <= n) {
      if (STORE) *reinterpret_cast<float4*>(g + i) = *reinterpret_cast<const float4*>(shared + i);
      else *reinterpret_cast<float4*>(shared + i) = __ldg(reinterpret_cast<const float4*>(g + i));
    } else {
      for (int k = i; k < n; ++k) {
        if (STORE) g[k] = shared[k];
        else shared[k] = g[k];
      }
    }
  }
}

__global__ void __launch_bounds__(kGeoThreads) geometry_kernel(GeoArgs a) {
  __shared__ __align__(16) float rows[kGeoThreads * 9];
  const int64_t first = int64_t(blockIdx.x) * kGeoThreads + pdl_enter(), e = first + threadIdx.x;
  if (e < a.E) {
    int64_t i = ldg(a.dst + e), j = ldg(a.src + e);
    if (a.safe_src) {
      i = i >= 0 && i < a.N ? i : 0;
      j = j >= 0 && j < a.N ? j : 0;
      a.safe_dst[e] = i;
      a.safe_src[e] = j;
    }
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = ldg(a.pos + 3 * i + k) - ldg(a.pos + 3 * j + k);
    if (a.shifts) {
      const float s0 = a.shifts[3 * e], s1 = a.shifts[3 * e + 1], s2 = a.shifts[3 * e + 2];
      if (a.cells) {
        const float* cell = a.cells + 9 * (a.batch ? graph_of(a.batch, j, a.graphs) : 0);
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] += s0 * ldg(cell + k) + s1 * ldg(cell + 3 + k) + s2 * ldg(cell + 6 + k);
      } else {
        v[0] += s0 * a.box[0];
        v[1] += s1 * a.box[1];
        v[2] += s2 * a.box[2];
      }
    }
    const float r = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const float rc = fmaxf(r, 1e-8f);
    const float x = v[0] / rc, y = v[1] / rc, z = v[2] / rc;
    a.geo[e] = make_float4(x, y, z, r);
    float val[9];
    harmonics_value(x, y, z, val);
#pragma unroll
    for (int h = 0; h < 9; ++h) rows[9 * threadIdx.x + h] = val[h];
    const int64_t u = a.gate_row ? ldg(a.gate_row + e) : e;
    if (!a.rep || ldg(a.rep + u) == e) {         // the radial basis of a pair is written once
      float env, denv;
      envelope(r, a.r_max, a.p, env, denv);
      const float pref = sqrtf(2.f / a.r_max) / fmaxf(r, 1e-12f);
      const float w = 3.14159265358979323846f / a.r_max;
      float* o = a.rb + u * a.num_basis;
      if (a.num_basis == 8) {
        float b[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) b[k] = env == 0.f ? 0.f : pref * sinf(r * (w * float(k + 1))) * env;
        reinterpret_cast<float4*>(o)[0] = make_float4(b[0], b[1], b[2], b[3]);
        reinterpret_cast<float4*>(o)[1] = make_float4(b[4], b[5], b[6], b[7]);
      } else {
        for (int k = 0; k < a.num_basis; ++k) o[k] = env == 0.f ? 0.f : pref * sinf(r * (w * float(k + 1))) * env;
      }
    }
  }
  __syncthreads();
  block_rows9<true>(a.sh, rows, first, a.E);
}

__global__ void __launch_bounds__(kGeoThreads) geometry_backward_kernel(GeoArgs a) {
  __shared__ __align__(16) float rows[2][kGeoThreads * 9];
  const int64_t first = int64_t(blockIdx.x) * kGeoThreads + pdl_enter(), e = first + threadIdx.x;
  block_rows9<false>(const_cast<float*>(a.dsh[0]), rows[0], first, a.E);
  block_rows9<false>(const_cast<float*>(a.dsh[1]), rows[1], first, a.E);
  __syncthreads();
  if (e >= a.E) return;
  const float4 q = a.geo[e];
  float g[9];
#pragma unroll
  for (int h = 0; h < 9; ++h) g[h] = rows[0][9 * threadIdx.x + h] + rows[1][9 * threadIdx.x + h];
  const int64_t u = a.gate_row ? ldg(a.gate_row + e) : e;
  float d[16];
  const bool mine = !a.rep || ldg(a.rep + u) == e;
  if (mine)
    for (int k = 0; k < a.num_basis; ++k)
      d[k] = ldg(a.drb[0] + u * a.num_basis + k) + ldg(a.drb[1] + u * a.num_basis + k);
  const float3 v = edge_vector_gradient(q.x, q.y, q.z, q.w, g, mine ? d : nullptr, a.num_basis, a.p, a.r_max);
  a.dvec[e] = make_float4(v.x, v.y, v.z, 0.f);
}

// out[i] = sign * (sum_{e: dst(e)=i} dvec[e] - sum_{e: src(e)=i} dvec[e]); eight lanes per atom, fixed order, no atomics.
struct GradArgs {
  int64_t n, n_dst_rows;
  const int64_t *dst_rowptr, *dst_order, *src_rowptr, *src_order;
  const float4* dvec;
  float sign;
  float* out;
  const double* energy_sum;    // sums per graph, or (parts > 0) the readout blocks' sums of the one graph
  float* energy;
  int64_t graphs, parts;
};

// The one graph's energy: the first block adds the readout blocks' sums, every thread its own and then a tree, in an order that
// depends on their number alone (the sweep is repeatable bit by bit).  131,072 atoms have 4,096 of them.
constexpr int kGradThreads = 256;
__device__ __forceinline__ void add_energy(const GradArgs& a) {
  __shared__ double part[kGradThreads];
  double s = 0.0;
  for (int64_t k = threadIdx.x; k < a.parts; k += kGradThreads) s += a.energy_sum[k];
  part[threadIdx.x] = s;
  for (int half = kGradThreads / 2; half > 0; half >>= 1) {
    __syncthreads();
    if (threadIdx.x < half) part[threadIdx.x] += part[threadIdx.x + half];
  }
  if (threadIdx.x == 0) a.energy[0] = float(part[0]);
}

__global__ void __launch_bounds__(kGradThreads) position_gradient8_kernel(GradArgs a) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (a.parts > 0) {
    if (blockIdx.x == 0) add_energy(a);
  } else if (t < a.graphs) {
    a.energy[t] = float(a.energy_sum[t]);
  }
  const int64_t i = t >> 3;
  const int sub = int(t & 7);
  float x = 0.f, y = 0.f, z = 0.f;
  if (i < a.n_dst_rows) {
    const int64_t end = ldg(a.dst_rowptr + i + 1);
    for (int64_t k = ldg(a.dst_rowptr + i) + sub; k < end; k += 8) {
      const float4 d = __ldg(a.dvec + (a.dst_order ? ldg(a.dst_order + k) : k));
      x += d.x; y += d.y; z += d.z;
    }
  }
  if (i < a.n) {
    const int64_t end = ldg(a.src_rowptr + i + 1);
    for (int64_t k = ldg(a.src_rowptr + i) + sub; k < end; k += 8) {
      const float4 d = __ldg(a.dvec + (a.src_order ? ldg(a.src_order + k) : k));
      x -= d.x; y -= d.y; z -= d.z;
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
    z += __shfl_xor_sync(0xffffffffu, z, o);
  }
  if (i < a.n && sub == 0) {
    a.out[3 * i] = a.sign * x;
    a.out[3 * i + 1] = a.sign * y;
    a.out[3 * i + 2] = a.sign * z;
  }
}

// out[i] = table[index[i]]; a sender order is not filled behind its last row (inert edges have no sender), so what stands
// there is not an index.
__global__ void gather_index_kernel(const int64_t* __restrict__ table, const int64_t* __restrict__ index, int64_t n, int64_t* out) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i >= n) return;
  const int64_t k = index[i];
  out[i] = k >= 0 && k < n ? table[k] : 0;
}
static int gather_index(const int64_t* table, const int64_t* index, int64_t n, int64_t* out, cudaStream_t st) {
  if (n > 0) launch_after(gather_index_kernel, (unsigned)((n + 255) / 256), 256, 0, st, table, index, n, out);
  return finish_launch("sweep_gather_index");
}

// ------------------------------------------------------------------------------------------------ readouts
// Both readouts and their adjoint in one pass, a warp per atom, two channels per lane.  With the product linear P, the
// self connection S_s and the readout matrix R the last hidden layer is z = R (P y + S_s h) = (R P) y + (R S_s) h, so
// two [H, 64] products per atom replace four [64, 64] ones and their adjoints.
//   energy = ro0 . h + sum_k w2[k] silu(z[k]);  dy = (R P)^T dz;  dh = (R S_s)^T dz + ro0
struct TailArgs {
  const float* y;              // [n, 64] product of the last interaction
  const float* h;              // scalar block of the first interaction's features
  int64_t h_ld;
  const int64_t* species;
  const float* rp;             // [H, 64]
  const float* rs;             // [S, H, 64]
  const float* w2;             // [H]
  const float* ro0;            // [64]
  int H;
  const float* mask;           // [n] or null
  const int64_t* batch;        // or null
  int64_t graphs;
  int mask_atomic;
  float* atomic;               // [n]
  double* energy;              // [graphs], added to; without a batch [blocks], written
  float* dy;                   // [n, 64]
  float* dh;                   // [n, 64]
  int64_t n;
};

// While the atoms do not fill the chip's warp slots (148 SMs x 64) a warp has one atom, beyond that four, which quarters the sums
// that the last kernel adds up (and a batch's atomics).  Recorded MD step with one atom / four: 216 atoms 262 / 267 us, 1,000
// 394 / 403, 2,744 774 / 780, 8,000 1,812 / 1,829; 17,576 3,891 / 3,850, larger systems within the runs' spread of 1 %.
constexpr int kTailWarps = 8;
constexpr int64_t kTailSlots = 148 * 64;
static int tail_nodes(int64_t n) { return n <= kTailSlots ? 1 : 4; }
static int64_t tail_blocks(int64_t n) { return (n + kTailWarps * tail_nodes(n) - 1) / (kTailWarps * tail_nodes(n)); }

__global__ void __launch_bounds__(kTailWarps * 32) tail_kernel(TailArgs a, int nodes) {
  __shared__ double block_energy[kTailWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int zero = pdl_enter();
  const int64_t first = (int64_t(blockIdx.x) * kTailWarps + warp) * nodes + zero;
  const float2 ro = __ldg(reinterpret_cast<const float2*>(a.ro0 + zero) + lane);
  double sum = 0.0;
  int64_t graph = -1;
  for (int64_t n = first; n < first + nodes && n < a.n; ++n) {
    const float2 y = __ldg(reinterpret_cast<const float2*>(a.y + n * kC) + lane);
    const float2 h = __ldg(reinterpret_cast<const float2*>(a.h + n * a.h_ld) + lane);
    const float2* rp = reinterpret_cast<const float2*>(a.rp + zero) + lane;
    const float2* rs = reinterpret_cast<const float2*>(a.rs + ldg(a.species + n) * a.H * kC) + lane;
    const float m = a.mask ? ldg(a.mask + n) : 1.f;
    float e = fmaf(h.x, ro.x, h.y * ro.y);
    float2 dy = make_float2(0.f, 0.f), dh = make_float2(ro.x * m, ro.y * m);
    for (int k0 = 0; k0 < a.H; k0 += 16) {
      float v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        v[k] = 0.f;
        if (k0 + k < a.H) {
          const float2 p = __ldg(rp + (k0 + k) * (kC / 2)), s = __ldg(rs + (k0 + k) * (kC / 2));
          v[k] = fmaf(y.x, p.x, fmaf(y.y, p.y, fmaf(h.x, s.x, h.y * s.y)));
        }
      }
      int idx;
      bool valid;
      const float z = warp_reduce_scatter<16>(v, lane, idx, valid);        // hidden unit k sits on lane 2k
      float dz = 0.f;
      if (valid && k0 + idx < a.H) {
        const float w = ldg(a.w2 + zero + k0 + idx);
        const float s = 1.f / (1.f + expf(-z));
        e = fmaf(w, z * s * kSilu, e);
        dz = w * m * kSilu * s * (1.f + z * (1.f - s));
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float d = __shfl_sync(0xffffffffu, dz, 2 * k);
        if (k0 + k < a.H) {
          const float2 p = __ldg(rp + (k0 + k) * (kC / 2)), s = __ldg(rs + (k0 + k) * (kC / 2));
          dy.x = fmaf(d, p.x, dy.x); dy.y = fmaf(d, p.y, dy.y);
          dh.x = fmaf(d, s.x, dh.x); dh.y = fmaf(d, s.y, dh.y);
        }
      }
    }
    reinterpret_cast<float2*>(a.dy + n * kC)[lane] = dy;
    reinterpret_cast<float2*>(a.dh + n * kC)[lane] = dh;
    e = warp_sum(e);
    if (lane == 0) {
      a.atomic[n] = a.mask_atomic ? e * m : e;
      if (a.batch) {
        const int64_t b = graph_of(a.batch, n, a.graphs);
        if (b != graph && graph >= 0) {
          atomicAdd(a.energy + graph, sum);
          sum = 0.0;
        }
        graph = b;
      }
      sum += double(e * m);
    }
  }
  if (a.batch) {
    if (lane == 0 && graph >= 0) atomicAdd(a.energy + graph, sum);
    return;
  }
  if (lane == 0) block_energy[warp] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int w = 0; w < kTailWarps; ++w) total += block_energy[w];
    a.energy[blockIdx.x] = total;
  }
}

// ------------------------------------------------------------------------------------------------ host sequence
// First-fit placement of the intermediates in the caller's workspace.  Every call replays the same takes and gives, so the
// offsets of one stage are known to the next; a buffer that was given back is reused by later launches of the same stream.
class Arena {
 public:
  int64_t take(int64_t bytes) {
    bytes = bytes > 0 ? (bytes + 255) / 256 * 256 : 256;
    for (size_t i = 0; i < free_.size(); ++i)
      if (free_[i].second >= bytes) {
        const int64_t at = free_[i].first;
        free_[i].first += bytes;
        free_[i].second -= bytes;
        if (free_[i].second == 0) free_.erase(free_.begin() + i);
        used_.emplace_back(at, bytes);
        return at;
      }
    int64_t at = top_;
    if (!free_.empty() && free_.back().first + free_.back().second == top_) {      // grow the hole at the top
      at = free_.back().first;
      free_.pop_back();
    }
    top_ = at + bytes;
    if (top_ > peak_) peak_ = top_;
    used_.emplace_back(at, bytes);
    return at;
  }
  void give(int64_t at) {
    for (size_t i = 0; i < used_.size(); ++i)
      if (used_[i].first == at) {
        auto block = used_[i];
        used_.erase(used_.begin() + i);
        size_t k = 0;
        while (k < free_.size() && free_[k].first < block.first) ++k;
        if (k < free_.size() && block.first + block.second == free_[k].first) {
          block.second += free_[k].second;
          free_.erase(free_.begin() + k);
        }
        if (k > 0 && free_[k - 1].first + free_[k - 1].second == block.first) {
          free_[k - 1].second += block.second;
        } else {
          free_.insert(free_.begin() + k, block);
        }
        return;
      }
  }
  int64_t peak() const { return peak_; }

 private:
  std::vector<std::pair<int64_t, int64_t>> free_, used_;      // (offset, bytes), free blocks sorted
  int64_t top_ = 0, peak_ = 0;
};

enum Label { kHiddenFwd, kGateFwd, kGraphFwd, kGraphAdj, kGateBwd, kHiddenBwd, kLinear, kContraction };

class Runner {
 public:
  // `dry`: placement only, nothing is launched
  Runner(const ictc_sweep& p, int stages, cudaStream_t st, bool dry) : p(p), stages(stages), st(st), dry(dry) {}
  int run();
  int64_t peak() const { return arena.peak(); }

 private:
  const ictc_sweep& p;
  const int stages;
  cudaStream_t st;
  const bool dry;
  Arena arena;
  int rc = 0;

  template <class T = float> T* buffer(int64_t count) {
    return reinterpret_cast<T*>(static_cast<char*>(p.work) + arena.take(count * int64_t(sizeof(T))));
  }
  void release(const void* ptr) { arena.give(static_cast<const char*>(ptr) - static_cast<const char*>(p.work)); }
  bool on(int stage) const { return rc == 0 && !dry && (stages & stage); }
  // one library call that launches `n` kernels; `label` >= 0: timed between two of the caller's events
  template <class F> void call(int stage, int label, int n, F f) {
    if (!on(stage)) return;
    const bool timed = label >= 0 && p.host_marks && p.host_counts[1] < p.host_marks_capacity;
    const int64_t k = timed ? p.host_counts[1]++ : 0;
    if (timed) {
      p.host_mark_labels[k] = label;
      cudaEventRecord(static_cast<cudaEvent_t>(p.host_marks[2 * k]), st);
    }
    rc = f();
    if (timed) cudaEventRecord(static_cast<cudaEvent_t>(p.host_marks[2 * k + 1]), st);
    if (p.host_counts) p.host_counts[0] += n;
  }
  int label(Label l, int layer) const { return int(l) * 2 + layer; }

  // One channel linear over the degree blocks of [rows, 576] buffers; `wide_in` / `wide_out`: that side is the
  // slot-major tensor-product layout [rows, path slots per degree, 2l+1, 64].
  void linear(int stage, int layer, const float* const (&w)[3], int64_t rows, const float* in, int64_t in_ld, bool wide_in,
              float* out, int64_t out_ld, bool wide_out, const float* bias = nullptr, const int64_t* bias_index = nullptr,
              int64_t bias_nodes = 0) {
    gg::Args a{};
    a.segments = 3;
    int64_t in_off = 0, out_off = 0;
    bool deep = false;
    for (int l = 0; l < 3; ++l) {
      const int mm = 2 * l + 1;
      const int64_t slots = p.layer[layer].slots[l];
      const int chunks = wide_in || wide_out ? int(slots) : 1;
      if (wide_in && slots > 1) deep = true;
      a.seg[l] = gg::segment(in + in_off, w[l], out + out_off, rows * mm, chunks, mm, in_ld, mm, out_ld);
      in_off += kC * mm * (wide_in ? slots : 1);
      out_off += kC * mm * (wide_out ? slots : 1);
    }
    a.bias = bias; a.bias_index = bias_index; a.bias_nodes = bias_nodes;
    call(stage, label(kLinear, layer), 1, [&] { return deep ? gg::launch_backward(a, st) : gg::launch_forward(a, st); });
  }

  // messages and feature gradients of a list without edges
  void clear(int stage, float* out, int64_t count) {
    call(stage, -1, 1, [&] {
      if (count > 0) cudaMemsetAsync(out, 0, count * sizeof(float), st);
      return finish_launch("sweep_clear");
    });
  }

  // Chunk bounds of a sweep over `rows` owner rows.
  int64_t chunk_rows(int64_t rows) const { return p.chunk_rows > 0 && p.chunk_rows < rows ? p.chunk_rows : rows; }

  void gates(int stage, int layer, const float* z3, float* out, int64_t rows, const int64_t* index, const int64_t* begin,
             const int64_t* end) {
    const ictc_sweep_layer& L = p.layer[layer];
    call(stage, label(kGateFwd, layer), 1, [&] {
      gg::Args a{};
      a.segments = 1;
      a.seg[0] = gg::segment(z3, L.w3, out, rows, int(L.num_gates / kC), 1, kC, 1, L.num_gates);
      a.act = 1; a.begin = begin; a.in_index = index; a.limit = end;
      return gg::launch_forward(a, st);
    });
  }
};

int Runner::run() {
  const int64_t n = p.n_owned, N = p.n_local, E = p.edges, U = p.rep && E > 0 ? p.pair_rows : E;
  const ictc_sweep_layer &L0 = p.layer[0], &L1 = p.layer[1];
  const int spec[2] = {ictc_tp_spec(0, 2, 2), ictc_tp_spec(2, 2, 2)};
  const int64_t W0 = 9 * kC, W1 = 35 * kC;
  const bool paired = p.rep != nullptr;
  const bool table = !(p.chunk_rows > 0 && p.chunk_rows < (n > N ? n : N) && p.stream_gates);
  // The interactions share launches when all stages run together; with timing every launch is one interaction's.  Both
  // reverse sweeps' hidden gradients (256 bytes an edge) are then alive together: not for lists beyond 4 M edges, where the time is
  // the same and the memory counts.  Recorded MD step, shared against separate: 216 atoms 262 / 276 us, 1,000 394 / 402, 2,744
  // 774 / 785, 8,000 1,816 / 1,831; from 10,164 atoms to 262,144 (8.4 M edges) within the runs' spread of 1 %.
  const bool merged = stages == 31 && !p.host_marks;
  const bool merged_back = merged && E <= (int64_t(4) << 20);

  // ---------------------------------------------------------------- stage 1
  // one graph: the readout's blocks leave their sums; several: they add to the graphs' sums
  const int64_t* batch = p.graphs > 1 ? p.batch : nullptr;
  const int64_t parts = batch ? 0 : tail_blocks(n);
  double* energy = buffer<double>(parts > p.graphs ? parts : p.graphs);
  float* u0 = buffer(N * kC);
  call(1, -1, 1, [&] {
    EmbedArgs a{p.numbers, p.species_table, p.species_table_size, p.species, p.up0_table, u0, energy, p.graphs, N, p.batch, p.status};
    const int64_t threads = 16 * N > p.graphs ? 16 * N : p.graphs;
    if (threads > 0) launch_after(embed_kernel, (unsigned)((threads + 255) / 256), 256, 0, st, a);
    return finish_launch("sweep_embed");
  });
  if (p.watch_count > 0)
    call(1, -1, 1, [&] {
      launch_after(watch_kernel, (unsigned)p.watch_count, kWatchThreads, 0, st, p.watch_tiles, p.watch_copy, p.status);
      return finish_launch("sweep_watch");
    });
  const int64_t *dst_rowptr = p.dst_rowptr, *dst_order = p.dst_order, *src_rowptr = p.src_rowptr, *src_order = p.src_order;
  if (!dst_rowptr || !src_rowptr) {
    CsrPair pair{};
    int sets = 0;
    const int64_t words = csr_scratch_elems(N, E);
    int64_t* scratch = buffer<int64_t>(2 * words);
    auto add = [&](const int64_t* keys, int32_t* flag, const int64_t*& rowptr, const int64_t*& order) {
      int64_t* r = buffer<int64_t>(N + 1);
      int64_t* o = buffer<int64_t>(E);
      pair.set[sets] = csr_set(keys, N, E, r, o, flag, scratch + sets * words);
      ++sets;
      rowptr = r;
      order = o;
    };
    if (!dst_rowptr) add(p.dst, p.status + 1, dst_rowptr, dst_order);
    if (!src_rowptr) add(p.src, p.status + 2, src_rowptr, src_order);
    // the tile totals of both sets sit behind the second set's words
    int64_t* sums = buffer<int64_t>(sets * (prefix_tiles(N) + 1));
    call(1, -1, 5, [&] { return csr_build(pair, sets, N, E, sums, st); });
    if (p.host_status)
      call(1, -1, 0, [&] {         // the caller looks at the flags when the sweep is queued, long before it has run
        cudaMemcpyAsync(p.host_status, p.status, 3 * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        cudaEventRecord(static_cast<cudaEvent_t>(p.host_status_event), st);
        return finish_launch("sweep_status");
      });
    release(scratch);
    release(sums);
  }
  GeoArgs geo{};
  geo.pos = p.pos; geo.src = p.src; geo.dst = p.dst; geo.shifts = p.shifts; geo.cells = p.cells; geo.batch = p.batch;
  geo.graphs = p.graphs;
  for (int k = 0; k < 3; ++k) geo.box[k] = float(p.box[k]);
  geo.r_max = float(p.r_max); geo.num_basis = int(p.num_basis); geo.p = int(p.poly_p); geo.E = E;
  geo.gate_row = paired ? p.gate_row : nullptr; geo.rep = p.rep;
  geo.sh = buffer(9 * E);
  geo.geo = buffer<float4>(E);
  geo.N = N;
  const int64_t *src = p.src, *dst = p.dst;
  if (p.numbers) {
    src = geo.safe_src = buffer<int64_t>(E);
    dst = geo.safe_dst = buffer<int64_t>(E);
  }
  geo.rb = buffer(U * p.num_basis);
  const unsigned geo_blocks = (unsigned)((E + kGeoThreads - 1) / kGeoThreads);
  call(1, -1, 1, [&] {
    if (E > 0) launch_after(geometry_kernel, geo_blocks, kGeoThreads, 0, st, geo);
    return finish_launch("sweep_geometry");
  });
  float* pre[2][3];
  for (auto& layer : pre)
    for (float*& z : layer) z = buffer(U * kC);
  auto hidden_forward = [&](int first, int count) {
    chain::Args a{};
    a.stacks = count;
    for (int k = 0; k < count; ++k) {
      const ictc_sweep_layer& L = p.layer[first + k];
      float** z = pre[first + k];
      a.stack[k] = chain::Stack{geo.rb, L.w0, L.hid[0], L.hid[1], z[0], z[1], z[2], nullptr};
    }
    a.limit = p.live; a.E = U; a.nb = int(p.num_basis);
    return U > 0 ? chain::launch_forward(a, st) : 0;
  };
  call(1, label(kHiddenFwd, 0), 1, [&] { return hidden_forward(0, merged ? 2 : 1); });

  // receiver sweep of one interaction: gates from the hidden state, message rows
  float* gate_table[2] = {nullptr, nullptr};
  auto graph_forward = [&](int stage, int layer, const float* x, float* out) {
    const ictc_sweep_layer& L = p.layer[layer];
    const int64_t width = layer == 0 ? W0 : W1;
    if (E == 0) return clear(stage, out, n * width);
    if (table) {
      gate_table[layer] = buffer(U * L.num_gates);
      if (U > 0) gates(stage, layer, pre[layer][2], gate_table[layer], U, nullptr, nullptr, p.live);
      call(stage, label(kGraphFwd, layer), 1, [&] {
        return ictc_tp_graph_forward_shared(spec[layer], kC, n, E, x, geo.sh, L.path_weight, gate_table[layer], geo.gate_row,
                                            src, dst_rowptr, dst_order, nullptr, out, st);
      });
      return;
    }
    float* buf = buffer(p.chunk_capacity_dst * L.num_gates);
    for (int64_t r0 = 0; r0 < n; r0 += chunk_rows(n)) {
      const int64_t r1 = r0 + chunk_rows(n) < n ? r0 + chunk_rows(n) : n;
      gates(stage, layer, pre[layer][2], buf, p.chunk_capacity_dst, geo.gate_row, dst_rowptr + r0, dst_rowptr + r1);
      call(stage, label(kGraphFwd, layer), 1, [&] {
        return tp_graph_forward_chunk(n, spec[layer], kC, r1 - r0, x, geo.sh, L.path_weight, buf, nullptr, dst_rowptr + r0,
                                           p.chunk_capacity_dst, src, dst_rowptr + r0, nullptr, nullptr, out + r0 * width,
                                           st);
      });
    }
    release(buf);
  };
  auto contraction = [&](int stage, int layer, const float* x, float* y) {
    call(stage, label(kContraction, layer), 1, [&] {
      return ictc_sc_forward(2, layer == 0 ? 2 : 0, kC, n, int(p.num_species), 1, x, p.species, p.layer[layer].bank, y, st);
    });
  };
  auto contraction_adjoint = [&](int stage, int layer, const float* x, const float* gy, float* gx) {
    call(stage, label(kContraction, layer), 1, [&] {
      return ictc_sc_adjoint(2, layer == 0 ? 2 : 0, kC, n, int(p.num_species), 1, x, p.species, p.layer[layer].bank, gy, gx,
                             nullptr, nullptr, st);
    });
  };

  float* features = p.features ? p.features : buffer(N * W0);
  float* feature_grad = p.feature_grad ? p.feature_grad : buffer(N * W0);
  float* M0 = buffer(n * W0);
  graph_forward(1, 0, u0, M0);
  float* m0 = buffer(n * W0);
  linear(1, 0, L0.ml, n, M0, W0, true, m0, W0, false);
  contraction(1, 0, m0, M0);                                   // M0 now holds the product
  linear(1, 0, L0.pl, n, M0, W0, false, features, W0, false, p.sc0_table, p.species, n);
  release(M0);

  // ---------------------------------------------------------------- stage 2
  if (!merged) call(2, label(kHiddenFwd, 1), 1, [&] { return hidden_forward(1, 1); });

  // ---------------------------------------------------------------- stage 4
  float* u1 = buffer(N * W0);
  linear(4, 1, L1.up, N, features, W0, false, u1, W0, false);
  float* M1 = buffer(n * W1);
  graph_forward(4, 1, u1, M1);
  float* m1 = buffer(n * W0);
  linear(4, 1, L1.ml, n, M1, W1, true, m1, W0, false);
  release(M1);
  float *y1 = buffer(n * kC), *dy1 = buffer(n * kC), *dh = buffer(n * kC);
  contraction(4, 1, m1, y1);
  call(4, -1, 1, [&] {
    TailArgs a{y1, features, W0, p.species, p.readout_rp, p.readout_rs, p.readout_w2, p.readout_ro0, int(p.hidden),
               p.row_mask, batch, p.graphs, int(p.mask_atomic), p.atomic, energy, dy1, dh, n};
    if (n > 0) launch_after(tail_kernel, (unsigned)tail_blocks(n), kTailWarps * 32, 0, st, a, tail_nodes(n));
    return finish_launch("sweep_tail");
  });
  float* dm = buffer(n * W0);
  contraction_adjoint(4, 1, m1, dy1, dm);
  release(m1);
  release(y1);
  release(dy1);
  float* v = buffer(n * W1);
  linear(4, 1, L1.ml_b, n, dm, W0, false, v, W1, true);
  release(dm);

  // sender sweep of one interaction: dx (optional), the harmonics' gradient and the gradient of silu(z3) per edge; the
  // gate gradients exist per chunk only
  const int64_t* gates_by_position = nullptr;
  auto graph_adjoint = [&](int stage, int layer, const float* x, const float* cot, float* dx, float* dsh, float* da3) {
    const ictc_sweep_layer& L = p.layer[layer];
    if (E == 0) {
      if (dx) clear(stage, dx, N * W0);
      return;
    }
    const int64_t xw = layer == 0 ? kC : W0, step = chunk_rows(N);
    const int64_t cap = step < N ? p.chunk_capacity_src : (E > 0 ? E : 1);
    float* dg = buffer(cap * L.num_gates);
    float* gbuf = table ? nullptr : buffer(cap * L.num_gates);
    const float* g = table ? gate_table[layer] : gbuf;
    for (int64_t s0 = 0; s0 < N; s0 += step) {
      const int64_t s1 = s0 + step < N ? s0 + step : N;
      const int64_t *b = src_rowptr + s0, *en = src_rowptr + s1;
      if (!table) gates(stage, layer, pre[layer][2], gbuf, cap, gates_by_position, b, en);
      call(stage, label(kGraphAdj, layer), 1, [&] {
        return tp_graph_adjoint_chunk(N, spec[layer], kC, s1 - s0, x + s0 * xw, geo.sh, L.path_weight, g,
                                           table ? geo.gate_row : nullptr, table ? 0 : 1, table ? nullptr : b,
                                           table ? 0 : cap, dst, b, src_order, nullptr, cot, dx ? dx + s0 * xw : nullptr,
                                           dsh, dg, b, cap, st);
      });
      call(stage, label(kGateBwd, layer), 1, [&] {
        gg::Args a{};
        a.segments = 1;
        a.seg[0] = gg::segment(dg, L.w3t, da3, cap, int(L.num_gates / kC), 1, L.num_gates, 1, kC);
        a.limit = en; a.begin = b; a.out_index = src_order;
        return gg::launch_backward(a, st);
      });
    }
    release(dg);
    if (gbuf) release(gbuf);
    if (table) release(gate_table[layer]);
  };
  auto hidden_backward = [&](int first, int count, const float* const* da3, float* const* drb) {
    chain::Args a{};
    a.stacks = count;
    for (int k = 0; k < count; ++k) {
      const ictc_sweep_layer& L = p.layer[first + k];
      float** z = pre[first + k];
      a.stack[k] = chain::Stack{da3[k], L.w0, L.hid_t[1], L.hid_t[0], z[0], z[1], z[2], drb[k]};
    }
    a.in_a = p.rep; a.in_b = p.other; a.limit = p.live; a.E = U; a.nb = int(p.num_basis);
    return U > 0 ? chain::launch_backward(a, st) : 0;
  };
  if (!table) {
    // gate row of the edge at every position of the sender order
    if (paired) {
      int64_t* by_pos = buffer<int64_t>(E);
      call(4, -1, 1, [&] { return gather_index(geo.gate_row, src_order, E, by_pos, st); });
      gates_by_position = by_pos;
    } else {
      gates_by_position = src_order;
    }
  }
  float *dsh[2], *da3[2], *drb[2];
  for (int k = 0; k < 2; ++k) drb[k] = buffer(U * p.num_basis);
  dsh[1] = buffer(9 * E);
  da3[1] = buffer(E * kC);
  float* du1 = buffer(N * W0);
  graph_adjoint(4, 1, u1, v, du1, dsh[1], da3[1]);
  release(v);
  release(u1);
  linear(4, 1, L1.up_b, N, du1, W0, false, feature_grad, W0, false, dh, nullptr, n);
  release(du1);

  // ---------------------------------------------------------------- stage 8
  if (!merged_back) {
    call(8, label(kHiddenBwd, 1), 1, [&] { return hidden_backward(1, 1, da3 + 1, drb + 1); });
    release(da3[1]);
  }

  // ---------------------------------------------------------------- stage 16
  float *dy0 = buffer(n * W0), *dm0 = buffer(n * W0);
  linear(16, 0, L0.pl_b, n, feature_grad, W0, false, dy0, W0, false);
  contraction_adjoint(16, 0, m0, dy0, dm0);
  linear(16, 0, L0.ml_b, n, dm0, W0, false, dy0, W0, true);
  release(dm0);
  dsh[0] = buffer(9 * E);
  da3[0] = buffer(E * kC);
  graph_adjoint(16, 0, u0, dy0, nullptr, dsh[0], da3[0]);
  call(16, label(kHiddenBwd, 0), 1, [&] {
    return merged_back ? hidden_backward(0, 2, da3, drb) : hidden_backward(0, 1, da3, drb);
  });
  float4* dvec = buffer<float4>(E);
  for (int k = 0; k < 2; ++k) {
    geo.dsh[k] = dsh[k];
    geo.drb[k] = drb[k];
  }
  geo.dvec = dvec;
  call(16, -1, 1, [&] {
    if (E > 0) launch_after(geometry_backward_kernel, geo_blocks, kGeoThreads, 0, st, geo);
    return finish_launch("sweep_geometry_backward");
  });
  call(16, -1, 1, [&] {
    GradArgs a{N, n, dst_rowptr, dst_order, src_rowptr, src_order, dvec, float(p.gradient_sign), p.gradient, energy,
               p.energy, p.graphs, parts};
    const int64_t threads = 8 * N > p.graphs ? 8 * N : p.graphs;
    if (threads > 0)
      launch_after(position_gradient8_kernel, (unsigned)((threads + kGradThreads - 1) / kGradThreads), kGradThreads, 0, st, a);
    return finish_launch("sweep_position_gradient");
  });
  return rc;
}

static int check(const ictc_sweep* p) {
  if (!p || p->n_local < 0 || p->n_owned < 0 || p->n_owned > p->n_local || p->edges < 0 || p->edges > 2147483647LL ||
      p->pair_rows < 0 || p->graphs < 1 || p->num_species < 1 || p->num_basis < 1 || p->num_basis > 8 || p->poly_p < 2 ||
      p->hidden < 1 || !(p->r_max > 0) || p->chunk_rows < 0 || p->watch_count < 0 || p->watch_count > 2147483647LL) {
    set_error("sweep: sizes");
    return ICTC_ERR_BAD_ARG;
  }
  return ICTC_OK;
}

// Weights and buffers that are read in pieces of 8, 16 or 32 bytes.
static int check_pointers(const ictc_sweep* p) {
  uintptr_t bits = 0;
  bool null = false;
  const auto need = [&](const void* at, int bytes) {
    null |= !at;
    bits |= reinterpret_cast<uintptr_t>(at) & (bytes - 1);
  };
  const auto may = [&](const void* at, int bytes) { bits |= reinterpret_cast<uintptr_t>(at) & (bytes - 1); };
  need(p->work, 32); may(p->features, 32); may(p->feature_grad, 32);
  need(p->up0_table, 16); need(p->sc0_table, 4);
  need(p->readout_rp, 8); need(p->readout_rs, 8); need(p->readout_ro0, 8); need(p->readout_w2, 4);
  for (int k = 0; k < 2; ++k) {
    const ictc_sweep_layer& L = p->layer[k];
    need(L.w0, 4); need(L.w3, 16); need(L.w3t, 16); need(L.bank, 4);
    for (int i = 0; i < 2; ++i) { need(L.hid[i], 16); need(L.hid_t[i], 16); }
    for (int l = 0; l < 3; ++l) {
      need(L.ml[l], 16); need(L.ml_b[l], 16);
      need(k ? L.up[l] : L.pl[l], 16); need(k ? L.up_b[l] : L.pl_b[l], 16);
    }
  }
  if (null || bits) {
    set_error(null ? "sweep: NULL weights or workspace"
                   : "sweep: workspace and feature buffers must be 32-byte, packed weights and up0_table 16-byte, the readout "
                     "matrices 8-byte aligned");
    return ICTC_ERR_BAD_ARG;
  }
  return ICTC_OK;
}

}  // namespace sweep
}  // namespace ictc

using namespace ictc;

extern "C" {

int64_t ictc_sweep_struct_bytes(void) { return int64_t(sizeof(ictc_sweep)); }

static int64_t sweep_bytes(const ictc_sweep& p, int stages) {
  ictc_sweep dry = p;
  dry.work = nullptr;
  sweep::Runner r(dry, stages, nullptr, true);
  r.run();
  return r.peak();
}

int64_t ictc_sweep_workspace(const ictc_sweep* p) {
  if (sweep::check(p)) return -1;
  // with all stages the interactions share launches and buffers live longer: the larger of both placements
  try {
    const int64_t one = sweep_bytes(*p, 1), all = sweep_bytes(*p, 31);
    return one > all ? one : all;
  } catch (const std::exception& e) {          // the placement's lists: host memory is exhausted
    set_error("sweep: %s", e.what());
    return -1;
  }
}

int ictc_sweep_run(const ictc_sweep* p, int stages, void* stream) {
  if (int rc = sweep::check(p)) return rc;
  if (!p->pos || !p->species || !p->energy || (p->n_owned > 0 && !p->atomic) || !p->gradient || !p->status ||
      !p->work || (p->edges > 0 && (!p->src || !p->dst))) {
    set_error("sweep: NULL buffer");
    return ICTC_ERR_BAD_ARG;
  }
  if (int rc = sweep::check_pointers(p)) return rc;
  if ((stages & 31) != 31 && (!p->features || !p->feature_grad)) {
    set_error("sweep: features and feature_grad are needed when the stages run one by one");
    return ICTC_ERR_BAD_ARG;
  }
  try {
    if (p->work_bytes < sweep_bytes(*p, stages & 31)) {
      set_error("sweep: workspace of %lld bytes is too small", (long long)p->work_bytes);
      return ICTC_ERR_BAD_ARG;
    }
    sweep::Runner r(*p, stages & 31, (cudaStream_t)stream, false);
    return r.run();
  } catch (const std::exception& e) {
    set_error("sweep: %s", e.what());
    return ICTC_ERR_BAD_ARG;
  }
}

}  // extern "C"
