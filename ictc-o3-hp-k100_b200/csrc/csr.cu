// CSR topology from an unsorted int64 key vector (receiver or sender of every edge).
//
// rowptr = exclusive prefix sum of the key histogram; order = edge ids grouped by key, ascending
// inside a row (what a stable sort by key would give), so every reduction that walks a row has a
// fixed summation order.  The histogram's atomic hands every edge a place in its row; the
// order is then made canonical by ranking the edge ids inside each row.  When the keys are
// already non-decreasing the order is the identity and the ranking pass exits immediately.
// The receiver and the sender CSR of an edge list are built by the same launches (blockIdx.y).
// Replaces ictc_o3/backends/k100/generated_csr_forward.py:17-31 (bincount + cumsum + stable argsort)
// and the device counting sort ictc_o3/ops/message_topology.py:15-36.
#include <mutex>
#include "csr.cuh"
#include "scan.cuh"

namespace ictc {

__global__ void csr_init_kernel(CsrPair p, int64_t N) {
  const CsrSet& c = p.set[blockIdx.y];
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i < N) c.counts[i] = 0;
  if (i == 0) {
    *c.flag = 1;
    c.rowptr[0] = 0;
  }
}

// `place` = how many edges of the row came earlier
__global__ void csr_count_kernel(CsrPair p, int64_t E, int64_t N) {
  const CsrSet& c = p.set[blockIdx.y];
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (e >= E) return;
  const int64_t k = c.keys[e];
  if (k < 0 || k >= N) {
    atomicMin(c.flag, -1);
    return;
  }
  if (e > 0 && c.keys[e - 1] > k) atomicMin(c.flag, 0);
  c.place[e] = int64_t(atomicAdd(reinterpret_cast<unsigned long long*>(c.counts + k), 1ULL));
}

struct CsrLoad {
  CsrPair p;
  __device__ int64_t operator()(int64_t i) const { return p.set[blockIdx.y].counts[i]; }
};
struct CsrStore {
  CsrPair p;
  __device__ void operator()(int64_t i, int64_t before, int64_t v) const { p.set[blockIdx.y].rowptr[i + 1] = before + v; }
};

__global__ void csr_fill_kernel(CsrPair p, int64_t E, int64_t N) {
  const CsrSet& c = p.set[blockIdx.y];
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (e >= E) return;
  if (*c.flag == 1) {
    c.order[e] = e;
    return;
  }
  const int64_t k = c.keys[e];
  if (k >= 0 && k < N) c.order[c.rowptr[k] + c.place[e]] = e;
}

// In-row ordering: `order` holds the ids of a row in arrival order; they are put in ascending order (a stable sort of the
// whole list).  The row's part of `place`, no longer needed, takes the unsorted copy.
//   rows of at most kLongRow edges: one warp per row ranks every id against the row (quadratic, but the row is
//     short and stays in L1);
//   longer rows: the block sorts the ids in place with a bitonic network whose every compare-exchange
//     keeps the minimum at the lower index, so positions beyond the row's end act as +infinity and are never
//     touched; O(L log^2 L) instead of O(L^2), which bounds the run time of degenerate inputs (few rows, a
//     million edges).
constexpr int64_t kLongRow = 2048;
constexpr int kRankRows = 8;

__global__ void __launch_bounds__(kRankRows * 32) csr_rank_kernel(CsrPair p, int64_t N) {
  __shared__ bool is_long[kRankRows];
  const int zero = pdl_enter();
  const CsrSet& c = p.set[blockIdx.y];
  if (*c.flag == 1) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t first = int64_t(blockIdx.x) * kRankRows + zero, row = first + warp;
  const int64_t begin = row < N ? c.rowptr[row] : 0, end = row < N ? c.rowptr[row + 1] : 0;
  if (lane == 0) is_long[warp] = end - begin > kLongRow;
  if (end - begin <= kLongRow) {
    for (int64_t a = begin + lane; a < end; a += 32) c.place[a] = c.order[a];
    __syncwarp();
    for (int64_t a = begin + lane; a < end; a += 32) {
      const int64_t mine = c.place[a];
      int64_t rank = 0;
      for (int64_t b = begin; b < end; ++b) rank += c.place[b] < mine;
      c.order[begin + rank] = mine;
    }
  }
  __syncthreads();
  for (int r = 0; r < kRankRows; ++r) {
    if (!is_long[r]) continue;
    const int64_t at = c.rowptr[first + r], len = c.rowptr[first + r + 1] - at;
    int64_t* v = c.order + at;
    int64_t padded = 1;
    while (padded < len) padded <<= 1;
    for (int64_t k = 2; k <= padded; k <<= 1) {
      for (int64_t j = k >> 1; j > 0; j >>= 1) {
        for (int64_t i = threadIdx.x; i < padded; i += blockDim.x) {
          const int64_t l = (j == (k >> 1)) ? (i ^ (k - 1)) : (i ^ j);     // first step of a stage mirrors the block
          if (l > i && l < len) {
            const int64_t x = v[i], y = v[l];
            if (x > y) { v[i] = y; v[l] = x; }
          }
        }
        __syncthreads();
      }
    }
  }
}

int64_t csr_scratch_elems(int64_t N, int64_t E) { return N + E + prefix_tiles(N) + 2; }

CsrSet csr_set(const int64_t* keys, int64_t N, int64_t E, int64_t* rowptr, int64_t* order, int32_t* flag, int64_t* scratch) {
  return CsrSet{keys, rowptr, order, flag, scratch, scratch + N};
}

int csr_build(const CsrPair& p, int sets, int64_t N, int64_t E, int64_t* sums, cudaStream_t st) {
  launch_after(csr_init_kernel, dim3((unsigned)(N / 256 + 1), sets), 256, 0, st, p, N);
  if (E > 0) launch_after(csr_count_kernel, dim3((unsigned)((E + 255) / 256), sets), 256, 0, st, p, E, N);
  prefix_sum<int64_t>(N, CsrLoad{p}, CsrStore{p}, sums, false, st, sets);
  if (E > 0) {
    launch_after(csr_fill_kernel, dim3((unsigned)((E + 255) / 256), sets), 256, 0, st, p, E, N);
    if (N > 0)
      launch_after(csr_rank_kernel, dim3((unsigned)((N + kRankRows - 1) / kRankRows), sets), kRankRows * 32, 0, st, p, N);
  }
  return finish_launch("csr_build");
}

// ---- built-in scratch for callers that cannot allocate (see ictc_csr_build_static) ----------------
constexpr int64_t kStaticMaxNodes = 1 << 16;   // 65,536 rows
constexpr int64_t kStaticMaxEdges = 1 << 20;   // 1,048,576 edges
constexpr int64_t kStaticElems = kStaticMaxNodes + kStaticMaxEdges + 64;   // + scan totals and padding
static __device__ __align__(256) int64_t g_csr_static_scratch[kStaticElems];   // ~8.9 MB per device

}  // namespace ictc

using namespace ictc;

extern "C" {

int64_t ictc_csr_scratch_bytes(int64_t N, int64_t E) {
  if (N < 0 || E < 0) return 0;
  return 8 * csr_scratch_elems(N, E);
}

// Device address of the built-in scratch on the current device, looked up on first use per device.
static int static_scratch(void** out) {
  static std::mutex lock;
  static void* cache[64] = {};
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("csr_build_static: cannot identify the current device");
    return ICTC_ERR_LAUNCH;
  }
  std::lock_guard<std::mutex> guard(lock);
  if (!cache[dev]) {
    void* p = nullptr;
    // In host code the array name is only a handle; the kernels need its address on THIS device.
    err = cudaGetSymbolAddress(&p, g_csr_static_scratch);
    if (err != cudaSuccess || !p) {
      set_error("csr_build_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(err));
      return ICTC_ERR_LAUNCH;
    }
    cache[dev] = p;
  }
  *out = cache[dev];
  return ICTC_OK;
}

int ictc_csr_build(const int64_t* keys, int64_t N, int64_t E, int64_t* rowptr, int64_t* order, int32_t* sorted_flag,
                   void* scratch, void* stream);

int ictc_csr_build_static(const int64_t* keys, int64_t N, int64_t E, int64_t* rowptr, int64_t* order,
                          int32_t* sorted_flag, void* stream) {
  if (N < 0 || E < 0) { set_error("csr_build_static: negative size"); return ICTC_ERR_BAD_ARG; }
  if (N > kStaticMaxNodes || E > kStaticMaxEdges) {
    set_error("csr_build_static: %lld rows / %lld edges exceed the built-in scratch (at most %lld rows and %lld "
              "edges); use ictc_csr_build with caller-owned scratch", (long long)N, (long long)E,
              (long long)kStaticMaxNodes, (long long)kStaticMaxEdges);
    return ICTC_ERR_TOO_LARGE;
  }
  if (ictc_csr_scratch_bytes(N, E) > kStaticElems * 8) {
    set_error("csr_build_static: internal size bound violated");
    return ICTC_ERR_TOO_LARGE;
  }
  void* scratch = nullptr;
  if (int rc = static_scratch(&scratch)) return rc;
  return ictc_csr_build(keys, N, E, rowptr, order, sorted_flag, scratch, stream);
}

struct ScanLoad {
  const int64_t* v;
  __device__ int64_t operator()(int64_t i) const { return v[i]; }
};
struct ScanStore {
  int64_t* v;
  __device__ void operator()(int64_t i, int64_t before, int64_t x) const { v[i] = before + x; }
};

// Inclusive scan of an int64 device vector in place (used by the neighbour build for its row offsets).
int64_t ictc_scan_scratch_bytes(int64_t n) { return n < 0 ? 0 : 8 * (prefix_tiles(n) + 2); }
int ictc_inclusive_scan_i64(int64_t* data, int64_t n, void* scratch, void* stream) {
  if (n < 0 || (n > 0 && (!data || !scratch))) { set_error("scan: invalid arguments"); return ICTC_ERR_BAD_ARG; }
  if (prefix_tiles(n) > 2147483647LL) { set_error("scan: too long"); return ICTC_ERR_TOO_LARGE; }
  prefix_sum<int64_t>(n, ScanLoad{data}, ScanStore{data}, reinterpret_cast<int64_t*>(scratch), true, (cudaStream_t)stream);
  return finish_launch("inclusive_scan");
}

int ictc_csr_static_limits(int64_t* max_nodes, int64_t* max_edges) {
  if (max_nodes) *max_nodes = kStaticMaxNodes;
  if (max_edges) *max_edges = kStaticMaxEdges;
  return ICTC_OK;
}

int ictc_csr_build(const int64_t* keys, int64_t N, int64_t E, int64_t* rowptr, int64_t* order, int32_t* sorted_flag,
                   void* scratch, void* stream) {
  if (N < 0 || E < 0) { set_error("csr_build: negative size"); return ICTC_ERR_BAD_ARG; }
  if (!rowptr || !sorted_flag || !scratch || (E > 0 && (!keys || !order))) {
    set_error("csr_build: NULL buffer");
    return ICTC_ERR_BAD_ARG;
  }
  if ((N + 256) / 256 > 2147483647LL || (E + 255) / 256 > 2147483647LL || (N + 7) / 8 > 2147483647LL) {
    set_error("csr_build: too many rows");
    return ICTC_ERR_TOO_LARGE;
  }
  int64_t* words = reinterpret_cast<int64_t*>(scratch);
  CsrPair p{};
  p.set[0] = csr_set(keys, N, E, rowptr, order, sorted_flag, words);
  return csr_build(p, 1, N, E, words + N + E, (cudaStream_t)stream);
}

}  // extern "C"
