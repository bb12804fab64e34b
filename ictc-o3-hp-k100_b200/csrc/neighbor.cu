// Cell-list neighbour build and velocity-Verlet helpers for the MD step.
//
// Edge convention of the reference's graph fill (lammps_user_mfftorch/src/USER-MFFTORCH/
// pair_mff_torch_kokkos.cpp:661-871): a full neighbour list, edge (src = j neighbour, dst = i centre)
// for every ordered pair with |r_i - r_j + S*box|^2 <= cutoff^2, centres restricted to the first
// `num_centres` rows (owned atoms), edges ordered by (dst, src, shift_x, shift_y, shift_z) — the
// reference's canonical order (:897-911).  The distance test is evaluated in double precision on the
// fp32 coordinates with individually rounded operations (no fused multiply-add), so it is bit-for-bit
// the same predicate a plain CPU loop evaluates.
//
// Phases: (1) cell of every atom, counting sort of the atoms by cell, (2) per-centre neighbour count, (3) exclusive
// scan, (4) per-centre fill + in-row sort by (src, shift), (5) reverse edges and pair rows.
#include "scan.cuh"

namespace ictc {

struct NbGrid {
  double lo[3];       // origin of the cell grid
  double box[3];      // periodic lengths (used for image shifts)
  double inv_w[3];    // 1 / cell width
  int nc[3];          // cells per axis
  int periodic[3];
  double cutsq;
  float rc, span;     // cutoff; box lengths plus three cell widths (bound of the coordinate differences, see nb_visit)
};

__device__ __forceinline__ void cell_of(const NbGrid& g, const float* p, int (&c)[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int v = int(floor((double(p[a]) - g.lo[a]) * g.inv_w[a]));
    c[a] = v < 0 ? 0 : (v >= g.nc[a] ? g.nc[a] - 1 : v);
  }
}

// Counting sort by cell: the histogram's atomic hands every atom its place inside the cell, so that the fill needs no
// atomics.  The order inside a cell is arbitrary; the edge list does not depend on it (rows are sorted by key).
__global__ void nb_bin_count_kernel(NbGrid g, const float* __restrict__ pos, int64_t n, int* count, int2* where) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i >= n) return;
  int c[3];
  cell_of(g, pos + 3 * i, c);
  const int cell = (c[0] * g.nc[1] + c[1]) * g.nc[2] + c[2];
  where[i] = make_int2(cell, atomicAdd(count + cell, 1));
}

// atoms[] = (x, y, z, index) grouped by cell: a candidate costs one 16-byte load, contiguous over the lanes
__global__ void nb_bin_fill_kernel(const float* __restrict__ pos, int64_t n, const int* __restrict__ cell_start,
                                   const int2* __restrict__ where, float4* atoms) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i >= n) return;
  const int2 w = where[i];
  atoms[cell_start[w.x] + w.y] = make_float4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], __int_as_float(int(i)));
}

// One warp per centre.  The 27 cells around it are one list of candidates (lane l describes cell l; prefix sums in
// shared memory), which the lanes walk 32 at a time: about 8 rounds for 250 candidates.  One thread per centre, the
// former split, left 8 of 148 SMs busy at 1,000 atoms and spent its time on dependent loads.  f(hit, key) is called by
// all lanes of the warp together.  Both passes: 1,000 atoms 375 -> 17 us, 131,072 atoms 766 -> 345 us (issue slots 73 %
// busy: the cell walk, not memory, bounds it).
constexpr int kNbWarps = 4;
struct NbCells { int start[27], first[28]; float shift[27][3]; unsigned char code[27]; };

template <class F>
__device__ __forceinline__ void nb_visit(const NbGrid& g, const float* __restrict__ pos,
                                         const int* __restrict__ cell_start, const float4* __restrict__ atoms,
                                         int64_t i, int lane, NbCells& cells, F f) {
  const float* p = pos + 3 * i;
  int c[3];
  cell_of(g, p, c);
  int count = 0;
  if (lane < 27) {
    const int o[3] = {lane / 9 - 1, (lane / 3) % 3 - 1, lane % 3 - 1};
    int at[3], s[3] = {0, 0, 0};
    bool inside = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      at[a] = c[a] + o[a];
      if (at[a] < 0 || at[a] >= g.nc[a]) {
        if (!g.periodic[a]) inside = false;
        s[a] = at[a] < 0 ? -1 : 1;
        at[a] -= s[a] * g.nc[a];
      }
    }
    if (inside) {
      const int cell = (at[0] * g.nc[1] + at[1]) * g.nc[2] + at[2];
      cells.start[lane] = cell_start[cell];
      count = cell_start[cell + 1] - cells.start[lane];
    }
    cells.code[lane] = (unsigned char)(((1 - s[0]) * 3 + (1 - s[1])) * 3 + (1 - s[2]));     // of the shift -s
#pragma unroll
    for (int a = 0; a < 3; ++a) cells.shift[lane][a] = float(-s[a] * g.box[a]);
  }
  // Nearly every candidate is decided in single precision: beyond (below) a radius that is larger (smaller) than the
  // cutoff by more than the rounding of the coordinate differences (terms up to |r_i| + box + three cells, three
  // operations of 2^-24 each per axis) it is out (in).  The double-precision predicate decides the shell in between; its
  // conversions alone cost more than the rest of the loop when every candidate goes through it.
  const float rc = g.rc, shell = 1e-5f * rc + 2e-6f * (fabsf(p[0]) + fabsf(p[1]) + fabsf(p[2]) + g.span);
  const float outer = (rc + shell) * (rc + shell), inner = shell < rc ? (rc - shell) * (rc - shell) : -1.f;
  int inc = count;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += up;
  }
  if (lane < 27) cells.first[lane + 1] = inc;
  if (lane == 0) cells.first[0] = 0;
  const int total = __shfl_sync(0xffffffffu, inc, 31);
  __syncwarp();
  int cell = 0;
  for (int base = 0; base < total; base += 32) {
    const int k = base + lane;
    bool hit = false;
    int64_t key = 0;
    if (k < total) {
      while (k >= cells.first[cell + 1]) ++cell;
      const float4 q = atoms[cells.start[cell] + (k - cells.first[cell])];
      const float fx = (p[0] - q.x) + cells.shift[cell][0], fy = (p[1] - q.y) + cells.shift[cell][1],
                  fz = (p[2] - q.z) + cells.shift[cell][2];
      const int64_t j = __float_as_int(q.w);
      const int code = cells.code[cell];
      key = j * 27 + code;
      const float near = fx * fx + fy * fy + fz * fz;
      hit = near <= inner;
      if (!hit && !(near > outer)) {
        // the image sits at r_j - shift * box: edge_vec = r_i - r_j + shift * box
        const double bx = (code / 9 - 1) * g.box[0], by = ((code / 3) % 3 - 1) * g.box[1], bz = (code % 3 - 1) * g.box[2];
        const double dx = __dadd_rn(__dadd_rn(double(p[0]), -double(q.x)), bx);
        const double dy = __dadd_rn(__dadd_rn(double(p[1]), -double(q.y)), by);
        const double dz = __dadd_rn(__dadd_rn(double(p[2]), -double(q.z)), bz);
        hit = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)) <= g.cutsq;
      }
      if (j == i && code == 13) hit = false;
    }
    f(hit, key);
  }
  __syncwarp();
}

// Counts of a row: all edges (low half) and the edges that represent their pair (high half), see nb_pair_kernel.
// Either output may be missing.
__global__ void __launch_bounds__(kNbWarps * 32) nb_count_kernel(NbGrid g, const float* __restrict__ pos,
                                                                 const int* __restrict__ cell_start,
                                                                 const float4* __restrict__ atoms, int64_t centres,
                                                                 int64_t* rowptr, uint2* packed) {
  __shared__ NbCells cells[kNbWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = int64_t(blockIdx.x) * kNbWarps + warp + pdl_enter();
  if (i >= centres) return;
  unsigned n = 0, self = 0, above = 0;
  nb_visit(g, pos, cell_start, atoms, i, lane, cells[warp], [&](bool hit, int64_t key) {
    if (!hit) return;
    const int64_t j = key / 27;
    ++n;
    self += j == i;
    above += j > i;
  });
  n = __reduce_add_sync(0xffffffffu, n);
  self = __reduce_add_sync(0xffffffffu, self);
  above = __reduce_add_sync(0xffffffffu, above);
  if (lane == 0) {
    if (rowptr) rowptr[i + 1] = n;
    if (rowptr && i == 0) rowptr[0] = 0;
    if (packed) packed[i] = make_uint2(n, above + self / 2);
  }
}

// Finds the row's keys again, sorts them by rank (rows are a few dozen keys long) and writes the edges.  Keys wait in
// shared memory for the ranking, those of rows longer than kNbStage in the row's part of `src`.
constexpr int kNbStage = 128;

__global__ void __launch_bounds__(kNbWarps * 32) nb_fill_kernel(NbGrid g, const float* __restrict__ pos,
                                                                const int* __restrict__ cell_start,
                                                                const float4* __restrict__ atoms, int64_t centres,
                                                                const int64_t* __restrict__ rowptr, int64_t capacity,
                                                                int64_t* src, int64_t* dst, float* shifts, int64_t* keys) {
  __shared__ NbCells cells[kNbWarps];
  __shared__ int64_t stage[kNbWarps][kNbStage];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = int64_t(blockIdx.x) * kNbWarps + warp + pdl_enter();
  if (i >= centres) return;
  const int64_t begin = rowptr[i], end = rowptr[i + 1];
  if (end > capacity || begin > end) return;   // offsets must have been clamped to the capacity
  const int len = int(end - begin);
  int64_t* raw = len <= kNbStage ? stage[warp] : src + begin;
  int found = 0;
  nb_visit(g, pos, cell_start, atoms, i, lane, cells[warp], [&](bool hit, int64_t key) {
    const unsigned vote = __ballot_sync(0xffffffffu, hit);
    const int at = found + __popc(vote & ((1u << lane) - 1));
    if (hit && at < len) raw[at] = key;        // row truncated by the capacity clamp: extra neighbours are dropped
    found += __popc(vote);
  });
  __syncwarp();
  for (int a = lane; a < len; a += 32) {
    const int64_t mine = raw[a];
    int rank = 0;
    for (int b = 0; b < len; ++b) rank += raw[b] < mine;
    keys[begin + rank] = mine;
  }
  __syncwarp();
  for (int a = lane; a < len; a += 32) {
    const int64_t key = keys[begin + a];
    const int code = int(key % 27);
    src[begin + a] = key / 27;
    dst[begin + a] = i;
    float* s = shifts + 3 * (begin + a);
    s[0] = float(code / 9 - 1);
    s[1] = float((code / 3) % 3 - 1);
    s[2] = float(code % 3 - 1);
  }
}

// Clamps row offsets to the capacity of fixed-size edge buffers (rows beyond it become empty, the row that
// straddles it is truncated) and raises *overflow when anything had to be clamped.  The flag is sticky (never
// cleared here) so that a host that looks only every few steps still sees an earlier overflow.
__global__ void nb_clamp_kernel(int64_t* rowptr, int64_t n1, int64_t capacity, int32_t* overflow) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n1) return;
  const int64_t v = rowptr[i];
  if (i == n1 - 1 && v > capacity) *overflow = 1;
  if (v > capacity) rowptr[i] = capacity;
}

// Fills the unused tail [count, capacity) of fixed-capacity edge buffers with inert edges so that every
// consumer can run over `capacity` rows without knowing the edge count on the host.
__global__ void nb_pad_kernel(const int64_t* __restrict__ count, int64_t capacity, int64_t pad_src, int64_t pad_dst,
                              int64_t* src, int64_t* dst, float* shifts, int32_t* overflow) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e == 0 && overflow) *overflow = *count > capacity ? 1 : 0;
  if (e >= capacity || e < *count) return;
  src[e] = pad_src;
  dst[e] = pad_dst;
  shifts[3 * e] = shifts[3 * e + 1] = shifts[3 * e + 2] = 0.f;
}

// ---- radial pairing --------------------------------------------------------------------------------
// Edge (j -> i, S) and its reverse (i -> j, -S) have bitwise the same length, so everything that depends
// on the length alone (radial basis, gate MLP) is evaluated once per pair.  `rev` finds the reverse edge by
// binary search in the sorted row of j; an edge is the pair's representative when it has no reverse in the
// list (sender is not a centre) or when its index is the smaller of the two.
__global__ void nb_pair_find_kernel(const int64_t* __restrict__ rowptr, const int64_t* __restrict__ dst,
                                    const int64_t* __restrict__ keys, int64_t centres, int64_t capacity,
                                    const int64_t* __restrict__ count, int64_t* rev, int64_t* flag) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= capacity) return;
  if (e >= *count) {
    rev[e] = -1;
    flag[e] = 0;
    return;
  }
  const int64_t key = keys[e];
  const int64_t j = key / 27, i = dst[e];
  int64_t r = -1;
  if (j < centres) {
    const int64_t want = i * 27 + (26 - key % 27);
    int64_t lo = rowptr[j], hi = rowptr[j + 1];
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid] < want) lo = mid + 1; else hi = mid;
    }
    if (lo < rowptr[j + 1] && keys[lo] == want) r = lo;
  }
  rev[e] = r;
  flag[e] = (r < 0 || e < r) ? 1 : 0;
}

// scan = inclusive prefix sum of the representative flags
__global__ void nb_pair_assign_kernel(const int64_t* __restrict__ scan, const int64_t* __restrict__ rev,
                                      int64_t capacity, int64_t unique_capacity, const int64_t* __restrict__ count,
                                      int64_t* gate_row, int64_t* rep_edge, int64_t* other_edge, int64_t* num_unique) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t n = *count < capacity ? *count : capacity;
  const int64_t total = n > 0 ? scan[n - 1] : 0;
  if (e == 0) *num_unique = total;
  if (e < capacity) {
    if (e < n) {
      const int64_t r = rev[e];
      const bool rep = r < 0 || e < r;
      const int64_t u = (rep ? scan[e] : scan[r]) - 1;
      // a pair table that is too small is reported through num_unique > unique_capacity; rows stay in range
      gate_row[e] = u < unique_capacity ? u : (unique_capacity > 0 ? unique_capacity - 1 : 0);
      if (rep && u < unique_capacity) {
        rep_edge[u] = e;
        other_edge[u] = r;
      }
    } else {
      gate_row[e] = 0;
    }
  }
  // rows of the pair table beyond the number of pairs point at the last (inert) edge slot
  if (e >= total && e < unique_capacity) {
    rep_edge[e] = capacity - 1;
    other_edge[e] = -1;
  }
}

// The same pairing where the list was just built and the number of representatives per row is known from the counting
// pass (u_row, exclusive prefix sums): inside a sorted row the representatives are the edges whose sender has the larger
// index, i.e. the end of the row (and of the edges between an atom and its own images the first half), so the pair row
// of an edge follows from its position in its own or its reverse's row and no scan over the edges is needed.  Also
// writes the inert edges behind the last one and, as `rev`, the sender order of a list in which every edge has its
// reverse: the edges that leave atom i are the reverses of those that arrive at it.
__global__ void nb_pair_kernel(const int64_t* __restrict__ rowptr, const int* __restrict__ u_row,
                               const int64_t* __restrict__ keys, int64_t centres, int64_t capacity,
                               int64_t unique_capacity, int64_t pad_src, int64_t* src, int64_t* dst, float* shifts,
                               int64_t* rev, int64_t* gate_row, int64_t* rep_edge, int64_t* other_edge) {
  const int zero = pdl_enter();
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + zero;
  const int64_t count = rowptr[centres + zero], total = u_row[centres + zero];
  if (e < capacity) {
    if (e < count) {
      const int64_t key = keys[e], j = key / 27, i = dst[e];
      const int code = int(key - j * 27);
      int64_t r = -1;
      if (j < centres) {
        const int64_t want = i * 27 + (26 - code), last = rowptr[j + 1];
        int64_t lo = rowptr[j], hi = last;
        while (lo < hi) {
          const int64_t mid = (lo + hi) >> 1;
          if (keys[mid] < want) lo = mid + 1; else hi = mid;
        }
        if (lo < last && keys[lo] == want) r = lo;
      }
      const bool rep = j > i || (j == i && code < 13);
      int64_t u;
      if (j != i) {
        const int64_t row = rep ? i : j, at = rep ? e : r;
        u = u_row[row + 1] - (rowptr[row + 1] - at);
      } else {
        int64_t first = rep ? e : r;
        u = u_row[i];
        while (first > rowptr[i] && keys[first - 1] / 27 == i) { --first; ++u; }
      }
      if (r < 0 && !rep) u = 0;             // only in a list that was cut off at the capacity
      u = u < 0 ? 0 : u;
      gate_row[e] = u < unique_capacity ? u : (unique_capacity > 0 ? unique_capacity - 1 : 0);
      rev[e] = r < 0 ? 0 : r;
      if (rep && u < unique_capacity) {
        rep_edge[u] = e;
        other_edge[u] = r;
      }
    } else {
      src[e] = pad_src;
      dst[e] = 0;
      shifts[3 * e] = shifts[3 * e + 1] = shifts[3 * e + 2] = 0.f;
      rev[e] = 0;
      gate_row[e] = 0;
    }
  }
  // rows of the pair table beyond the number of pairs point at the last (inert) edge slot
  if (e >= total && e < unique_capacity) {
    rep_edge[e] = capacity - 1;
    other_edge[e] = -1;
  }
}

// ---- velocity Verlet (positions in A, velocities in A/fs, forces in eV/A, masses in amu) ----------
constexpr float kAccel = 9.64853321e-3f;   // 1 eV/(A amu) in A/fs^2

__global__ void md_kick_drift_kernel(int64_t n, float dt, const float* __restrict__ force,
                                     const float* __restrict__ inv_mass, float* vel, float* pos, const float* box,
                                     int drift) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x + pdl_enter();
  if (i >= n) return;
  const float s = 0.5f * dt * kAccel * inv_mass[i];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float v = fmaf(s, force[3 * i + a], vel[3 * i + a]);
    vel[3 * i + a] = v;
    if (drift) {
      float x = fmaf(dt, v, pos[3 * i + a]);
      const float L = box[a];
      if (L > 0.f) {           // periodic axis: wrap into [0, L)
        if (x >= L) x -= L;
        if (x < 0.f) x += L;
        if (x >= L) x = 0.f;   // x was -tiny and x + L rounded to L
      }
      pos[3 * i + a] = x;
    }
  }
}

}  // namespace ictc

using namespace ictc;

extern "C" {

// scratch: atoms[N] float4 | where[N] int2 | packed[N] uint2 | sums[tiles] u64 | cell counts, cell_start[cells + 1],
// u_row[N + 1] int32
static int64_t nb_cells(const double* lo, const double* hi, double cutoff, int* nc) {
  int64_t total = 1;
  for (int a = 0; a < 3; ++a) {
    const double extent = hi[a] - lo[a];
    int n = int(floor(extent / cutoff));
    if (n < 1) n = 1;
    if (n > 1024) n = 1024;
    nc[a] = n;
    total *= n;
  }
  return total;
}

struct NbScratch {
  float4* atoms;
  int2* where;
  uint2* packed;
  unsigned long long* sums;
  int *cell_count, *cell_start, *u_row;
};

static int64_t nb_carve(void* scratch, int64_t N, int64_t cells, NbScratch* s) {
  char* p = reinterpret_cast<char*>(scratch);
  int64_t used = 0;
  auto take = [&](int64_t bytes) { char* at = p + used; used += (bytes + 15) / 16 * 16; return at; };
  s->atoms = reinterpret_cast<float4*>(take(16 * N));
  s->where = reinterpret_cast<int2*>(take(8 * N));
  s->packed = reinterpret_cast<uint2*>(take(8 * N));
  s->sums = reinterpret_cast<unsigned long long*>(take(8 * (prefix_tiles(N > cells ? N : cells) + 1)));
  s->cell_count = reinterpret_cast<int*>(take(4 * cells));
  s->cell_start = reinterpret_cast<int*>(take(4 * (cells + 1)));
  s->u_row = reinterpret_cast<int*>(take(4 * (N + 1)));
  return used;
}

int64_t ictc_neighbor_scratch_bytes(int64_t num_atoms, const double* host_lo, const double* host_hi, double cutoff) {
  if (num_atoms < 0 || !host_lo || !host_hi || !(cutoff > 0)) return 0;
  int nc[3];
  NbScratch s;
  return nb_carve(nullptr, num_atoms, nb_cells(host_lo, host_hi, cutoff, nc), &s) + 64;
}

static int nb_setup(int64_t N, const double* lo, const double* hi, const double* box, const int* periodic,
                    double cutoff, NbGrid* g, int64_t* cells) {
  if (N < 0 || !lo || !hi || !box || !periodic || !(cutoff > 0)) {
    set_error("neighbor: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  *cells = nb_cells(lo, hi, cutoff, g->nc);
  for (int a = 0; a < 3; ++a) {
    g->lo[a] = lo[a];
    g->box[a] = box[a];
    g->inv_w[a] = g->nc[a] / (hi[a] - lo[a]);
    g->periodic[a] = periodic[a];
    if (periodic[a] && (hi[a] - lo[a]) / g->nc[a] < cutoff && g->nc[a] > 1) {
      set_error("neighbor: cell narrower than the cutoff");
      return ICTC_ERR_BAD_ARG;
    }
    if (periodic[a] && box[a] < cutoff) {
      set_error("neighbor: periodic box shorter than the cutoff needs more than one image per axis");
      return ICTC_ERR_BAD_ARG;
    }
  }
  g->cutsq = cutoff * cutoff;
  g->rc = float(cutoff);
  g->span = 0.f;
  for (int a = 0; a < 3; ++a) g->span += float(box[a] + 3.0 / g->inv_w[a]);
  if (N > 2147483647LL) { set_error("neighbor: too many atoms"); return ICTC_ERR_TOO_LARGE; }
  return ICTC_OK;
}

struct LoadInt {
  const int* v;
  __device__ int operator()(int64_t i) const { return v[i]; }
};
struct StoreCellStart {
  int* start;
  __device__ void operator()(int64_t i, int before, int v) const {
    start[i] = before;
    start[i + 1] = before + v;        // the next value's own store writes the same number
  }
};
struct LoadPacked {
  const uint2* v;
  __device__ unsigned long long operator()(int64_t i) const {
    const uint2 p = v[i];
    return (unsigned long long)p.x | ((unsigned long long)p.y << 32);
  }
};
// Row offsets clamped to the capacity (rows beyond it become empty, the row that straddles it is truncated), pair rows
// per row, number of pairs, and the sticky overflow flag.
struct StoreRows {
  int64_t* rowptr;
  int* u_row;
  int64_t n, capacity;
  int64_t* num_unique;
  int32_t* overflow;
  __device__ void operator()(int64_t i, unsigned long long before, unsigned long long v) const {
    const unsigned long long next = before + v;
    const int64_t end = int64_t(next & 0xffffffffull);
    if (i == 0) { rowptr[0] = 0; u_row[0] = 0; }
    rowptr[i + 1] = end < capacity ? end : capacity;
    u_row[i + 1] = int(next >> 32);
    if (i == n - 1) {
      *num_unique = int64_t(next >> 32);
      if (end > capacity) *overflow = 1;
    }
  }
};

static void nb_bin(const NbGrid& g, const float* pos, int64_t N, int64_t cells, const NbScratch& s, cudaStream_t st) {
  cudaMemsetAsync(s.cell_count, 0, 4 * cells, st);
  if (N > 0) launch_after(nb_bin_count_kernel, (unsigned)((N + 255) / 256), 256, 0, st, g, pos, N, s.cell_count, s.where);
  prefix_sum<int>(cells, LoadInt{s.cell_count}, StoreCellStart{s.cell_start}, reinterpret_cast<int*>(s.sums), false, st);
  if (N > 0) launch_after(nb_bin_fill_kernel, (unsigned)((N + 255) / 256), 256, 0, st, pos, N, s.cell_start, s.where, s.atoms);
}

int ictc_neighbor_count(const float* pos, int64_t num_atoms, int64_t num_centres, const double* host_lo,
                        const double* host_hi, const double* host_box, const int* host_periodic, double cutoff,
                        int64_t* rowptr, void* scratch, void* stream) {
  NbGrid g;
  int64_t cells;
  if (int rc = nb_setup(num_atoms, host_lo, host_hi, host_box, host_periodic, cutoff, &g, &cells)) return rc;
  if (num_centres < 0 || num_centres > num_atoms || !rowptr || !scratch || (num_atoms > 0 && !pos)) {
    set_error("neighbor_count: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  NbScratch s;
  nb_carve(scratch, num_atoms, cells, &s);
  nb_bin(g, pos, num_atoms, cells, s, st);
  if (num_centres > 0)
    launch_after(nb_count_kernel, (unsigned)((num_centres + kNbWarps - 1) / kNbWarps), kNbWarps * 32, 0, st,
        g, pos, s.cell_start, s.atoms, num_centres, rowptr, nullptr);
  else
    cudaMemsetAsync(rowptr, 0, 8, st);
  return finish_launch("neighbor_count");
}

int ictc_neighbor_fill(const float* pos, int64_t num_atoms, int64_t num_centres, const double* host_lo,
                       const double* host_hi, const double* host_box, const int* host_periodic, double cutoff,
                       const int64_t* rowptr, int64_t capacity, int64_t* src, int64_t* dst, float* shifts,
                       int64_t* edge_keys, void* scratch, void* stream) {
  NbGrid g;
  int64_t cells;
  if (int rc = nb_setup(num_atoms, host_lo, host_hi, host_box, host_periodic, cutoff, &g, &cells)) return rc;
  if (num_centres == 0 || capacity == 0) return ICTC_OK;
  if (!rowptr || !src || !dst || !shifts || !edge_keys || !scratch) {
    set_error("neighbor_fill: NULL buffer");
    return ICTC_ERR_BAD_ARG;
  }
  NbScratch s;
  nb_carve(scratch, num_atoms, cells, &s);
  launch_after(nb_fill_kernel, (unsigned)((num_centres + kNbWarps - 1) / kNbWarps), kNbWarps * 32, 0, (cudaStream_t)stream,
      g, pos, s.cell_start, s.atoms, num_centres, rowptr, capacity, src, dst, shifts, edge_keys);
  return finish_launch("neighbor_fill");
}

int ictc_neighbor_build(const float* pos, int64_t num_atoms, int64_t num_centres, const double* host_lo,
                        const double* host_hi, const double* host_box, const int* host_periodic, double cutoff,
                        int64_t capacity, int64_t unique_capacity, int64_t pad_src, int64_t* rowptr, int64_t* src,
                        int64_t* dst, float* shifts, int64_t* edge_keys, int64_t* rev, int64_t* gate_row,
                        int64_t* rep_edge, int64_t* other_edge, int64_t* num_unique, int32_t* overflow, void* scratch,
                        void* stream) {
  NbGrid g;
  int64_t cells;
  if (int rc = nb_setup(num_atoms, host_lo, host_hi, host_box, host_periodic, cutoff, &g, &cells)) return rc;
  if (num_centres < 1 || num_centres > num_atoms || capacity < 1 || unique_capacity < 0 || capacity > 2147483647LL ||
      unique_capacity > 2147483647LL) {
    set_error("neighbor_build: sizes");
    return ICTC_ERR_BAD_ARG;
  }
  if (!pos || !rowptr || !src || !dst || !shifts || !edge_keys || !rev || !gate_row || !rep_edge || !other_edge ||
      !num_unique || !overflow || !scratch) {
    set_error("neighbor_build: NULL buffer");
    return ICTC_ERR_BAD_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  NbScratch s;
  nb_carve(scratch, num_atoms, cells, &s);
  nb_bin(g, pos, num_atoms, cells, s, st);
  const unsigned blocks = (unsigned)((num_centres + kNbWarps - 1) / kNbWarps);
  launch_after(nb_count_kernel, blocks, kNbWarps * 32, 0, st, g, pos, s.cell_start, s.atoms, num_centres, nullptr, s.packed);
  // capacity - 1: the last slot always stays an inert edge
  prefix_sum<unsigned long long>(num_centres, LoadPacked{s.packed},
                                 StoreRows{rowptr, s.u_row, num_centres, capacity - 1, num_unique, overflow}, s.sums,
                                 false, st);
  launch_after(nb_fill_kernel, blocks, kNbWarps * 32, 0, st, g, pos, s.cell_start, s.atoms, num_centres, rowptr, capacity, src,
                                                  dst, shifts, edge_keys);
  const int64_t span = capacity > unique_capacity ? capacity : unique_capacity;
  launch_after(nb_pair_kernel, (unsigned)((span + 255) / 256), 256, 0, st, rowptr, s.u_row, edge_keys, num_centres, capacity,
                                                                unique_capacity, pad_src, src, dst, shifts, rev,
                                                                gate_row, rep_edge, other_edge);
  return finish_launch("neighbor_build");
}

int ictc_neighbor_clamp(int64_t* rowptr, int64_t num_centres, int64_t capacity, int32_t* overflow, void* stream) {
  if (num_centres < 0 || capacity < 0 || !rowptr || !overflow) {
    set_error("neighbor_clamp: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  nb_clamp_kernel<<<(unsigned)((num_centres + 1 + 255) / 256), 256, 0, (cudaStream_t)stream>>>(rowptr, num_centres + 1,
                                                                                             capacity, overflow);
  return finish_launch("neighbor_clamp");
}

int ictc_neighbor_pad(const int64_t* count, int64_t capacity, int64_t pad_src, int64_t pad_dst, int64_t* src,
                      int64_t* dst, float* shifts, int32_t* overflow, void* stream) {
  if (capacity < 0 || !count || (capacity > 0 && (!src || !dst || !shifts))) {
    set_error("neighbor_pad: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  const int64_t blocks = capacity > 0 ? (capacity + 255) / 256 : 1;
  if (blocks > 2147483647LL) { set_error("neighbor_pad: too many edges"); return ICTC_ERR_TOO_LARGE; }
  nb_pad_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(count, capacity, pad_src, pad_dst, src, dst,
                                                                    shifts, overflow);
  return finish_launch("neighbor_pad");
}

extern "C" int ictc_inclusive_scan_i64(int64_t* data, int64_t n, void* scratch, void* stream);

int ictc_neighbor_pairs(const int64_t* rowptr, const int64_t* dst, const int64_t* edge_keys, int64_t num_centres,
                        int64_t capacity, int64_t unique_capacity, const int64_t* count, int64_t* rev, int64_t* scan,
                        int64_t* gate_row, int64_t* rep_edge, int64_t* other_edge, int64_t* num_unique,
                        void* scan_scratch, void* stream) {
  if (num_centres < 0 || capacity < 0 || unique_capacity < 0 || !count || !num_unique) {
    set_error("neighbor_pairs: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  const int64_t span = capacity > unique_capacity ? capacity : unique_capacity;
  if (span == 0) return ICTC_OK;
  if (!rowptr || !dst || !edge_keys || !rev || !scan || !gate_row || !rep_edge || !other_edge || !scan_scratch) {
    set_error("neighbor_pairs: NULL buffer");
    return ICTC_ERR_BAD_ARG;
  }
  if ((span + 255) / 256 > 2147483647LL) { set_error("neighbor_pairs: too many edges"); return ICTC_ERR_TOO_LARGE; }
  cudaStream_t st = (cudaStream_t)stream;
  if (capacity > 0) {
    nb_pair_find_kernel<<<(unsigned)((capacity + 255) / 256), 256, 0, st>>>(rowptr, dst, edge_keys, num_centres,
                                                                           capacity, count, rev, scan);
    if (int rc = ictc_inclusive_scan_i64(scan, capacity, scan_scratch, stream)) return rc;
  }
  nb_pair_assign_kernel<<<(unsigned)((span + 255) / 256), 256, 0, st>>>(scan, rev, capacity, unique_capacity, count,
                                                                      gate_row, rep_edge, other_edge, num_unique);
  return finish_launch("neighbor_pairs");
}

int ictc_md_kick(int64_t num_atoms, float dt, const float* force, const float* inv_mass, float* vel, float* pos,
                 const float* box, int drift, void* stream) {
  if (num_atoms < 0 || (num_atoms > 0 && (!force || !inv_mass || !vel || (drift && (!pos || !box))))) {
    set_error("md_kick: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  if (num_atoms == 0) return ICTC_OK;
  launch_after(md_kick_drift_kernel, (unsigned)((num_atoms + 255) / 256), 256, 0, (cudaStream_t)stream,
      num_atoms, dt, force, inv_mass, vel, pos, box, drift);
  return finish_launch("md_kick");
}

}  // extern "C"
