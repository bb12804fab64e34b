// Fused edge-geometry, radial-basis, activation and force-assembly kernels of the force engine.
//
// These are the element-wise ends of the model that the reference leaves to a chain of PyTorch
// operators: edge vectors / lengths / unit vectors (mace_ictc/models/mace/backbone.py:941-952), the
// Bessel basis with polynomial envelope (mace_ictc/models/radial_basis.py:11-92), the direction
// harmonics (ictc_o3/basis/ictd_irreps.py:1153-1208), SiLU * 1.679 (mace_ictc/models/mace/layers.py:307-314)
// and the position gradient scatter of autograd.  One kernel each way instead of ~30 launches.
#include "geometry.cuh"

namespace ictc {

constexpr int kRadialMax = 16;

struct GeomArgs {
  const float* pos;          // [N,3]
  const int64_t* src;        // [E]
  const int64_t* dst;        // [E]
  const float* shifts;       // [E,3] lattice units or null
  float box[3];
  float r_max;
  int num_basis, p;
  int64_t E;
  float* sh;                 // [E,9]
  float* rb;                 // [E,num_basis]
  float* unit;               // [E,3]
  float* length;             // [E]
  const float* dsh;          // backward inputs
  const float* drb;
  float* dvec;               // [E,3]
};

__global__ void geom_forward_kernel(GeomArgs a) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= a.E) return;
  const int64_t i = a.dst[e], j = a.src[e];
  float v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v[k] = a.pos[3 * i + k] - a.pos[3 * j + k];
    if (a.shifts) v[k] += a.shifts[3 * e + k] * a.box[k];
  }
  const float r = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  const float rc = fmaxf(r, 1e-8f);
  const float x = v[0] / rc, y = v[1] / rc, z = v[2] / rc;
  a.unit[3 * e + 0] = x;
  a.unit[3 * e + 1] = y;
  a.unit[3 * e + 2] = z;
  a.length[e] = r;
  float val[9];
  harmonics_value(x, y, z, val);
#pragma unroll
  for (int h = 0; h < 9; ++h) a.sh[9 * e + h] = val[h];
  float env, denv;
  envelope(r, a.r_max, a.p, env, denv);
  const float pref = sqrtf(2.f / a.r_max) / fmaxf(r, 1e-12f);
  const float w = 3.14159265358979323846f / a.r_max;
  for (int k = 0; k < a.num_basis; ++k) a.rb[e * a.num_basis + k] = pref * sinf(r * (w * float(k + 1))) * env;
}

__global__ void geom_backward_kernel(GeomArgs a) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= a.E) return;
  const float x = a.unit[3 * e], y = a.unit[3 * e + 1], z = a.unit[3 * e + 2];
  const float r = a.length[e];
  float g[9];
#pragma unroll
  for (int h = 0; h < 9; ++h) g[h] = a.dsh[9 * e + h];
  const float3 v = edge_vector_gradient(x, y, z, r, g, a.drb + e * a.num_basis, a.num_basis, a.p, a.r_max);
  a.dvec[3 * e + 0] = v.x;
  a.dvec[3 * e + 1] = v.y;
  a.dvec[3 * e + 2] = v.z;
}

// grad[i] = sum_{e: dst(e)=i} dvec[e] - sum_{e: src(e)=i} dvec[e]; fixed CSR order, no atomics.
__global__ void position_gradient_kernel(int64_t n, int64_t n_dst_rows, const int64_t* __restrict__ dst_rowptr,
                                         const int64_t* __restrict__ src_rowptr, const int64_t* __restrict__ src_order,
                                         const float* __restrict__ dvec, float* grad) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  if (i < n_dst_rows) {
    for (int64_t e = dst_rowptr[i]; e < dst_rowptr[i + 1]; ++e) {
      gx += dvec[3 * e];
      gy += dvec[3 * e + 1];
      gz += dvec[3 * e + 2];
    }
  }
  for (int64_t k = src_rowptr[i]; k < src_rowptr[i + 1]; ++k) {
    const int64_t e = src_order ? src_order[k] : k;
    gx -= dvec[3 * e];
    gy -= dvec[3 * e + 1];
    gz -= dvec[3 * e + 2];
  }
  grad[3 * i] = gx;
  grad[3 * i + 1] = gy;
  grad[3 * i + 2] = gz;
}

// Scaled SiLU and its derivatives, element by element, memory bound: 16-byte accesses where every buffer allows them.
//   MODE 0: y = scale * silu(x)      MODE 1: y = g * scale * silu'(x)
//   MODE 2, the adjoint of MODE 1 with cotangent h: y = h * g * scale * silu''(x) (or null), z = h * scale * silu'(x) (or null)
// In training each derivative was a chain of framework operators over the [E, 64] hidden rows, ten passes over memory for
// MODE 2: 1.05 M x 64 elements 1.6 ms as such a chain, 0.16 ms now (6.6 TB/s of 5 passes); training step 67.2 -> 57.0 ms.
template <int MODE> __device__ __forceinline__ void silu_element(float scale, float x, float g, float h, float& y, float& z) {
  const float s = 1.f / (1.f + expf(-x));
  if (MODE == 0) { y = x / (1.f + expf(-x)) * scale; return; }
  const float d = scale * s * (1.f + x * (1.f - s));
  if (MODE == 1) { y = g * d; return; }
  y = h * g * (scale * s * (1.f - s) * (2.f + x * (1.f - 2.f * s)));
  z = h * d;
}
template <int MODE>
__global__ void __launch_bounds__(256) silu_kernel(int64_t n, bool wide, float scale, const float* __restrict__ x,
                                                   const float* __restrict__ g, const float* __restrict__ h, float* y,
                                                   float* z) {
  const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  if (wide && i + 4 <= n) {
    auto in = [&](const float* p) { return __ldg(reinterpret_cast<const float4*>(p + i)); };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 xv = in(x), gv = MODE >= 1 ? in(g) : zero, hv = MODE == 2 ? in(h) : zero;
    float4 yv, zv;
    silu_element<MODE>(scale, xv.x, gv.x, hv.x, yv.x, zv.x);
    silu_element<MODE>(scale, xv.y, gv.y, hv.y, yv.y, zv.y);
    silu_element<MODE>(scale, xv.z, gv.z, hv.z, yv.z, zv.z);
    silu_element<MODE>(scale, xv.w, gv.w, hv.w, yv.w, zv.w);
    if (MODE != 2 || y) *reinterpret_cast<float4*>(y + i) = yv;
    if (MODE == 2 && z) *reinterpret_cast<float4*>(z + i) = zv;
    return;
  }
  for (int64_t k = i; k < i + 4 && k < n; ++k) {
    float yv, zv;
    silu_element<MODE>(scale, x[k], MODE >= 1 ? g[k] : 0.f, MODE == 2 ? h[k] : 0.f, yv, zv);
    if (MODE != 2 || y) y[k] = yv;
    if (MODE == 2 && z) z[k] = zv;
  }
}

// Whole-row layout conversion between mul_ir (block [C][m]) and ir_mul (block [m][C]) for a row made of
// degree blocks, each holding `count` path slots.
constexpr int kLayoutBlocks = 8;
struct LayoutArgs {
  int64_t rows;
  int width, C, nblocks;
  int count[kLayoutBlocks], m[kLayoutBlocks], off[kLayoutBlocks + 1];
};

// Rows of 2l+1 = 1, 3, 5 or 7 components and channels in fours (the network's own layouts), 16-byte aligned buffers.
// A thread turns one quad, 4 channels x M components, in registers: its 4M floats are M consecutive 16-byte pieces of the
// mul_ir row and one piece in each of the M component rows on the ir_mul side.  The ir_mul side is accessed in global
// memory (neighbouring quads are neighbouring pieces); the mul_ir side, where a thread's pieces lie M apart, through
// a tile of whole rows in shared memory that moves in consecutive pieces (M is odd, so 16-byte accesses M apart hit
// different banks).  Bound by memory: one read and one write of the rows.  The tile is small enough for eight blocks per
// SM, which hide each other's barriers.  20,011 rows of 576 and of 2,240 floats, both ways: 568 -> 218 us, 4.1 TB/s.
constexpr int kTileThreads = 256, kTileBytes = 24 * 1024;
struct LayoutTile {
  int rows;                    // rows of a tile
  int quads;                   // quads of a row
  int first[kLayoutBlocks + 1];      // first quad of a block
};

template <int M> __device__ __forceinline__ void turn_quad(float4* mul_ir, float4* ir_mul, int pitch, bool to_ir_mul) {
  float4 q[M];
  if (to_ir_mul) {
    float v[4 * M];
#pragma unroll
    for (int k = 0; k < M; ++k) q[k] = mul_ir[k];
#pragma unroll
    for (int k = 0; k < M; ++k) { v[4 * k] = q[k].x; v[4 * k + 1] = q[k].y; v[4 * k + 2] = q[k].z; v[4 * k + 3] = q[k].w; }
#pragma unroll
    for (int k = 0; k < M; ++k) ir_mul[k * pitch] = make_float4(v[k], v[M + k], v[2 * M + k], v[3 * M + k]);
  } else {
    float v[4 * M];
#pragma unroll
    for (int k = 0; k < M; ++k) q[k] = __ldg(ir_mul + k * pitch);
#pragma unroll
    for (int k = 0; k < M; ++k) { v[k] = q[k].x; v[M + k] = q[k].y; v[2 * M + k] = q[k].z; v[3 * M + k] = q[k].w; }
#pragma unroll
    for (int k = 0; k < M; ++k) mul_ir[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  }
}

__global__ void __launch_bounds__(kTileThreads) layout_tile_kernel(LayoutArgs a, LayoutTile t, const float* __restrict__ in,
                                                                   float* __restrict__ out, int to_ir_mul) {
  extern __shared__ __align__(16) float4 layout_tile[];
  const int row_pieces = a.width / 4, pitch = a.C / 4;
  for (int64_t r0 = int64_t(blockIdx.x) * t.rows; r0 < a.rows; r0 += int64_t(gridDim.x) * t.rows) {
    const int rows = int(min(int64_t(t.rows), a.rows - r0)), pieces = rows * row_pieces;
    const float4* from = reinterpret_cast<const float4*>(in) + r0 * row_pieces;
    float4* to = reinterpret_cast<float4*>(out) + r0 * row_pieces;
    if (to_ir_mul) {
      for (int i = threadIdx.x; i < pieces; i += kTileThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unsigned(__cvta_generic_to_shared(layout_tile + i))),
                     "l"(from + i)
                     : "memory");
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    for (int item = threadIdx.x; item < rows * t.quads; item += kTileThreads) {
      const int row = item / t.quads, q = item - row * t.quads;
      int b = 0;
      while (b + 1 < a.nblocks && q >= t.first[b + 1]) ++b;
      const int m = a.m[b], rel = q - t.first[b], slot = rel / pitch, c = rel - slot * pitch;
      const int block = row * row_pieces + a.off[b] / 4 + slot * pitch * m;
      float4* tile = layout_tile + block + c * m;
      float4* global = (to_ir_mul ? to : const_cast<float4*>(from)) + block + c;
      switch (m) {
        case 1: turn_quad<1>(tile, global, pitch, to_ir_mul); break;
        case 3: turn_quad<3>(tile, global, pitch, to_ir_mul); break;
        case 5: turn_quad<5>(tile, global, pitch, to_ir_mul); break;
        default: turn_quad<7>(tile, global, pitch, to_ir_mul); break;
      }
    }
    __syncthreads();
    if (!to_ir_mul) {
      for (int i = threadIdx.x; i < pieces; i += kTileThreads) to[i] = layout_tile[i];
      __syncthreads();
    }
  }
}

// Other component counts, channel counts and alignments.
// One block per group of rows: a row is read as it lies in memory (coalesced) into shared memory, and written in the
// other order from there (the transposed reads hit shared memory with odd strides 2l+1, or stride C across the
// 2l+1 <= 5 components: no bank conflicts worth mentioning), so both global accesses are contiguous.
__global__ void __launch_bounds__(256) layout_copy_kernel(LayoutArgs a, const float* __restrict__ in,
                                                          float* __restrict__ out, int to_ir_mul) {
  extern __shared__ float layout_row[];
  for (int64_t r = blockIdx.x; r < a.rows; r += gridDim.x) {
    const float* src_row = in + r * a.width;
    for (int col = threadIdx.x; col < a.width; col += blockDim.x) layout_row[col] = src_row[col];
    __syncthreads();
    float* dst_row = out + r * a.width;
    for (int col = threadIdx.x; col < a.width; col += blockDim.x) {
      int b = 0;
      while (b + 1 < a.nblocks && col >= a.off[b + 1]) ++b;
      const int m = a.m[b], C = a.C;
      const int rel = col - a.off[b];
      const int slot = rel / (C * m), q = rel - slot * (C * m);
      // output index q -> (outer, inner) of the OUTPUT block; the input block is its transpose
      const int outer = to_ir_mul ? q / C : q / m, inner = to_ir_mul ? q - outer * C : q - outer * m;
      const int src = to_ir_mul ? inner * m + outer : inner * C + outer;
      dst_row[col] = layout_row[a.off[b] + slot * C * m + src];
    }
    __syncthreads();
  }
}

template <int MODE>
static int silu_launch(const char* what, int64_t n, float scale, const float* x, const float* g, const float* h, float* y,
                       float* z, void* stream) {
  if (n < 0 || (n + 1023) / 1024 > 2147483647LL) { set_error("%s: size", what); return ICTC_ERR_TOO_LARGE; }
  if (n == 0) return ICTC_OK;
  if (!x || (MODE < 2 && !y) || (MODE >= 1 && !g) || (MODE == 2 && !h)) { set_error("%s: NULL buffer", what); return ICTC_ERR_BAD_ARG; }
  uintptr_t bits = 0;
  for (const void* p : {(const void*)x, (const void*)g, (const void*)h, (const void*)y, (const void*)z})
    bits |= reinterpret_cast<uintptr_t>(p);
  silu_kernel<MODE><<<(unsigned)((n + 1023) / 1024), 256, 0, (cudaStream_t)stream>>>(n, (bits & 15) == 0, scale, x, g, h, y, z);
  return finish_launch(what);
}

}  // namespace ictc

using namespace ictc;

extern "C" {

static int geom_fill(GeomArgs& a, const float* pos, const int64_t* src, const int64_t* dst, const float* shifts,
                     const float* host_box, float r_max, int num_basis, int p, int64_t E) {
  if (E < 0 || num_basis < 1 || num_basis > kRadialMax || p < 2 || !(r_max > 0)) {
    set_error("edge geometry: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  if ((E + 255) / 256 > 2147483647LL) { set_error("edge geometry: too many edges"); return ICTC_ERR_TOO_LARGE; }
  a.pos = pos; a.src = src; a.dst = dst; a.shifts = shifts;
  for (int k = 0; k < 3; ++k) a.box[k] = host_box ? host_box[k] : 0.f;
  a.r_max = r_max; a.num_basis = num_basis; a.p = p; a.E = E;
  return ICTC_OK;
}

int ictc_edge_geometry_forward(const float* pos, const int64_t* src, const int64_t* dst, const float* shifts,
                               const float* host_box, float r_max, int num_basis, int p, int64_t num_edges,
                               float* sh, float* rb, float* unit, float* length, void* stream) {
  GeomArgs a{};
  if (int rc = geom_fill(a, pos, src, dst, shifts, host_box, r_max, num_basis, p, num_edges)) return rc;
  if (num_edges == 0) return ICTC_OK;
  if (!pos || !src || !dst || !sh || !rb || !unit || !length) { set_error("edge geometry: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  a.sh = sh; a.rb = rb; a.unit = unit; a.length = length;
  geom_forward_kernel<<<(unsigned)((num_edges + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a);
  return finish_launch("edge_geometry_forward");
}

int ictc_edge_geometry_backward(const float* unit, const float* length, float r_max, int num_basis, int p,
                                int64_t num_edges, const float* dsh, const float* drb, float* dvec, void* stream) {
  GeomArgs a{};
  if (int rc = geom_fill(a, nullptr, nullptr, nullptr, nullptr, nullptr, r_max, num_basis, p, num_edges)) return rc;
  if (num_edges == 0) return ICTC_OK;
  if (!unit || !length || !dsh || !drb || !dvec) { set_error("edge geometry backward: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  a.unit = const_cast<float*>(unit); a.length = const_cast<float*>(length); a.dsh = dsh; a.drb = drb; a.dvec = dvec;
  geom_backward_kernel<<<(unsigned)((num_edges + 255) / 256), 256, 0, (cudaStream_t)stream>>>(a);
  return finish_launch("edge_geometry_backward");
}

int ictc_position_gradient(int64_t num_rows, int64_t num_dst_rows, const int64_t* dst_rowptr,
                           const int64_t* src_rowptr, const int64_t* src_order, const float* dvec, float* grad,
                           void* stream) {
  if (num_rows < 0 || num_dst_rows < 0 || num_dst_rows > num_rows) { set_error("position gradient: sizes"); return ICTC_ERR_BAD_ARG; }
  if (num_rows == 0) return ICTC_OK;
  if (!dst_rowptr || !src_rowptr || !grad) { set_error("position gradient: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  position_gradient_kernel<<<(unsigned)((num_rows + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
      num_rows, num_dst_rows, dst_rowptr, src_rowptr, src_order, dvec, grad);
  return finish_launch("position_gradient");
}

int ictc_silu_forward(int64_t n, float scale, const float* x, float* y, void* stream) {
  return silu_launch<0>("silu_forward", n, scale, x, nullptr, nullptr, y, nullptr, stream);
}

int ictc_silu_backward(int64_t n, float scale, const float* x, const float* dy, float* dx, void* stream) {
  return silu_launch<1>("silu_backward", n, scale, x, dy, nullptr, dx, nullptr, stream);
}

int ictc_silu_second(int64_t n, float scale, const float* x, const float* dy, const float* h, float* gx, float* gdy,
                     void* stream) {
  return silu_launch<2>("silu_second", n, scale, x, dy, h, gx, gdy, stream);
}

int ictc_layout_copy(int64_t rows, int channels, int num_blocks, const int* host_counts, const int* host_ms,
                     const float* in, float* out, int to_ir_mul, void* stream) {
  if (rows < 0 || channels < 1 || num_blocks < 1 || num_blocks > kLayoutBlocks || !host_counts || !host_ms) {
    set_error("layout copy: invalid arguments");
    return ICTC_ERR_BAD_ARG;
  }
  LayoutArgs a;
  a.rows = rows; a.C = channels; a.nblocks = num_blocks;
  int off = 0;
  for (int b = 0; b < num_blocks; ++b) {
    if (host_counts[b] < 0 || host_ms[b] < 1) { set_error("layout copy: invalid block"); return ICTC_ERR_BAD_ARG; }
    a.count[b] = host_counts[b]; a.m[b] = host_ms[b]; a.off[b] = off;
    off += host_counts[b] * host_ms[b] * channels;
  }
  a.off[num_blocks] = off;
  a.width = off;
  const int64_t total = rows * int64_t(off);
  if (total == 0) return ICTC_OK;
  if (!in || !out) { set_error("layout copy: NULL buffer"); return ICTC_ERR_BAD_ARG; }
  bool quads = channels % 4 == 0 && off <= kTileBytes / 4 &&
               ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  LayoutTile t{};
  for (int b = 0; b < num_blocks; ++b) {
    quads = quads && (a.m[b] == 1 || a.m[b] == 3 || a.m[b] == 5 || a.m[b] == 7);
    t.first[b] = t.quads;
    t.quads += a.count[b] * (channels / 4);
  }
  t.first[num_blocks] = t.quads;
  if (quads) {
    const int64_t spread = (rows + 148 * 8 - 1) / (148 * 8);        // few rows: one block each before tiles grow
    t.rows = int(spread < kTileBytes / (4 * off) ? spread : kTileBytes / (4 * off));
    const int64_t tiles = (rows + t.rows - 1) / t.rows;
    const unsigned blocks = unsigned(tiles < 148 * 8 ? tiles : 148 * 8);
    layout_tile_kernel<<<blocks, kTileThreads, size_t(t.rows) * off * 4, (cudaStream_t)stream>>>(a, t, in, out, to_ir_mul);
    return finish_launch("layout_tile");
  }
  const size_t smem = size_t(off) * sizeof(float);
  if (smem > 200 * 1024) { set_error("layout copy: rows of %d floats do not fit shared memory", off); return ICTC_ERR_TOO_LARGE; }
  if (smem > 48 * 1024) {
    const cudaError_t attr = cudaFuncSetAttribute(layout_copy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (attr != cudaSuccess) { set_error("layout copy smem: %s", cudaGetErrorString(attr)); return ICTC_ERR_LAUNCH; }
  }
  const int64_t blocks = rows < 148 * 8 * 4 ? rows : 148 * 8 * 4;       // a few waves of row-looping blocks
  layout_copy_kernel<<<(unsigned)blocks, 256, smem, (cudaStream_t)stream>>>(a, in, out, to_ir_mul);
  return finish_launch("layout_copy");
}

}  // extern "C"
