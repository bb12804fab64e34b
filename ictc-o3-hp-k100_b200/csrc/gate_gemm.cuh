// Launch interface of the tensor-core linears (gate_gemm.cu) inside the library.
#pragma once
#include "tc05.cuh"

namespace ictc {
namespace gg {

constexpr int kMaxSegments = 3;

// One matrix product.  Row addressing (units: floats): row g is sub-row g % mm of node g / mm; its 64-float block number
// b (the only block of the 64-wide side, chunk c * cs of the wide side) starts at
//   base + (g / mm) * ld + (b + g % mm) * 64.
// Plain matrices: mm = 1, ld = row length, cs = 1.  Per-degree feature blocks [node][path slot][m][C]:
// mm = 2l+1, ld = node stride, cs = mm (the slot-major layout is read and written in place).
struct Segment {
  const float* in;
  const float* w;         // packed chunks, 8192 floats each
  float* out;
  int64_t rows;
  int chunks;             // 64-wide blocks of the wide side
  int in_mm, out_mm, in_cs, out_cs;
  int64_t in_ld, out_ld;
};

struct Args {
  Segment seg[kMaxSegments];
  int segments;
  const int64_t* pair_a;  // backward, optional: row g is in[pair_a[g]] + in[pair_b[g]] (one segment)
  const int64_t* pair_b;
  const int64_t* limit;   // optional device scalar: only min(rows, *limit) rows of every segment are processed
  // Row windows (one segment, plain matrices).  With `begin` (device scalar) the launch covers the window
  // [*begin, min(*begin + rows, *limit)) of a longer row list: local row g = 0.. stands for list entry *begin + g.
  const int64_t* begin;
  const int64_t* in_index;   // forward: local row g reads in[in_index[*begin + g]] (null: in[*begin + g])
  const int64_t* out_index;  // backward: local row g is written to out[out_index[*begin + g]] (null: out[*begin + g])
  // forward, optional: bias[bias_index ? bias_index[n] : n][0..63] is added to block 0 of the first segment for its
  // nodes n < bias_nodes (mm must be 1)
  const float* bias;
  const int64_t* bias_index;
  int64_t bias_nodes;
  int act;                // forward: apply the scaled SiLU to the input
  int* status;
};

// out [rows, 64 * chunks] = act(in [rows, 64]) @ W^T, and out [rows, 64] = in [rows, 64 * chunks] @ W.
// Buffers 32-byte aligned, strides multiples of 8 floats (checked by the callers).
int launch_forward(Args a, cudaStream_t st);
int launch_backward(Args a, cudaStream_t st);

inline Segment segment(const float* in, const float* w, float* out, int64_t rows, int chunks, int in_mm, int64_t in_ld,
                       int out_mm, int64_t out_ld) {
  return Segment{in, w, out, rows, chunks, in_mm, out_mm, in_mm, out_mm, in_ld, out_ld};
}

}  // namespace gg
}  // namespace ictc
