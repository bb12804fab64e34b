// The chunk entry points of the graph message for callers inside the library: `sweep_rows` is the number of owner rows of
// the whole sweep that the chunk belongs to, which decides how the rows are shared among warps (a chunk of unknown context
// counts as part of a large sweep).
#pragma once
#include "ictc_common.cuh"

namespace ictc {

int tp_graph_forward_chunk(int64_t sweep_rows, int spec, int channels, int64_t num_rows, const float* x, const float* sh,
                           const float* w, const float* g, const int64_t* gate_row, const int64_t* g_base,
                           int64_t g_capacity, const int64_t* src, const int64_t* dst_rowptr, const int64_t* dst_order,
                           const float* mask, float* out, void* stream);
int tp_graph_adjoint_chunk(int64_t sweep_rows, int spec, int channels, int64_t num_rows, const float* x, const float* sh,
                           const float* w, const float* g, const int64_t* gate_row, int g_by_position,
                           const int64_t* g_base, int64_t g_capacity, const int64_t* dst, const int64_t* src_rowptr,
                           const int64_t* src_order, const float* mask, const float* v, float* dx, float* dsh, float* dg,
                           const int64_t* dg_base, int64_t dg_capacity, void* stream);

}  // namespace ictc
