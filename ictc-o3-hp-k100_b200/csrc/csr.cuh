// CSR builder (csr.cu) for callers inside the library: one or two key vectors of the same length per call.
#pragma once
#include "ictc_common.cuh"

namespace ictc {

struct CsrSet {
  const int64_t* keys;     // [E]
  int64_t* rowptr;         // [N + 1]
  int64_t* order;          // [E]
  int32_t* flag;           // 1: keys sorted, 0: not, -1: a key outside [0, N)
  int64_t* counts;         // [N] scratch
  int64_t* place;          // [E] scratch
};
struct CsrPair { CsrSet set[2]; };

// Words of scratch per key vector: counts, places and the tile totals of the prefix sum behind them.
int64_t csr_scratch_elems(int64_t N, int64_t E);
CsrSet csr_set(const int64_t* keys, int64_t N, int64_t E, int64_t* rowptr, int64_t* order, int32_t* flag, int64_t* scratch);
// sums: sets * prefix_tiles(N) words
int csr_build(const CsrPair& p, int sets, int64_t N, int64_t E, int64_t* sums, cudaStream_t st);

}  // namespace ictc
