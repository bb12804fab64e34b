// Launch interface of the hidden radial layers (mlp_chain.cu) inside the library.
#pragma once
#include "tc05.cuh"

namespace ictc {
namespace chain {

// One stack of hidden layers; a launch takes up to two over the same rows.
struct Stack {
  const float* in;     // forward: rb [*, nb]; backward: da3 [*, 64]
  const float* w0;     // [64, nb] (forward: W0; backward: W0 as well, used as dz1 @ W0)
  const float* wa;     // packed 64 x 64 operand of the first MMA layer (forward: W1, backward: W2 transposed use)
  const float* wb;     // packed operand of the second MMA layer (forward: W2, backward: W1 transposed use)
  float* z1;           // forward outputs / backward inputs [E, 64]
  float* z2;
  float* z3;
  float* drb;          // backward output [*, nb]
};

struct Args {
  Stack stack[2];
  int stacks;
  const int64_t* rows; // optional row index: forward reads rb[rows[r]], backward writes / adds to drb[rows[r]]
  const int64_t* in_a; // backward, optional: row r starts from in[in_a[r]] + in[in_b[r]] (in_b[r] < 0: first term only)
  const int64_t* in_b;
  int accumulate;      // backward: drb[...] += instead of =
  const int64_t* limit; // optional device scalar: only min(E, *limit) rows are processed (recorded graphs)
  int64_t E;
  int nb;
  int* status;
};

int launch_forward(Args a, cudaStream_t st);
int launch_backward(Args a, cudaStream_t st);

}  // namespace chain
}  // namespace ictc
