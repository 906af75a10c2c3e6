// Host interface of the encoder / head MLP kernel on bf16 tensor-core tiles (mlp_kernels.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bnb_trunk.h"

namespace bnb {
namespace mlp {

// True when the tiled kernel serves these (padded) widths: the hidden layer is walked in chunks of
// 64 columns and both weights have to fit in shared memory beside a slice of rows.
bool supported(int in_pad, int hidden, int out_dim);

constexpr int MAX_CHAINS = 4;
// One chain Linear(w1, b1) -> RMSNorm(g1) -> GELU -> Linear(w2, b2) [-> RMSNorm(g2)]: parameters as
// nn.Linear stores them (float32), of w2 / b2 the first out_store rows; output row r goes to y + r * y_ld.
struct MlpChain {
  const float *w1, *b1, *g1, *w2, *b2, *g2;
  __nv_bfloat16* y;
  int out_store, y_ld;
};
// Up to MAX_CHAINS chains of the same widths over the same rows, in one launch.
struct MlpCall {
  const void* x;            // (rows, in_dim) float32, or bfloat16 with x_bf16
  int x_bf16, n_rows, in_dim;
  int w1_ld;                // elements per row of w1: in_dim, or in_pad when its rows are padded with zeros
  // group_rows > 0: row r of the call is input row (r / group_rows) * group_stride + r % group_rows
  // (the ships of every environment out of all of its tokens)
  int group_rows, group_stride;
  const uint8_t* active;    // only rows with a non-zero byte are computed and written; null: all
  MlpChain chain[MAX_CHAINS];
};
// more: chains of the same widths over other rows, in the same launch where the row tiles take both.
int run(const MlpCall& call, int n_chains, int in_pad, int hidden, int out_dim, cudaStream_t st, const MlpCall* more = nullptr, int n_more = 0);

// bfloat16 contract (see bnb_encoder_mlp_fwd / bnb_head_mlp_fwd).  g2 null: no final norm.
// x holds float32 rows, or (x_bf16) bfloat16 rows on a 16-byte boundary with in_dim == in_pad.
int encoder_mlp_bf16(const float* w1, const float* b1, const float* g1, const float* w2, const float* b2, const float* g2,
                     int in_dim, int in_pad, int hidden, int out_dim, int out_store, const void* x, bool x_bf16, void* y,
                     int n_rows, cudaStream_t st);

}  // namespace mlp
}  // namespace bnb
