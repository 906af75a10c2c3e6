// The policy's heads on tcgen05 tiles (head_tiles.cu).
#pragma once
#include <cuda_runtime.h>

#include "mlp_kernels.h"

namespace bnb {
namespace mlp {

// Whether the tiles serve a call of mlp::run: heads (rows of 128) or an encoder with its last norm.  They do
// at every size: a single tile takes no longer than the same rows in slices of 16 there.
bool head_tiles_serve(const MlpCall& call, int n_chains, int in_pad, int hidden, int out_dim);
int head_tiles(const MlpCall& call, int n_chains, int out_dim, cudaStream_t st);

}  // namespace mlp
}  // namespace bnb
