// The policy's heads on tcgen05 tiles (head_tiles.cu).
#pragma once
#include <cuda_runtime.h>

#include "mlp_kernels.h"

namespace bnb {
namespace mlp {

// Whether the tiles serve a call of mlp::run: heads (rows of 128) or an encoder with its last norm.  They do
// at every size: a single tile takes no longer than the same rows in slices of 16 there.  What they are not built
// for stays on k_mlp_bf16, the host included (measured beside the nearest call that the tiles take):
//   rows of odd width     encoder of 65 columns 27 us for 192 rows, 80 for 98 304 (66 columns: 21, 63); of 25 columns 19 and 56
//                         (26 columns: 21, 58)
//   wanted rows only      26 columns, 22 % wanted: 27 us for 192 rows, 49 for 98 304, 127 for 655 360 (all rows: 21, 58, 283;
//                         but 46 against 21 for 2048 rows, where 128 slots per warp leave most of the chip idle)
//   rows between 16-byte  heads of float32 rows 19 us for 128 rows, 43 for 65 536 (12, 29 on a boundary)
//   boundaries
bool head_tiles_serve(const MlpCall& call, int n_chains, int in_pad, int hidden, int out_dim);
int head_tiles(const MlpCall& call, int n_chains, int out_dim, cudaStream_t st, const MlpCall* more = nullptr, int n_more = 0);

}  // namespace mlp
}  // namespace bnb
