// One step of the trunk under the float32 contract on tensor-core tiles (split_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "bnb_trunk.h"

namespace bnb {
namespace split {

// The widths the kernels are built for.
inline bool supported(int D, int H) { return D == 128 && H == 4; }

// Images of one sublayer's weights.
size_t spatial_image_bytes();
size_t temporal_image_bytes();

struct Scratch {
  int* status;
  float* qkv;     // (rows, 384)
  float* o;       // (rows, 128)
  float* kvb;     // (kvb_envs * bullets, 256), or null
  int kvb_envs;   // environments per slice of the bullet projection
};

// The trunk over one step: every sublayer of the blocks in order, the weight images (the structs' `packed`
// fields) written first.  y may not alias x.
int step(const BnbSpatialWeights* spatial, const BnbTemporalWeights* temporal, int n_blocks, int n_spatial, int n_temporal,
         const float* x, const uint8_t* alive, const BnbBullets* bullets, float* y, const float* hidden_in, float* hidden_out,
         const uint8_t* reset_env, const BnbBatch& batch, const Scratch& scratch, cudaStream_t st);

}  // namespace split
}  // namespace bnb
