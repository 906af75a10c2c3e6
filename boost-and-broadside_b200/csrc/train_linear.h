// The Linear layers of the training path on tensor-core tiles (train_linear.cu), for d_model 128 under the
// bfloat16 contract: up to three layers that share an input in one pass, forward and backward.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace bnb {
namespace train_linear {

constexpr int MAX_BLOCKS = 3;             // 128-row blocks of weights in one call
constexpr size_t BLOCK_IMAGE = 32768;     // bfloat16 image of one block

// Images of n (128, 128) weight blocks (row-major, 512 bytes a row), one after the other at `image`.
[[nodiscard]] int pack(const float* const* blocks, int n, uint8_t* image, cudaStream_t st);

// out[b] = n W_b^T (+ bias[b]) (+ residual, one block only) for the blocks at `image`.  With a gain, n = bf16 of
// x's RMSNorm, written to n_out, the reciprocal roots to inv; without, n = bf16(x).
struct Forward {
  const float* x = nullptr;
  const float* gain = nullptr;
  void* n_out = nullptr;
  float* inv = nullptr;
  const uint8_t* image = nullptr;
  int blocks = 1;
  float* out[MAX_BLOCKS] = {};
  const float* bias[MAX_BLOCKS] = {};
  int ld_out = 128;
  const float* residual = nullptr;
  size_t rows = 0;
  const int* count = nullptr;   // on the device: how many of the rows there are, or null: all
};
[[nodiscard]] int forward(const Forward& f, int* status, cudaStream_t st);

// Given dy[b]: dn = sum_b dy_b W_b; d_weight[b] (128, 128) += dy_b^T n; without a gain d_bias[b] += column sums of dy_b.
// Without a gain (one or two blocks, n float32): dx = dn (+ dx before, if accumulate).
// With one (two or three blocks, n bfloat16): dn goes on through the norm of x: dx = dres + d norm, d_gain accumulated;
// dx may be dres.
struct Backward {
  const float* dy[MAX_BLOCKS] = {};
  const void* n = nullptr;
  const uint8_t* image = nullptr;
  int blocks = 1;
  float* d_weight[MAX_BLOCKS] = {};
  float* d_bias[MAX_BLOCKS] = {};
  float* dx = nullptr;
  bool accumulate = false;
  const float* x = nullptr;
  const float* gain = nullptr;
  const float* inv = nullptr;
  const float* dres = nullptr;
  float* d_gain = nullptr;
  size_t rows = 0;
  const int* count = nullptr;   // as in Forward
};
[[nodiscard]] int backward(const Backward& b, int* status, cudaStream_t st);

}  // namespace train_linear
}  // namespace bnb
