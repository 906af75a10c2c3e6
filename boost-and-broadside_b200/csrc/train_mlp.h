// The GatedMLP of the training path on tensor-core tiles (train_mlp.cu): forward and gradient under the
// bfloat16 contract for d_model 128.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace bnb {
namespace train_mlp {

constexpr int MAX_JOBS = 16;
struct Weights { const float *gate, *up, *down; };   // (512, 128), (512, 128), (128, 512)

size_t image_bytes();                        // bfloat16 images of one MLP's weights
size_t rows_image_bytes(size_t rows);        // bfloat16 tile images of a (rows, 128) tensor
// Images of n MLPs, one after the other at `image` (image_bytes() apart); as many launches as n takes.
[[nodiscard]] int pack(const Weights* w, int n, uint8_t* image, cudaStream_t st);

// y = x1 + down(gelu(gate n) * up n), n = bf16(rmsnorm(x1) * gain).
[[nodiscard]] int forward(const float* x1, const float* gain, const uint8_t* image, float* y, size_t rows, int* status, cudaStream_t st);
// Given dy: dx1 (may alias neither x1 nor dy), and accumulated into: d_gain, d_gate, d_up, d_down.
// n_image / dy_image: rows_image_bytes(rows) each, scratch.
[[nodiscard]] int backward(const float* x1, const float* gain, const uint8_t* image, const float* dy, float* dx1, float* d_gain, float* d_gate,
             float* d_up, float* d_down, uint8_t* n_image, uint8_t* dy_image, size_t rows, int* status, cudaStream_t st);

}  // namespace train_mlp
}  // namespace bnb
