// Attention of the training path for small environments (train_attention.cu): forward and gradient of
// the self-attention and the bullet branch, float32.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace bnb {
namespace train_attn {

struct Call {
  const float* qkv;         // (G * n, 3 * 128) q | k | v, four heads of 32 side by side in each
  const uint8_t* alive;     // (G * n) or null
  const float* kvb;         // (G * nb, 2 * 128) bullet keys | values, or null
  const uint8_t* bactive;   // (G * nb) or null: every slot is a key
  const int* boff;          // or rows of the slots that are keys only: those of group g are [boff[g], boff[g + 1]), in kvb and dkvb
  int G, n, nb;
  float* o;                 // forward: (G * n, 128)
  const float* d_o;         // gradient: (G * n, 128) in; out q | k | v and keys | values, rows ld apart, the parts off apart
  float* dqkv;
  float* dkvb;
  int ld_dqkv, ld_dkvb;
  size_t off_dqkv, off_dkvb;
};

// d_model 128, 4 heads, up to 32 tokens per environment.
bool supported(int d_model, int n_heads, int n, int nb);
[[nodiscard]] int forward(const Call& c, cudaStream_t st);
[[nodiscard]] int backward(const Call& c, cudaStream_t st);

}  // namespace train_attn
}  // namespace bnb
