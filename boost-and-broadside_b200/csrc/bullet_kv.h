// Keys and values of the bullet tokens (bullet_kv.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace bnb {
namespace tensor {

// norm_bullet + kv_bullet of bullet rows into kvb (rows, 256) = k | v: all n_rows rows in order, or, with index and
// n_rows_dev (on the device, at most n_rows), the first *n_rows_dev rows of index.  image: the packed weights, keys
// then values, with the norm's gain inside.
int bullet_kv(const void* rows, bool rows_bf16, int n_rows, const int* index, const int* n_rows_dev, const uint8_t* image, __nv_bfloat16* kvb,
              int* status, cudaStream_t st);

}  // namespace tensor
}  // namespace bnb
