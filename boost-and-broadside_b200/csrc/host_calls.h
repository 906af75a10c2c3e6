// Calls of the library that its own Python binding makes beside the C ABI (host_path.cpp): the same
// validation and dispatch as the entry points of include/bnb_trunk.h, with what only a caller that
// owns the whole call can ask for.
#pragma once
#include <stddef.h>

#include "bnb_trunk.h"

namespace bnb {
namespace host {

// bnb_trunk_step / bnb_trunk_sequence (is_sequence).  pack: the weight images named by the structs'
// `packed` fields are written from the live parameters first, by a launch that also clears the status
// word, so that the call needs no memset of its own.
int trunk_call(const BnbSpatialWeights* spatial, const BnbTemporalWeights* temporal, int n_blocks, int n_spatial, int n_temporal,
               int D, int H, const void* x, const uint8_t* alive, const BnbBullets* bullets, void* y, const float* hidden_in,
               float* hidden_out, const uint8_t* done, const uint8_t* reset_env, const BnbBatch* batch, int T, int precision,
               int engine, void* scratch, size_t scratch_bytes, void* stream, bool is_sequence, bool pack);

// n bfloat16 elements as float32 (n a multiple of 8, both 16-byte aligned).
int widen(const void* bf16, float* out, size_t n, void* stream);

}  // namespace host
}  // namespace bnb
