// What follows the trunk in a rollout step under the bfloat16 contract (policy_tail.cu): team pooling on
// the trunk's bfloat16 output, and the last kernel of the step (action draw, win values).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bnb_trunk.h"

namespace bnb {
namespace tail {

constexpr int MAX_SHIPS = 160;   // ships per environment the pooling kernel holds scores for

// Ships of the step: environment e's ship n is token row e * tokens + n of x, alive and team_id
// (team_id with rows of team_ld elements of its own).
struct Ships {
  const __nv_bfloat16* x;
  const uint8_t* alive;
  const void* team_id;
  int team_is_64, team_ld;
  int n_envs, ships, tokens;
};

size_t scratch_bytes();
// TeamPMA up to the gather: rows (n_envs * 2, 128) bfloat16, row 2 e + t = team t of environment e.
int team_rows(const Ships& s, const float* seeds, const float* in_proj_w, const float* out_w, const float* norm_w, void* scratch,
              __nv_bfloat16* rows, cudaStream_t st);
// The draw of bnb_action_dist_fwd from bfloat16 logits (n_envs * ships, 12) and uniforms (.., 3), with a
// bfloat16 logprob; and value[ship][cols[i]] = win[its team's row][i].
int finish(const Ships& s, const __nv_bfloat16* logits, const float* uniforms, int64_t* action, __nv_bfloat16* logprob,
           const __nv_bfloat16* win, int n_win, const uint8_t* cols, __nv_bfloat16* value, int value_ld, cudaStream_t st);

}  // namespace tail
}  // namespace bnb
