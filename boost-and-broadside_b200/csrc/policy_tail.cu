// Team pooling and the last kernel of a rollout step, on the trunk's bfloat16 output.
//
// TeamPMA (models/yemong/policy.py:78-121) attends from one seed per team over that team's alive ships.
// Two identities take the key / value projection of every ship out of it:
//   score(t, h, n) = q_th . (Wk_h x_n) = (Wk_h^T q_th) . x_n     the folded query is the same for every ship
//   sum_n p_n (Wv_h x_n)               = Wv_h (sum_n p_n x_n)    pool first, project one row per team and head
// so the kernel reads each ship row (256 bytes) twice and multiplies 2 x 4 rows per environment instead
// of every ship.  Against the key/value product it replaces (65 536 ships x 256 float32 columns written
// and read back, 31 + 77 us at 8192 environments of 8 ships) the traffic is the ship rows alone.
#include "policy_tail.h"

#include "common.cuh"
#include "launch_after.h"
#include "tensor_common.cuh"

namespace bnb {
namespace tail {

using tensor::ldsm_x4;
using tensor::mma_bf16;
using tensor::pack_bf16;
using tensor::smem_u32;

namespace {

constexpr int D = 128, H = 4, DH = 32;
constexpr int ENVS = 16;              // environments per CTA round: one per warp, 32 team rows
constexpr int WARPS = ENVS, THREADS = 32 * WARPS;
constexpr int LDW = D + 8;            // bf16 row strides: ldmatrix without bank conflicts
constexpr int LDP = H * D + 8;
constexpr int LDR = D + 4;            // float row stride

// shared memory (bytes)
constexpr int OFF_WV = 0;
constexpr int OFF_WO = OFF_WV + D * LDW * 2;
constexpr int OFF_P = OFF_WO + D * LDW * 2;             // pooled rows (32, 4 x 128)
constexpr int OFF_O = OFF_P + 2 * ENVS * LDP * 2;       // projected rows (32, 128)
constexpr int OFF_R = OFF_O + 2 * ENVS * LDW * 2;       // out_proj rows, float
constexpr int OFF_QK = OFF_R + 2 * ENVS * LDR * 4;      // folded queries (2, 4, 128)
constexpr int OFF_HAS = OFF_QK + 8 * D * 4;
constexpr int OFF_SC = OFF_HAS + 2 * ENVS * 4;          // per warp: ships x 4 weights

__device__ __forceinline__ int team_of(const Ships& s, size_t e, int n) {
  return s.team_is_64 ? (int)static_cast<const int64_t*>(s.team_id)[e * s.team_ld + n] : static_cast<const int32_t*>(s.team_id)[e * s.team_ld + n];
}

// One block per (team, head): q = bf16(Wq_h seed), folded query = Wk_h^T q / sqrt(32).
__global__ void __launch_bounds__(128) k_fold_query(const float* __restrict__ seeds, const float* __restrict__ in_proj, float* __restrict__ qk) {
  __shared__ float q[DH];
  tensor::let_next_start();
  tensor::wait_for_previous();
  const int t = blockIdx.x / H, h = blockIdx.x % H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float4 sv = *reinterpret_cast<const float4*>(seeds + t * D + lane * 4);
  for (int d = warp; d < DH; d += 4) {
    const float4 w = *reinterpret_cast<const float4*>(in_proj + (size_t)(h * DH + d) * D + lane * 4);
    float a = round_bf16(sv.x) * round_bf16(w.x) + round_bf16(sv.y) * round_bf16(w.y) + round_bf16(sv.z) * round_bf16(w.z) + round_bf16(sv.w) * round_bf16(w.w);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) q[d] = round_bf16(a);
  }
  __syncthreads();
  const float* wk = in_proj + (size_t)(D + h * DH) * D + threadIdx.x;
  float acc = 0.f;
#pragma unroll 8
  for (int d = 0; d < DH; ++d) acc = fmaf(q[d], round_bf16(wk[(size_t)d * D]), acc);
  qk[blockIdx.x * D + threadIdx.x] = acc * 0.17677669529663687f;
}

// out[32 x 8 columns of this warp] = A[32 x 128] * W[8 rows n0.. x 128]^T
__device__ __forceinline__ void rows_product(float (&acc)[2][4], uint32_t sA, int lda, uint32_t sW, int n0, int lane) {
  const int a_row = lane & 15, a_k = (lane >> 4) * 8;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[m][i] = 0.f;
#pragma unroll
  for (int kp = 0; kp < 4; ++kp) {   // two k steps of 16 per B load
    uint32_t b0, b1, b2, b3;
    ldsm_x4(sW + ((n0 + (lane & 7)) * LDW + kp * 32 + (lane >> 3) * 8) * 2, b0, b1, b2, b3);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      uint32_t a0, a1, a2, a3;
      ldsm_x4(sA + ((m * 16 + a_row) * lda + kp * 32 + a_k) * 2, a0, a1, a2, a3);
      mma_bf16(acc[m], a0, a1, a2, a3, b0, b1);
      ldsm_x4(sA + ((m * 16 + a_row) * lda + kp * 32 + 16 + a_k) * 2, a0, a1, a2, a3);
      mma_bf16(acc[m], a0, a1, a2, a3, b2, b3);
    }
  }
}

// Persistent CTAs of 16 warps, both weights resident as bfloat16.  A round is 16 environments: a warp
// scores and pools one of them (a lane owns 4 channels, so a ship row is one 256-byte request), then the
// 32 team rows go through Wv and out_proj as mma.sync products of 8 columns per warp.  Bound by latency: 55 us for
// 8192 environments of 8 ships, issue slots 27 % busy, DRAM 4 % of its peak, a warp's rows read one after the other.
__global__ void __launch_bounds__(THREADS, 1) k_team_rows(const Ships s, const float* __restrict__ qk, const float* __restrict__ in_proj,
                                                          const float* __restrict__ out_w, const float* __restrict__ norm_w,
                                                          __nv_bfloat16* __restrict__ rows) {
  extern __shared__ __align__(16) uint8_t sm[];
  tensor::let_next_start();
  tensor::wait_for_previous();
  __nv_bfloat16* P = reinterpret_cast<__nv_bfloat16*>(sm + OFF_P);
  __nv_bfloat16* O = reinterpret_cast<__nv_bfloat16*>(sm + OFF_O);
  float* R = reinterpret_cast<float*>(sm + OFF_R);
  float* QK = reinterpret_cast<float*>(sm + OFF_QK);
  float* has = reinterpret_cast<float*>(sm + OFF_HAS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* sc = reinterpret_cast<float*>(sm + OFF_SC) + (size_t)warp * s.ships * H;
#pragma unroll 4
  for (int i = tid; i < 2 * D * (D / 4); i += THREADS) {
    const int w = i / (D * (D / 4)), j = i - w * D * (D / 4), r = j / (D / 4), q = j % (D / 4);
    const float4 v = *reinterpret_cast<const float4*>((w ? out_w : in_proj + (size_t)2 * D * D) + (size_t)r * D + q * 4);
    *reinterpret_cast<uint2*>(sm + (w ? OFF_WO : OFF_WV) + (r * LDW + q * 4) * 2) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
  }
  for (int i = tid; i < 8 * D; i += THREADS) QK[i] = qk[i];
  __syncthreads();
  const float4 gain = *reinterpret_cast<const float4*>(norm_w + lane * 4);

  for (int e0 = blockIdx.x * ENVS; e0 < s.n_envs; e0 += gridDim.x * ENVS) {
    const int e = e0 + warp;
    float acc[2][H][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int h = 0; h < H; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][h][i] = 0.f;
    bool any[2] = {false, false};
    if (e < s.n_envs) {
      const uint2* xr = reinterpret_cast<const uint2*>(s.x + (size_t)e * s.tokens * D) + lane;
      const uint8_t* al = s.alive + (size_t)e * s.tokens;
      // scores: four heads of the ship's own team, reduced over the lanes four values at a time
      for (int n = 0; n < s.ships; ++n) {
        const int t = team_of(s, e, n);
        const bool ok = al[n] && (t == 0 || t == 1);
        float v = -INFINITY;
        if (ok) {
          const uint2 w = xr[(size_t)n * (D / 4)];
          const float x0 = tensor::bf16_lo(w.x), x1 = tensor::bf16_hi(w.x), x2 = tensor::bf16_lo(w.y), x3 = tensor::bf16_hi(w.y);
          float p[H];
#pragma unroll
          for (int h = 0; h < H; ++h) {
            const float4 k = *reinterpret_cast<const float4*>(QK + (t * H + h) * D + lane * 4);
            p[h] = fmaf(k.x, x0, fmaf(k.y, x1, fmaf(k.z, x2, k.w * x3)));
          }
          // lanes below 16 keep heads 0, 1, the others heads 2, 3; then one head per group of eight
          const bool up = lane & 16;
          const float s0 = __shfl_xor_sync(0xffffffffu, up ? p[0] : p[2], 16), s1 = __shfl_xor_sync(0xffffffffu, up ? p[1] : p[3], 16);
          const float a = (up ? p[2] : p[0]) + s0, b = (up ? p[3] : p[1]) + s1;
          const bool odd = lane & 8;
          v = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 2);
          v += __shfl_xor_sync(0xffffffffu, v, 1);
          any[0] |= t == 0;
          any[1] |= t == 1;
        }
        if ((lane & 7) == 0) sc[n * H + (lane >> 3)] = v;
      }
      __syncwarp();
      // softmax per (team, head): eight lanes per head walk the ships
      {
        const int h = lane >> 3, j0 = lane & 7;
        float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
        for (int n = j0; n < s.ships; n += 8) {
          const int t = min(max(team_of(s, e, n), 0), 1);
          m[t] = fmaxf(m[t], sc[n * H + h]);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
          m[1] = fmaxf(m[1], __shfl_xor_sync(0xffffffffu, m[1], o));
        }
        for (int n = j0; n < s.ships; n += 8) {
          const int t = min(max(team_of(s, e, n), 0), 1);
          const float v = sc[n * H + h];
          const float ex = v == -INFINITY ? 0.f : expf(v - m[t]);
          sc[n * H + h] = ex;
          l[t] += ex;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          l[0] += __shfl_xor_sync(0xffffffffu, l[0], o);
          l[1] += __shfl_xor_sync(0xffffffffu, l[1], o);
        }
        for (int n = j0; n < s.ships; n += 8) {
          const int t = min(max(team_of(s, e, n), 0), 1);
          if (l[t] > 0.f) sc[n * H + h] /= l[t];
        }
      }
      __syncwarp();
      for (int n = 0; n < s.ships; ++n) {
        const int t = team_of(s, e, n);
        if (!al[n] || (t != 0 && t != 1)) continue;
        const uint2 w = xr[(size_t)n * (D / 4)];
        const float x[4] = {tensor::bf16_lo(w.x), tensor::bf16_hi(w.x), tensor::bf16_lo(w.y), tensor::bf16_hi(w.y)};
        const float4 p4 = *reinterpret_cast<const float4*>(sc + n * H);
        const float p[H] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
        for (int tt = 0; tt < 2; ++tt)
          if (tt == t) {
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
              for (int i = 0; i < 4; ++i) acc[tt][h][i] = fmaf(p[h], x[i], acc[tt][h][i]);
          }
      }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
      for (int h = 0; h < H; ++h)
        *reinterpret_cast<uint2*>(P + (2 * warp + t) * LDP + h * D + lane * 4) =
            make_uint2(pack_bf16(acc[t][h][0], acc[t][h][1]), pack_bf16(acc[t][h][2], acc[t][h][3]));
      if (lane == 0) has[2 * warp + t] = any[t] ? 1.f : 0.f;
    }
    __syncthreads();
    const int g = lane >> 2, c = warp * 8 + 2 * (lane & 3);
    float out[2][4];
    rows_product(out, smem_u32(P + (warp >> 2) * D), LDP, smem_u32(sm + OFF_WV), warp * 8, lane);   // columns of head warp / 4
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      *reinterpret_cast<uint32_t*>(O + (m * 16 + g) * LDW + c) = pack_bf16(out[m][0], out[m][1]);
      *reinterpret_cast<uint32_t*>(O + (m * 16 + g + 8) * LDW + c) = pack_bf16(out[m][2], out[m][3]);
    }
    __syncthreads();
    rows_product(out, smem_u32(O), LDW, smem_u32(sm + OFF_WO), warp * 8, lane);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = m * 16 + g + 8 * i;
        *reinterpret_cast<float2*>(R + r * LDR + c) = make_float2(round_bf16(out[m][2 * i]) * has[r], round_bf16(out[m][2 * i + 1]) * has[r]);
      }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int r = 2 * warp + t;
      const float4 v = *reinterpret_cast<const float4*>(R + r * LDR + lane * 4);
      float ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float inv = rsqrtf(ss * (1.0f / D) + kRmsEps);
      if (e < s.n_envs)
        *reinterpret_cast<uint2*>(rows + ((size_t)e * 2 + t) * D + lane * 4) =
            make_uint2(pack_bf16(v.x * inv * gain.x, v.y * inv * gain.y), pack_bf16(v.z * inv * gain.z, v.w * inv * gain.w));
    }
    // the next round's first writes to P, has, O and R each come after a barrier that follows these reads
  }
}

struct WinCols { uint8_t c[32]; };

// One thread per ship: three categorical draws over the logit slices [0, 3), [3, 10), [10, 12)
// (constants.py:43-48) by inverse CDF, the sum of their log-probabilities rounded as
// torch.distributions.Categorical's are under autocast, and the win values of the ship's team.
__global__ void __launch_bounds__(128) k_finish(const Ships s, const __nv_bfloat16* __restrict__ logits, const float* __restrict__ uniforms,
                                                int64_t* __restrict__ action, __nv_bfloat16* __restrict__ logprob,
                                                const __nv_bfloat16* __restrict__ win, int n_win, const WinCols cols,
                                                __nv_bfloat16* __restrict__ value, int value_ld) {
  tensor::let_next_start();
  tensor::wait_for_previous();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= s.n_envs * s.ships) return;
  float lg[12];
  {
    const uint2* p = reinterpret_cast<const uint2*>(logits + (size_t)r * 12);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint2 w = p[i];
      lg[4 * i] = tensor::bf16_lo(w.x); lg[4 * i + 1] = tensor::bf16_hi(w.x);
      lg[4 * i + 2] = tensor::bf16_lo(w.y); lg[4 * i + 3] = tensor::bf16_hi(w.y);
    }
  }
  float lp_sum = 0.f;
  constexpr int lo[3] = {0, 3, 10}, hi[3] = {3, 10, 12};
#pragma unroll
  for (int sl = 0; sl < 3; ++sl) {
    float m = -INFINITY;
#pragma unroll
    for (int k = lo[sl]; k < hi[sl]; ++k) m = fmaxf(m, lg[k]);
    float l = 0.f;
#pragma unroll
    for (int k = lo[sl]; k < hi[sl]; ++k) l += expf(lg[k] - m);
    const float lse = round_bf16(m + logf(l));
    const float target = uniforms[(size_t)r * 3 + sl] * l;   // the first k with target < sum_{j <= k} exp(v_j - m)
    float c = 0.f, chosen = lg[hi[sl] - 1];
    int pick = hi[sl] - 1 - lo[sl];
    bool found = false;
#pragma unroll
    for (int k = lo[sl]; k < hi[sl]; ++k) {
      c += expf(lg[k] - m);
      if (!found && target < c) {
        found = true;
        pick = k - lo[sl];
        chosen = lg[k];
      }
    }
    action[(size_t)r * 3 + sl] = pick;
    lp_sum = round_bf16(lp_sum + round_bf16(chosen - lse));
  }
  logprob[r] = __float2bfloat16_rn(lp_sum);
  if (n_win > 0) {
    const int e = r / s.ships;
    const int t = min(max(team_of(s, e, r - e * s.ships), 0), 1);
    for (int i = 0; i < n_win; ++i) value[(size_t)r * value_ld + cols.c[i]] = win[((size_t)e * 2 + t) * n_win + i];
  }
}

}  // namespace

size_t scratch_bytes() { return 8 * D * sizeof(float); }

int team_rows(const Ships& s, const float* seeds, const float* in_proj_w, const float* out_w, const float* norm_w, void* scratch,
              __nv_bfloat16* rows, cudaStream_t st) {
  if (s.ships < 1 || s.ships > MAX_SHIPS) return BNB_ERR_TOO_MANY_TOKENS;
  if (s.n_envs <= 0) return BNB_OK;
  const size_t smem = OFF_SC + (size_t)WARPS * s.ships * H * sizeof(float);
  if (cudaFuncSetAttribute(k_team_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return BNB_ERR_LAUNCH;
  float* qk = static_cast<float*>(scratch);
  if (const int rc = launch_after(k_fold_query, dim3(2 * H), 128, 0, st, seeds, in_proj_w, qk)) return rc;
  const int rounds = (s.n_envs + ENVS - 1) / ENVS;
  return launch_after(k_team_rows, dim3(rounds < 148 ? rounds : 148), THREADS, smem, st, s, qk, in_proj_w, out_w, norm_w, rows);
}

int finish(const Ships& s, const __nv_bfloat16* logits, const float* uniforms, int64_t* action, __nv_bfloat16* logprob,
           const __nv_bfloat16* win, int n_win, const uint8_t* cols, __nv_bfloat16* value, int value_ld, cudaStream_t st) {
  const int n = s.n_envs * s.ships;
  if (n <= 0) return BNB_OK;
  WinCols wc{};
  for (int i = 0; i < n_win && i < 32; ++i) wc.c[i] = cols[i];
  return launch_after(k_finish, dim3((n + 127) / 128), 128, 0, st, s, logits, uniforms, action, logprob, win, n_win, wc, value, value_ld);
}

}  // namespace tail
}  // namespace bnb
