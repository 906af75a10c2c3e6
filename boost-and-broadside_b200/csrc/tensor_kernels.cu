// Host side of the tensor-core trunk (bfloat16 contract): weight images, tile plans, the split of a call into
// launches, and the kernels around the fused one (pipelined_tile_kernel.cu): attention of environments larger than a
// tile or with bullets, compaction of the active bullets.
//
// A tile is 128 token rows of whole environments.  A call is a program of sublayers (S = spatial, T = temporal) that
// one launch walks tile by tile; a spatial sublayer that needs the separate attention kernel splits the program there.
//
// Every wait on an mbarrier is bounded; a wait that runs out records a code in the status word and the kernel drains
// without hanging.
//
// Reference arithmetic: models/yemong/attention.py:76-169, models/yemong/griffin.py:67-317.
#include "bullet_kv.h"
#include "bullet_slices.h"
#include "tensor_kernels.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "launch_after.h"

#include "tensor_common.cuh"

namespace bnb {
namespace tensor {

int g_debug_poll_limit = 0;
int g_debug_skip_op = -1;

// ------------------------------------------------------------------ weight image

// Source of row `r` (0..127) of chunk `c` of a sublayer image: pointer to 64 consecutive
// floats, or nullptr for a zero row.
__device__ __forceinline__ const float* ffn_chunk_row(int c, int r, const float* gate, const float* up, const float* down) {
  int cc = c / 3, i = c % 3;
  if (i < 2) return (r < 64 ? gate + (size_t)(64 * cc + r) * D : up + (size_t)(64 * cc + r - 64) * D) + i * 64;
  return down + (size_t)r * 4 * D + 64 * cc;
}
__device__ __forceinline__ const float* spatial_chunk_row(const BnbSpatialWeights& w, int c, int r) {
  // two K halves each of q, k, v (all heads) and out_proj
  if (c < 6) return w.qkv_w + (size_t)((c >> 1) * D + r) * D + (c & 1) * 64;
  if (c < 8) return w.out_w + (size_t)r * D + (c & 1) * 64;
  if (c >= N_SPATIAL_CHUNKS) {
    // kv_bullet (2D, D): rows 0..127 are the keys of all heads, 128..255 the values
    if (!w.kv_bullet_w) return nullptr;
    const int i = c - N_SPATIAL_CHUNKS;
    return w.kv_bullet_w + (size_t)((i >> 1) * D + r) * D + (i & 1) * 64;
  }
  return ffn_chunk_row(c - 8, r, w.gate_w, w.up_w, w.down_w);
}
__device__ __forceinline__ const float* temporal_chunk_row(const BnbTemporalWeights& w, int c, int r) {
  int kh = c & 1;
  switch (c >> 1) {
    case 0: return w.linear2_w + (size_t)r * D + kh * 64;
    case 1: return w.linear1_w + (size_t)r * D + kh * 64;
    case 2: return (r < 64 ? w.a_w + (size_t)r * D : w.x_w + (size_t)(r - 64) * D) + kh * 64;
    case 3: return (r < 64 ? w.a_w + (size_t)(64 + r) * D : w.x_w + (size_t)r * D) + kh * 64;
    case 4: return w.field_sub_w ? w.field_sub_w + (size_t)r * D + kh * 64 : nullptr;
    case 5: return w.out_w + (size_t)r * D + kh * 64;
    default: return ffn_chunk_row(c - 12, r, w.gate_w, w.up_w, w.down_w);
  }
}

// RMSNorm gain folded into chunk `c`: the 64 gains of the chunk's K columns when the chunk's
// input is a normed activation, else nullptr.  The kernels then feed x * rsqrt(mean x^2 + eps)
// without the gain, and the products see W[n][k] * g[k] rounded to bf16 once.
__device__ __forceinline__ const float* spatial_chunk_gain(const BnbSpatialWeights& w, int c) {
  if (c < 8) return c < 6 ? w.norm1_w + (c & 1) * 64 : nullptr;
  if (c >= N_SPATIAL_CHUNKS) return w.norm_bullet_w ? w.norm_bullet_w + ((c - N_SPATIAL_CHUNKS) & 1) * 64 : nullptr;
  const int i = (c - 8) % 3;
  return i < 2 ? w.norm2_w + i * 64 : nullptr;
}
__device__ __forceinline__ const float* temporal_chunk_gain(const BnbTemporalWeights& w, int c) {
  if (c < 4) return w.norm1_w + (c & 1) * 64;        // linear2, linear1
  if (c < 12) return nullptr;                         // gates, field_sub, linear_out: not fed by a norm
  const int i = (c - 12) % 3;
  return i < 2 ? w.norm2_w + i * 64 : nullptr;
}

// Some rows are stored halved (exactly): the elementwise part of the GatedMLP works on gate / 2 (gelu_half_mul).
__device__ __forceinline__ bool ffn_gate_row(int c, int r) { return c % 3 < 2 && r < 64; }

template <class W, class F, class G, class H>
__device__ __forceinline__ void pack_image(const W& w, int n_chunks, uint8_t* out, F row_of, G gain_of, H halved) {
  // one thread per 16-byte group: (chunk, row, group of 8 columns)
  const int total = n_chunks * TILE * 8;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int c = i / (TILE * 8), r = (i / 8) % TILE, g = i % 8;
    const float* src = row_of(w, c, r);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (src) {
      float4 a = *reinterpret_cast<const float4*>(src + g * 8);
      float4 b = *reinterpret_cast<const float4*>(src + g * 8 + 4);
      if (const float* gain = gain_of(w, c)) {
        const float4 ga = *reinterpret_cast<const float4*>(gain + g * 8), gb = *reinterpret_cast<const float4*>(gain + g * 8 + 4);
        a.x *= ga.x; a.y *= ga.y; a.z *= ga.z; a.w *= ga.w;
        b.x *= gb.x; b.y *= gb.y; b.z *= gb.z; b.w *= gb.w;
      }
      if (halved(c, r)) {
        a.x *= 0.5f; a.y *= 0.5f; a.z *= 0.5f; a.w *= 0.5f;
        b.x *= 0.5f; b.y *= 0.5f; b.z *= 0.5f; b.w *= 0.5f;
      }
      v = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
    }
    *reinterpret_cast<uint4*>(out + (size_t)c * CHUNK_BYTES + swz(r, g)) = v;
  }
}
__device__ __forceinline__ bool spatial_chunk_halved(int c, int r) { return c >= 8 && c < N_SPATIAL_CHUNKS && ffn_gate_row(c - 8, r); }
// linear2 (GELU) and the recurrence's gates (tanh form of the sigmoid) are wanted halved as well
__device__ __forceinline__ bool temporal_chunk_halved(int c, int r) { return c < 12 ? c < 2 || (c >= 4 && c < 8) : ffn_gate_row(c - 12, r); }
// What stands behind the chunks of a temporal image (SubLayer::decay_log2).
__device__ __forceinline__ void pack_recurrence(const BnbTemporalWeights& w, uint8_t* out) {
  float* t = reinterpret_cast<float*>(out + (size_t)N_TEMPORAL_CHUNKS * CHUNK_BYTES);
  const int i = threadIdx.x;
  const float sg = 1.0f / (1.0f + expf(-w.log_lambda[i]));
  t[i] = kRglruC * (sg == 0.f ? kLogOfZero : log2f(sg));
  t[D + i] = 0.5f * w.a_b[i];
  t[2 * D + i] = 0.5f * w.x_b[i];
}
__global__ void k_pack_spatial(BnbSpatialWeights w, uint8_t* out) {
  pack_image(w, N_SPATIAL_IMAGE, out, [](const BnbSpatialWeights& ww, int c, int r) { return spatial_chunk_row(ww, c, r); },
             [](const BnbSpatialWeights& ww, int c) { return spatial_chunk_gain(ww, c); }, [](int c, int r) { return spatial_chunk_halved(c, r); });
}
__global__ void k_pack_temporal(BnbTemporalWeights w, uint8_t* out) {
  if (blockIdx.x == 0 && threadIdx.x < D) pack_recurrence(w, out);
  pack_image(w, N_TEMPORAL_CHUNKS, out, [](const BnbTemporalWeights& ww, int c, int r) { return temporal_chunk_row(ww, c, r); },
             [](const BnbTemporalWeights& ww, int c) { return temporal_chunk_gain(ww, c); }, [](int c, int r) { return temporal_chunk_halved(c, r); });
}

// Every image of a trunk in one launch: blockIdx.y selects the sublayer.
constexpr int MAX_PACK_JOBS = 8;
// One 16-byte group per thread: with a sixth of the blocks, six of them one after the other, the launch took 4.4 us; step of 16 x 12 tokens 78.6 -> 77.1 us with the masks of a row table read at once.
constexpr int PACK_BLOCKS = (N_TEMPORAL_CHUNKS > N_SPATIAL_IMAGE ? N_TEMPORAL_CHUNKS : N_SPATIAL_IMAGE) * TILE * 8 / 256;
struct PackJobs {
  int n_spatial, n_temporal;
  int* status;   // zeroed by the launch (null: nobody asked)
  BnbSpatialWeights sw[MAX_PACK_JOBS];
  BnbTemporalWeights tw[MAX_PACK_JOBS];
};
__global__ void k_pack_trunk(const __grid_constant__ PackJobs jobs) {
  const int j = blockIdx.y;
  let_next_start();
  wait_for_previous();
  if (jobs.status && j == 0 && blockIdx.x == 0 && threadIdx.x == 0) *jobs.status = 0;
  if (j < jobs.n_spatial) {
    const BnbSpatialWeights& w = jobs.sw[j];
    pack_image(w, N_SPATIAL_IMAGE, static_cast<uint8_t*>(const_cast<void*>(w.packed)),
               [](const BnbSpatialWeights& ww, int c, int r) { return spatial_chunk_row(ww, c, r); },
               [](const BnbSpatialWeights& ww, int c) { return spatial_chunk_gain(ww, c); }, [](int c, int r) { return spatial_chunk_halved(c, r); });
  } else {
    const BnbTemporalWeights& w = jobs.tw[j - jobs.n_spatial];
    uint8_t* out = static_cast<uint8_t*>(const_cast<void*>(w.packed));
    if (blockIdx.x == 0 && threadIdx.x < D) pack_recurrence(w, out);
    pack_image(w, N_TEMPORAL_CHUNKS, out, [](const BnbTemporalWeights& ww, int c, int r) { return temporal_chunk_row(ww, c, r); },
               [](const BnbTemporalWeights& ww, int c) { return temporal_chunk_gain(ww, c); }, [](int c, int r) { return temporal_chunk_halved(c, r); });
  }
}

// ------------------------------------------------------------------ attention kernel of the split path
//
// One CTA per (environment, head): q, k, v of that head are staged from the bf16 scratch the
// PRE phase wrote, then each warp takes blocks of 16 query rows and walks the keys in blocks of
// 32 (the last up to 16 by themselves) with a running maximum (mma.sync, fp32 softmax).  Dead keys score kMaskedScore, so their
// weight is exactly 0 unless no key of the environment is alive, in which case every key gets
// the same weight (models/yemong/attention.py:101-112 of the reference).  When the sublayer
// reads bullets, the environment's bullet keys and values (written by bullet_kv.cu) are
// staged too and get a softmax of their own; its output, gated to zero when the environment has
// no active bullet, is added to the self-attention output (attention.py:149-166).
// A CTA stages HPC heads of one environment (all four when they fit in shared memory, else one):
// a staged row holds HPC x 32 bf16 plus 16 bytes of padding, which keeps ldmatrix conflict-free.
__host__ __device__ constexpr int flash_stride(int hpc) { return hpc * 64 + 16; }

// Running softmax of a block of 16 queries: a lane's two query rows, the sums of its own columns side by side.  A row's sum takes
// its two columns of 8 keys together and those of the blocks one after the other, whatever the stage: an order of its own for
// each size moves the last bits of the result, and bfloat16 roundings of the sublayers behind it carry that on (1e-4 of the state).
struct FlashState {
  float m[2];
  F2 l;
  float acc[4][4];
};
// One block of 8 NT keys from key0 on (at least one of them a key).  k and v: staged rows at this head and this lane's ldmatrix
// column.  bias: one float per key, 0 for a live one, kMaskedScore for a dead one, -inf past the last.  Scores are carried in the log2
// domain: t = (q.k) * log2(e) / sqrt(32) + bias, p = 2^(t - max).  FIRST: nothing to rescale.
template <int HPC, int NT, bool FIRST>
__device__ __forceinline__ void flash_block(FlashState& f, const uint32_t (&qa)[2][4], uint32_t k, uint32_t v, const float* bias, int key0, int last, int lane) {
  constexpr int STRIDE = flash_stride(HPC);
  float sc[NT][4];
#pragma unroll
  for (int h = 0; h < NT / 2; ++h) {
    const uint32_t row = k + min(key0 + h * 16 + (lane >> 4) * 8 + (lane & 7), last) * STRIDE;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      uint32_t b0, b1, b2, b3;
      ldsm_x4(row + ks * 32, b0, b1, b2, b3);
      if (ks == 0) {
        mma_bf16_fresh(sc[2 * h], qa[ks], b0, b1);
        mma_bf16_fresh(sc[2 * h + 1], qa[ks], b2, b3);
      } else {
        mma_bf16(sc[2 * h], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
        mma_bf16(sc[2 * h + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
      }
    }
  }
  const F2 c2 = f2(0.17677669529663687f * 1.4426950408889634f);
  F2 t[NT][2];
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    // a dead key's bias swallows its score: kMaskedScore exactly (weight 0 unless every key is dead)
    F2 bj;
    bj.v = *reinterpret_cast<const unsigned long long*>(bias + key0 + nt * 8 + 2 * (lane & 3));
    t[nt][0] = fma(f2(sc[nt][0], sc[nt][1]), c2, bj);
    t[nt][1] = fma(f2(sc[nt][2], sc[nt][3]), c2, bj);
    const float2 a = halves(t[nt][0]), b = halves(t[nt][1]);
    m0 = fmaxf(m0, fmaxf(a.x, a.y));
    m1 = fmaxf(m1, fmaxf(b.x, b.y));
  }
  m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1));
  m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2));
  m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1));
  m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
  if constexpr (!FIRST) {
    m0 = fmaxf(m0, f.m[0]);
    m1 = fmaxf(m1, f.m[1]);
    const float c0 = ex2_fast(f.m[0] - m0), c1 = ex2_fast(f.m[1] - m1);
    f.l = mul(f.l, f2(c0, c1));
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 a = halves(mul(f2(f.acc[nt][0], f.acc[nt][1]), f2(c0))), b = halves(mul(f2(f.acc[nt][2], f.acc[nt][3]), f2(c1)));
      f.acc[nt][0] = a.x; f.acc[nt][1] = a.y; f.acc[nt][2] = b.x; f.acc[nt][3] = b.y;
    }
  }
  f.m[0] = m0;
  f.m[1] = m1;
  uint32_t p[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const float2 d0 = halves(add(t[nt][0], f2(-m0))), d1 = halves(add(t[nt][1], f2(-m1)));
    const float2 e0 = make_float2(ex2_fast(d0.x), ex2_fast(d0.y)), e1 = make_float2(ex2_fast(d1.x), ex2_fast(d1.y));
    const F2 both = add(f2(e0.x, e1.x), f2(e0.y, e1.y));
    f.l = FIRST && nt == 0 ? both : add(f.l, both);
    p[nt][0] = pack_bf16(e0.x, e0.y);
    p[nt][1] = pack_bf16(e1.x, e1.y);
  }
#pragma unroll
  for (int h = 0; h < NT / 2; ++h) {
    const uint32_t row = v + min(key0 + h * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), last) * STRIDE;
    const uint32_t a[4] = {p[2 * h][0], p[2 * h][1], p[2 * h + 1][0], p[2 * h + 1][1]};
#pragma unroll
    for (int np = 0; np < 2; ++np) {
      uint32_t b0, b1, b2, b3;
      ldsm_x4_t(row + np * 32, b0, b1, b2, b3);
      if (FIRST && h == 0) {
        mma_bf16_fresh(f.acc[np * 2], a, b0, b1);
        mma_bf16_fresh(f.acc[np * 2 + 1], a, b2, b3);
      } else {
        mma_bf16(f.acc[np * 2], a[0], a[1], a[2], a[3], b0, b1);
        mma_bf16(f.acc[np * 2 + 1], a[0], a[1], a[2], a[3], b2, b3);
      }
    }
  }
}
// n > 0 keys, 32 at a time and the last up to 16 by themselves; fresh: the first ones of their softmax.
template <int HPC>
__device__ __forceinline__ void flash_walk(FlashState& f, bool fresh, const uint32_t (&qa)[2][4], uint32_t k, uint32_t v, const float* bias, int n, int lane) {
  int key = 0;
  if (fresh) {
    if (n > 16) flash_block<HPC, 4, true>(f, qa, k, v, bias, 0, n - 1, lane);
    else flash_block<HPC, 2, true>(f, qa, k, v, bias, 0, n - 1, lane);
    key = n > 16 ? 32 : 16;
  }
#pragma unroll 1
  for (; key + 16 < n; key += 32) flash_block<HPC, 4, false>(f, qa, k, v, bias, key, n - 1, lane);
  if (key < n) flash_block<HPC, 2, false>(f, qa, k, v, bias, key, n - 1, lane);
}
// The normalised output.
__device__ __forceinline__ void flash_finish(FlashState& f) {
  const float2 sums = halves(f.l);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float l = r ? sums.y : sums.x;
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const float inv = 1.0f / l;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      f.acc[nt][2 * r] *= inv;
      f.acc[nt][2 * r + 1] *= inv;
    }
  }
}

// env_base: first environment (group-major) of this launch.  kvb holds the bullet keys and values
// of the launch's environments (null: none): with env_off, the rows of the active bullets only,
// environment i of the launch owning rows [env_off[i], env_off[i+1]) (an inactive bullet has
// weight exactly 0 and an environment without active bullets is gated off, so neither needs a
// row); without env_off, nb rows per environment, all of them keys (no mask was given).
// blockIdx.y selects a group of HPC heads; the warps (4 to 8, chosen by the launcher so that the
// (head, query block) pairs divide evenly) share the pairs out.
// stage: bullet rows staged at a time.  Fewer than an environment may have only where every warp has one pair at most, whose
// softmax then goes on over the next rows.
//
// Bound by latency and issue around small mma.sync tiles.  8192 environments of 12 tokens with 18 of 80 bullets 73.3 -> 48.5 us, 1024
// of 152 tokens 93.0 -> 80.2: keys past a block of 32 in one of 16, nothing to rescale in the first block (every block of most
// environments), pairs of scores in one instruction, the heads of a CTA a constant (divisions by it), 32 bullet rows of shared
// memory instead of every slot's (with 64 the step takes 837 us instead of 828), results out as whole rows.  A row's sum over pairs of
// its columns instead of over even and odd ones, and a division instead of a reciprocal, take 1.0 and 1.6 us of that.  One copy of the walk and
// loops that stay loops: a small launch waits for its instructions (28 environments of 6 tokens with bullets 117.3 us a step with a copy
// each, unrolled, 115.7 so; 1024 of 152 1404 and 1396).  Eighty registers with a few spilled: with 126 the steps take
// 844 us instead of 835 and 1432 instead of 1404, with 64 860 and 1404.
template <int HPC, bool BULLETS>
__global__ void __launch_bounds__(256, 3) k_attention_flash(const __nv_bfloat16* __restrict__ qkv, const uint8_t* __restrict__ alive,
                                                         __nv_bfloat16* __restrict__ o, EnvMap map, int env_base, int stage,
                                                         const __nv_bfloat16* __restrict__ kvb,
                                                         const int* __restrict__ env_off, int nb) {
  extern __shared__ __align__(16) uint8_t fs[];
  let_next_start();
  wait_for_previous();
  constexpr int STRIDE = flash_stride(HPC), GPR = HPC * 4;   // 16-byte groups per staged row
  const int env_g = env_base + blockIdx.x, hd0 = blockIdx.y * HPC;
  const int grp = env_g / map.n_envs, e = env_g - grp * map.n_envs;
  const size_t tok0 = (size_t)grp * map.total_tokens + map.env_tok_begin(e);
  const int n = map.env_tok_count(e);
  size_t brow0 = 0;
  if constexpr (!BULLETS) {
    nb = stage = 0;
  } else if (env_off) {
    brow0 = (size_t)env_off[blockIdx.x];
    nb = env_off[blockIdx.x + 1] - (int)brow0;
  } else {
    brow0 = (size_t)blockIdx.x * nb;
  }
  const int n_stage = min(nb, stage), n32 = (n + 31) & ~31, nb32 = (n_stage + 31) & ~31;
  // q, k, v rows, then bullet keys and values (stage rows each), then the biases; strides are multiples of 16 bytes
  const uint32_t q_at = smem_u32(fs), k_at = q_at + n * STRIDE, v_at = k_at + n * STRIDE, kb_at = v_at + n * STRIDE, vb_at = kb_at + n_stage * STRIDE;
  float* bias_s = reinterpret_cast<float*>(fs + (size_t)(3 * n + 2 * n_stage) * STRIDE);
  float* bias_b = bias_s + n32;
  const int threads = blockDim.x;
  // asynchronous 16-byte copies: all of them are in flight before the first one is waited for
  {
    const __nv_bfloat16* src = qkv + tok0 * (3 * D) + hd0 * DH;
#pragma unroll 1
    for (int i = threadIdx.x; i < n * 3 * GPR; i += threads) {
      const uint32_t r = (uint32_t)i / (3 * GPR), rem = (uint32_t)i % (3 * GPR), part = rem / GPR, q = rem % GPR;
      cp_async16(q_at + (part * n + r) * STRIDE + q * 16, src + r * (3 * D) + part * D + q * 8);
    }
  }
  auto stage_bullets = [&](int b0, int rows) {
    const __nv_bfloat16* src = kvb + (brow0 + b0) * (2 * D) + hd0 * DH;
#pragma unroll 1
    for (int i = threadIdx.x; i < rows * 2 * GPR; i += threads) {
      const uint32_t r = (uint32_t)i / (2 * GPR), rem = (uint32_t)i % (2 * GPR), part = rem / GPR, q = rem % GPR;
      cp_async16((part ? vb_at : kb_at) + r * STRIDE + q * 16, src + r * (2 * D) + part * D + q * 8);
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < nb32; i += threads) bias_b[i] = i < rows ? 0.f : -INFINITY;
  };
  if (BULLETS && nb > 0) stage_bullets(0, n_stage);
#pragma unroll 1
  for (int i = threadIdx.x; i < n32; i += threads)
    bias_s[i] = i < n ? ((!alive || alive[tok0 + i]) ? 0.f : kMaskedScore) : -INFINITY;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int last = n - 1;
  const int items = HPC * ((n + 15) >> 4), n_warps = threads >> 5;
  const uint32_t k_lane = ((lane >> 3) & 1) * 16, v_lane = (lane >> 4) * 16;
  // a turn may have barriers in it (bullets that are staged piecewise): every warp takes part then
  const int turns = nb > stage ? 1 : (items - warp + n_warps - 1) / n_warps;
#pragma unroll 1
  for (int turn = 0; turn < turns; ++turn) {
    const int item = warp + turn * n_warps;
    const bool mine = item < items;
    const int hl = item % HPC, qb = item / HPC;
    const uint32_t hoff = (uint32_t)hl * 64;
    uint32_t qa[2][4], out[4][2];
    FlashState f;
    if (mine) {
      const int row = min(qb * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, last);
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
        ldsm_x4(q_at + hoff + row * STRIDE + (ks * 16 + (lane >> 4) * 8) * 2, qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
    }
    // The environment's own keys, then its bullets: one copy of the walk.
#pragma unroll 1
    for (int pass = 0; pass < (BULLETS && nb > 0 ? 2 : 1); ++pass) {
      const int keys = pass ? nb : n, step = pass ? stage : n;
      const uint32_t k = (pass ? kb_at : k_at) + hoff + k_lane, v = (pass ? vb_at : v_at) + hoff + v_lane;
#pragma unroll 1
      for (int b0 = 0; b0 < keys; b0 += step) {
        const int rows = min(step, keys - b0);
        if (b0 > 0) {   // bullets past the first stage
          __syncthreads();   // the rows before have been read
          if constexpr (BULLETS) stage_bullets(b0, rows);
          asm volatile("cp.async.wait_all;" ::: "memory");
          __syncthreads();
        }
        if (mine) flash_walk<HPC>(f, b0 == 0, qa, k, v, pass ? bias_b : bias_s, rows, lane);
      }
      if (!mine) continue;
      flash_finish(f);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t o16 = pack_bf16(f.acc[nt][2 * r], f.acc[nt][2 * r + 1]);
          // both outputs are bf16 tensors in the reference; so is their sum
          out[nt][r] = pass ? pack_bf16(bf16_lo(out[nt][r]) + bf16_lo(o16), bf16_hi(out[nt][r]) + bf16_hi(o16)) : o16;
        }
    }
    // into the place of these queries, which this warp alone reads
    if (mine) {
      const int q0 = qb * 16 + g;
      uint8_t* at = fs + q0 * STRIDE + hoff + 4 * t;
      __syncwarp();
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        if (q0 <= last) *reinterpret_cast<uint32_t*>(at + nt * 16) = out[nt][0];
        if (q0 + 8 <= last) *reinterpret_cast<uint32_t*>(at + 8 * STRIDE + nt * 16) = out[nt][1];
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int i = threadIdx.x; i < n * GPR; i += threads) {
    const int r = i / GPR, q = i % GPR;
    *reinterpret_cast<uint4*>(o + (tok0 + r) * D + hd0 * DH + q * 8) = *reinterpret_cast<const uint4*>(fs + r * STRIDE + q * 16);
  }
}

// ------------------------------------------------------------------ compaction of the active bullets
//
// Three small kernels turn the active mask of a slice of environments into (a) env_off, the
// exclusive prefix sum of the per-environment active counts (n_env + 1 entries), and (b) idx,
// the bullet rows of the slice that are active, in order.  The key/value projection then runs
// over idx only and the attention kernel stages rows [env_off[e], env_off[e+1]).

// one warp per environment: cnt[e] = number of active slots
__global__ void __launch_bounds__(256) k_bullet_count(const uint8_t* __restrict__ active, int n_env, int nb, int* __restrict__ cnt) {
  let_next_start();
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  for (int e = blockIdx.x * 8 + (threadIdx.x >> 5); e < n_env; e += gridDim.x * 8) {
    int c = 0;
    for (int j0 = 0; j0 < nb; j0 += 32) {
      const int j = j0 + lane;
      const bool a = j < nb && active[(size_t)e * nb + j];
      c += __popc(__ballot_sync(0xffffffffu, a));
    }
    if (lane == 0) cnt[e] = c;
  }
}
// one CTA: env_off = exclusive scan of cnt, in place (env_off[n_env] = total).  Eight counts a thread and turn: the barriers of
// a turn are what it takes (8192 environments in one turn instead of eight: step of 8192 x 12 tokens with bullets 870 -> 868 us).
constexpr int SCAN_ITEMS = 8;
__global__ void __launch_bounds__(1024) k_bullet_scan(int* __restrict__ env_off, int n_env) {
  let_next_start();
  wait_for_previous();
  __shared__ int warp_sum[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n_env; base += 1024 * SCAN_ITEMS) {
    const int first = base + (int)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      v[k] = first + k < n_env ? env_off[first + k] : 0;
      sum += v[k];
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    int before = carry + (warp ? warp_sum[warp - 1] : 0) + inc - sum;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      if (first + k < n_env) env_off[first + k] = before;
      before += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = before;
    __syncthreads();
  }
  if (threadIdx.x == 0) env_off[n_env] = carry;
}
// one warp per environment: the active slots of environment e, in order, at idx[env_off[e]...]
__global__ void __launch_bounds__(256) k_bullet_fill(const uint8_t* __restrict__ active, int n_env, int nb,
                                                     const int* __restrict__ env_off, int* __restrict__ idx) {
  let_next_start();
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  for (int e = blockIdx.x * 8 + (threadIdx.x >> 5); e < n_env; e += gridDim.x * 8) {
    int off = env_off[e];
    for (int j0 = 0; j0 < nb; j0 += 32) {
      const int j = j0 + lane;
      const bool a = j < nb && active[(size_t)e * nb + j];
      const uint32_t m = __ballot_sync(0xffffffffu, a);
      if (a) idx[off + __popc(m & ((1u << lane) - 1u))] = e * nb + j;
      off += __popc(m);
    }
  }
}

// The three steps in one CTA for up to 256 environments, eight per warp: three launches (about 2 us each) cost more there
// than the other SMs save.  A step of 16 environments with 80 slots 154.5 -> 146.3 us, of 128 156.7 -> 152.7, equal at
// about 300, slower from there on (512: 174 -> 182).
constexpr int SMALL_ENVS = 256;
__global__ void __launch_bounds__(1024) k_bullet_compact(const uint8_t* __restrict__ active, int n_env, int nb, int* __restrict__ env_off,
                                                         int* __restrict__ idx) {
  let_next_start();
  wait_for_previous();
  __shared__ int off[SMALL_ENVS], warp_sum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = warp; e < n_env; e += 32) {
    int c = 0;
    for (int j0 = 0; j0 < nb; j0 += 32) c += __popc(__ballot_sync(0xffffffffu, j0 + lane < nb && active[(size_t)e * nb + j0 + lane]));
    if (lane == 0) off[e] = c;
  }
  __syncthreads();
  const int v = tid < n_env ? off[tid] : 0;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    warp_sum[lane] = w;
  }
  __syncthreads();
  const int before = (warp ? warp_sum[warp - 1] : 0) + inc - v;
  if (tid < n_env) {
    off[tid] = before;
    env_off[tid] = before;
  }
  if (tid == n_env - 1) env_off[n_env] = before + v;
  __syncthreads();
  for (int e = warp; e < n_env; e += 32) {
    int at = off[e];
    for (int j0 = 0; j0 < nb; j0 += 32) {
      const bool on = j0 + lane < nb && active[(size_t)e * nb + j0 + lane];
      const uint32_t m = __ballot_sync(0xffffffffu, on);
      if (on) idx[at + __popc(m & ((1u << lane) - 1u))] = e * nb + j0 + lane;
      at += __popc(m);
    }
  }
}

// ------------------------------------------------------------------ host side

constexpr int MAX_ENV_TOKENS = 512;  // split-attention path: q, k, v of one head of one environment in shared memory

bool supported(int d_model, int n_heads, int max_tokens_per_env) {
  return d_model == D && n_heads == HEADS && max_tokens_per_env >= 1 && max_tokens_per_env <= MAX_ENV_TOKENS;
}
// Environments that fit one 128-row tile run fully fused; larger ones take the split path.
static bool fits_tile(const BnbBatch& b) { return b.max_tokens_per_env <= TILE; }
bool supported_batch(int d_model, int n_heads, const BnbBatch& b) {
  if (!supported(d_model, n_heads, b.max_tokens_per_env)) return false;
  if (b.tok_off) return fits_tile(b) && b.tile_env_begin != nullptr && b.tile_env_ids != nullptr && b.n_tiles > 0;
  return b.tokens_per_env >= 1;
}

int plan_tiles(const int32_t* tok_off, int n_envs, int32_t* tile_env_begin, int32_t* tile_env_ids, int capacity,
               int* n_tiles) {
  // Best-fit decreasing: environments sorted by size (counting sort, sizes 1..128), each put into
  // the open tile with the least room that still takes it.  Tiles are then listed as ranges of
  // tile_env_ids.  Near-full tiles matter: a tile costs about the same whatever its fill.
  // Flat arrays throughout (16 384 environments: about 0.1 ms; with a vector per tile and per room
  // it was 0.7 ms of a step's host time): open tiles of one room form a stack linked through
  // next_open, a 129-bit mask says which rooms have any, the environments of a tile a chain.
  if (capacity < n_envs + 1) return BNB_ERR_SCRATCH_TOO_SMALL;
  int begin[TILE + 2] = {};
  for (int e = 0; e < n_envs; ++e) {
    const int n = tok_off[e + 1] - tok_off[e];
    if (n <= 0 || n > TILE) return BNB_ERR_TOO_MANY_TOKENS;
    ++begin[TILE - n + 1];   // largest first
  }
  for (int i = 1; i <= TILE; ++i) begin[i] += begin[i - 1];
  std::vector<int> store((size_t)n_envs * 6);
  int* order = store.data();
  int* next_env = order + n_envs;      // next environment of the same tile
  int* first_env = next_env + n_envs;  // per tile
  int* last_env = first_env + n_envs;
  int* next_open = last_env + n_envs;
  for (int e = 0; e < n_envs; ++e) order[begin[TILE - (tok_off[e + 1] - tok_off[e])]++] = e;
  int open[TILE + 1];
  for (int& o : open) o = -1;
  uint64_t mask[3] = {0, 0, 0};
  int tiles = 0;
  for (int i = 0; i < n_envs; ++i) {
    const int e = order[i], n = tok_off[e + 1] - tok_off[e];
    int room = -1;
    for (int w = n >> 6; w < 3; ++w) {
      const uint64_t m = w == n >> 6 ? mask[w] >> (n & 63) << (n & 63) : mask[w];
      if (m) { room = w * 64 + __builtin_ctzll(m); break; }
    }
    int t;
    if (room < 0) {
      t = tiles++;
      room = TILE;
      first_env[t] = e;
    } else {
      t = open[room];
      open[room] = next_open[t];
      if (open[room] < 0) mask[room >> 6] &= ~(1ull << (room & 63));
      next_env[last_env[t]] = e;
    }
    last_env[t] = e;
    next_env[e] = -1;
    const int left = room - n;
    next_open[t] = open[left];
    open[left] = t;
    mask[left >> 6] |= 1ull << (left & 63);
  }
  int k = 0;
  for (int t = 0; t < tiles; ++t) {
    tile_env_begin[t] = k;
    for (int e = first_env[t]; e >= 0; e = next_env[e]) tile_env_ids[k++] = e;
  }
  tile_env_begin[tiles] = k;
  *n_tiles = tiles;
  return BNB_OK;
}

static size_t round256(size_t v) { return (v + 255) / 256 * 256; }
// Shared memory of the attention kernel for environments of up to max_tokens tokens and nb bullets.
static size_t flash_smem(int max_tokens, int nb, int hpc) {
  // staged q, k, v (and bullet k, v) rows, then one bias float per key, each set padded to 32 keys
  return (size_t)(3 * max_tokens + 2 * nb) * flash_stride(hpc) + 4 * (size_t)(((max_tokens + 31) & ~31) + ((nb + 31) & ~31)) + 16;
}
constexpr size_t FLASH_SMEM_MAX = 227 * 1024;
// Bullet rows staged at a time: 32 where every warp (there are four at least) has one (head, query block) pair, so that registers and not
// shared memory bound the CTAs of an SM (six).  Whole blocks of 32 keys, or the stage would decide which keys share a block.
static int flash_stage(int max_tokens, int nb, int hpc) { return hpc * ((max_tokens + 15) / 16) <= 4 && nb > 32 ? 32 : nb; }
// All four heads in one CTA while that leaves room for three CTAs per SM, else one head per CTA.
static int flash_heads_per_cta(int max_tokens, int nb) {
  return flash_smem(max_tokens, flash_stage(max_tokens, nb, HEADS), HEADS) <= 72 * 1024 ? HEADS : 1;
}
bool supported_bullets(const BnbBatch& b, int bullets_per_env) {
  return bullets_per_env >= 1 && flash_smem(b.max_tokens_per_env, bullets_per_env, 1) <= FLASH_SMEM_MAX;
}

// Layout: status area | q|k|v and attention output of every row (split path: environments larger
// than a tile, or any sublayer reading bullets) | bullet keys and values of one slice of environments.
size_t scratch_bytes(int, const BnbBatch& b, int T, int bullets_per_env) {
  size_t bytes = 65536;  // status word (and cycle accounting)
  if (!fits_tile(b) || bullets_per_env > 0)
    bytes += round256((size_t)T * b.total_tokens * 4 * D * sizeof(__nv_bfloat16));
  bytes += round256(bullet_slice_bytes((long long)T * b.n_envs, bullets_per_env, D, sizeof(__nv_bfloat16)));
  if (bullets_per_env > 0) {
    // env_off (slice environments + 1) and idx (one int per bullet row of a slice)
    const size_t envs = (size_t)bullet_slice_envs((long long)T * b.n_envs, bullets_per_env, D, sizeof(__nv_bfloat16));
    bytes += round256((envs + 1) * sizeof(int)) + round256(envs * bullets_per_env * sizeof(int));
  }
  return bytes;
}
size_t packed_spatial_bytes(int d_model) { return d_model == D ? (size_t)N_SPATIAL_IMAGE * CHUNK_BYTES : 0; }
size_t packed_temporal_bytes(int d_model) { return d_model == D ? (size_t)N_TEMPORAL_CHUNKS * CHUNK_BYTES + 2048 : 0; }

int pack_spatial(const BnbSpatialWeights& w, int d_model, int n_heads, void* packed, cudaStream_t st) {
  if (d_model != D || n_heads != HEADS) return BNB_ERR_UNSUPPORTED_DIMS;
  count_launch();
  k_pack_spatial<<<148, 256, 0, st>>>(w, static_cast<uint8_t*>(packed));
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH;
}
int pack_temporal(const BnbTemporalWeights& w, int d_model, void* packed, cudaStream_t st) {
  if (d_model != D) return BNB_ERR_UNSUPPORTED_DIMS;
  count_launch();
  k_pack_temporal<<<148, 256, 0, st>>>(w, static_cast<uint8_t*>(packed));
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH;
}

int pack_trunk(const BnbSpatialWeights* spatial, int n_spatial, const BnbTemporalWeights* temporal, int n_temporal,
               int d_model, int n_heads, cudaStream_t st, int* status) {
  if (d_model != D || n_heads != HEADS) return BNB_ERR_UNSUPPORTED_DIMS;
  // as many launches as it takes at MAX_PACK_JOBS sublayers of each kind per launch (one for the
  // trunks of the shipped profiles)
  for (int s0 = 0, t0 = 0; s0 < n_spatial || t0 < n_temporal;) {
    PackJobs jobs{};
    jobs.status = status;
    for (; s0 < n_spatial && jobs.n_spatial < MAX_PACK_JOBS; ++s0) {
      if (!spatial[s0].packed) return BNB_ERR_NULL_POINTER;
      jobs.sw[jobs.n_spatial++] = spatial[s0];
    }
    for (; t0 < n_temporal && jobs.n_temporal < MAX_PACK_JOBS; ++t0) {
      if (!temporal[t0].packed) return BNB_ERR_NULL_POINTER;
      jobs.tw[jobs.n_temporal++] = temporal[t0];
    }
    if (const int rc = launch_after(k_pack_trunk, dim3(PACK_BLOCKS, jobs.n_spatial + jobs.n_temporal), 256, 0, st, jobs)) return rc;
  }
  return BNB_OK;
}

// ------------------------------------------------------------------ status word on the host
//
// The bounded waits record a code in the status word at the head of the scratch buffer, and the wait
// that runs out writes the same code straight to a pinned, device-mapped host word of its device, so
// that a call that goes well costs no copy (a 4-byte download per call took 3.4 us of the stream);
// whoever asks later -- the next call, or bnb_last_status -- finds a non-zero code there and keeps it
// until it is cleared.
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_status_mutex;
int* g_host_status[kMaxDevices] = {};
int g_sticky_status[kMaxDevices] = {};

void latch_status(int dev) {
  if (g_host_status[dev]) {
    const int v = *static_cast<volatile int*>(g_host_status[dev]);
    if (v != 0 && g_sticky_status[dev] == 0) g_sticky_status[dev] = v;
  }
}
}  // namespace

// Device address of the host word of the current device, allocating it on the first call (null
// during a stream capture without it: that capture's launches then report to their scratch only).
int* host_status_word(cudaStream_t st) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  if (!g_host_status[dev]) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return nullptr;
    void* p = nullptr;
    if (cudaHostAlloc(&p, 64, cudaHostAllocMapped) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    g_host_status[dev] = static_cast<int*>(p);
    *g_host_status[dev] = 0;
  }
  latch_status(dev);
  return g_host_status[dev];   // one address space: the host address is the device's too
}
int last_status() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  latch_status(dev);
  return g_sticky_status[dev];
}
void clear_status() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  g_sticky_status[dev] = 0;
  if (g_host_status[dev]) *g_host_status[dev] = 0;
}
void debug_wait_test(int skip_op, int poll_limit) {
  g_debug_skip_op = skip_op;
  g_debug_poll_limit = poll_limit;
}

// Tiles that the environments of a batch fill at one timestep, as many environments to a tile as fit.
static long long full_tiles(const BnbBatch& b, bool flat) {
  if (flat) return (b.total_tokens + TILE - 1) / TILE;
  if (b.tok_off) return b.n_tiles;
  const int per = TILE / b.tokens_per_env;
  return (b.n_envs + per - 1) / per;
}
// Timesteps per tile of a temporal sublayer over T timesteps, or 0 for a walk over tiles of one timestep: the fewest passes over
// the busiest SM.  A pass takes 21.9 us in the walk and 21.4 in chunks at 2368 environments of 8 tokens, 22.2 and 21.6 at 16384, so
// passes are what is compared; at as many of them, chunks (the walk: 8 % faster to 4 % slower).  What stays with the walk: a batch
// that fills the chip, for step counts that would leave much of the last chunk empty -- 2368 environments: 5 steps 542 against 684
// us in chunks of 4, 9 steps 927 against 1 066; 8192 environments of 12 tokens: 3 steps 1 714 against 1 890.  Chunks with
// the same number of passes lie within 2 % of each other; the smallest is taken.
static int steps_per_tile(const BnbBatch& b, bool flat, int T) {
  const auto rounds = [](long long tiles) { return (tiles + 147) / 148; };
  const long long walk = rounds(full_tiles(b, flat)) * T;
  long long best = walk + 1;
  int chunk = 0;
  for (int c = 4; c <= 32; c *= 2) {
    const long long passes = rounds(((long long)b.total_tokens * c + TILE - 1) / TILE) * ((T + c - 1) / c);
    if (passes < best) {
      best = passes;
      chunk = c;
    }
  }
  return chunk;
}

static int launch(TrunkArgs& a, const BnbBatch& b, cudaStream_t st) {
  a.map = make_env_map(b);
  if (a.chunk) {
    a.tile_env_begin = nullptr;
    a.flat_rows = 0;
    a.envs_per_tile = 0;
    a.env_tiles = (int)(((long long)b.total_tokens * a.chunk + TILE - 1) / TILE);
  } else if (a.flat_rows) {
    a.tile_env_begin = nullptr;
    a.envs_per_tile = 0;
    a.env_tiles = (b.total_tokens + TILE - 1) / TILE;
  } else if (b.tok_off) {
    a.tile_env_begin = b.tile_env_begin;
    a.tile_env_ids = b.tile_env_ids;
    a.envs_per_tile = 0;
    a.env_tiles = b.n_tiles;
  } else {
    a.tile_env_begin = nullptr;
    // Full tiles decide how many rounds over the SMs the launch takes; within that number the
    // environments are spread out: a tile's attention and recurrence cost what its environments cost
    // (16 environments of 12 tokens: 115 us as two tiles, 96 us as sixteen).
    const int full = TILE / b.tokens_per_env;
    const auto tiles = [&](int per) { return (long long)((b.n_envs + per - 1) / per) * a.n_groups; };
    const long long slots = (tiles(full) + 147) / 148 * 148;
    a.envs_per_tile = full;
    while (a.envs_per_tile > 1 && tiles(a.envs_per_tile - 1) <= slots) --a.envs_per_tile;
    a.env_tiles = (b.n_envs + a.envs_per_tile - 1) / a.envs_per_tile;
  }
  a.n_tiles = a.env_tiles * a.n_groups;
  a.has_fields = b.total_tokens > b.total_ships ? 1 : 0;
  a.poll_limit = g_debug_poll_limit;
  a.skip_op = g_debug_skip_op;
  a.host_status = host_status_word(st);
  uintptr_t places = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.y);
  for (int i = 0; i < a.n_sub; ++i)
    places |= reinterpret_cast<uintptr_t>(a.sub[i].hid_in) | reinterpret_cast<uintptr_t>(a.sub[i].hid_out) |
              reinterpret_cast<uintptr_t>(a.sub[i].qkv_out) | reinterpret_cast<uintptr_t>(a.sub[i].o_in);
  a.wide = places % 32 == 0;
  if (a.n_tiles == 0) return BNB_OK;
  return launch_pipelined(a, st);
}

static int prepare_status(void* scratch, size_t scratch_bytes, cudaStream_t st, bool clear, int** status) {
  if (!scratch) return BNB_ERR_NULL_POINTER;
  if (scratch_bytes < 65536) return BNB_ERR_SCRATCH_TOO_SMALL;
  *status = static_cast<int*>(scratch);
  if (clear && cudaMemsetAsync(scratch, 0, 256, st) != cudaSuccess) return BNB_ERR_LAUNCH;
  return BNB_OK;
}

static void fill_spatial(SubLayer& s, const BnbSpatialWeights& w) {
  s = SubLayer{};
  s.type = SUB_SPATIAL;
  s.packed = static_cast<const uint8_t*>(w.packed);
}
static void fill_temporal(SubLayer& s, const BnbTemporalWeights& w, const float* hin, float* hout) {
  s = SubLayer{};
  s.type = SUB_TEMPORAL;
  s.packed = static_cast<const uint8_t*>(w.packed);
  s.conv_w = w.conv_w;
  s.conv_b = w.conv_b;
  s.decay_log2 = reinterpret_cast<const float*>(static_cast<const uint8_t*>(w.packed) + (size_t)N_TEMPORAL_CHUNKS * CHUNK_BYTES);
  s.hid_in = hin;
  s.hid_out = hout;
}

// Attention of the environments [env_base, env_base + n_env) (group-major), with the bullet keys
// of the same environments in kvb when nb > 0.
static int launch_attention(const __nv_bfloat16* qkv, const uint8_t* alive, __nv_bfloat16* o, const BnbBatch& b,
                            int env_base, int n_env, const __nv_bfloat16* kvb, const int* env_off, int nb,
                            cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BNB_ERR_NO_DEVICE;
  if (!configured[dev]) {
    for (auto kernel : {k_attention_flash<HEADS, true>, k_attention_flash<1, true>, k_attention_flash<HEADS, false>, k_attention_flash<1, false>})
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FLASH_SMEM_MAX) != cudaSuccess) return BNB_ERR_LAUNCH;
    configured[dev] = true;
  }
  if (n_env <= 0) return BNB_OK;
  const int hpc = flash_heads_per_cta(b.max_tokens_per_env, kvb ? nb : 0);
  const int stage = flash_stage(b.max_tokens_per_env, kvb ? nb : 0, hpc);
  size_t smem = flash_smem(b.max_tokens_per_env, stage, hpc);
  if (smem > FLASH_SMEM_MAX) return BNB_ERR_TOO_MANY_TOKENS;
  dim3 grid(n_env, HEADS / hpc);
  // The launch before leaves the SMs one after the other, and the first to be free takes as many CTAs as fit.  Up to four a SM, shared
  // memory is asked for so that no SM takes more than its share (228 KB a SM, 1 KB of it for each CTA).  A step of 43 environments of 96
  // tokens with 160 slots (172 CTAs) 156.7 -> 150.1 us, 100 of them 169.5 -> 166.8, 43 of 114 tokens 173.5 -> 165.7; 300 have more than four.
  const long long per_sm = ((long long)n_env * (HEADS / hpc) + 147) / 148;
  if (per_sm <= 4) smem = std::max(smem, (size_t)228 * 1024 / (size_t)(per_sm + 1) - 512);
  // warps per CTA: the fewest idle warp-rounds over the (head, query block) pairs of a full environment
  const int items = hpc * ((b.max_tokens_per_env + 15) / 16);
  int n_warps = 4, best_idle = 1 << 30;
  for (int w = 4; w <= 8; ++w) {
    const int idle = (items + w - 1) / w * w - items;
    if (idle < best_idle) { best_idle = idle; n_warps = w; }
  }
  const auto kernel = kvb ? (hpc == HEADS ? k_attention_flash<HEADS, true> : k_attention_flash<1, true>)
                          : (hpc == HEADS ? k_attention_flash<HEADS, false> : k_attention_flash<1, false>);
  return launch_after(kernel, grid, 32 * n_warps, smem, st, qkv, alive, o, make_env_map(b), env_base, stage,
                      kvb, env_off, nb);
}

// env_off / idx of the active bullets of n_env environments (see the compaction kernels).
int compact_active(const uint8_t* active, int n_env, int nb, int* env_off, int* idx, cudaStream_t st) {
  if (n_env <= 0) return BNB_OK;
  if (n_env <= SMALL_ENVS) return launch_after(k_bullet_compact, dim3(1), 1024, 0, st, active, n_env, nb, env_off, idx);
  const int blocks = (n_env + 7) / 8 < 148 * 8 ? (n_env + 7) / 8 : 148 * 8;
  if (const int rc = launch_after(k_bullet_count, dim3(blocks), 256, 0, st, active, n_env, nb, env_off)) return rc;
  if (const int rc = launch_after(k_bullet_scan, dim3(1), 1024, 0, st, env_off, n_env)) return rc;
  return launch_after(k_bullet_fill, dim3(blocks), 256, 0, st, active, n_env, nb, env_off, idx);
}

// Accumulates sublayers into tile-kernel launches.  In split mode (environments larger than
// one tile) a spatial sublayer becomes PRE | attention kernel | POST, and the tile kernel
// walks plain 128-row slices.  A sublayer that reads bullets takes the same three-part form
// whatever the environment size, with the bullet key/value projection and the attention kernel
// run once per slice of environments.
struct Plan {
  const BnbBatch& b;
  cudaStream_t st;
  int* status;
  bool split;
  const uint8_t* alive;
  const uint8_t* done;
  const uint8_t* reset_env;
  const float* cur;      // where the residual stream currently lives
  float* y;
  const BnbBullets* bullets;
  __nv_bfloat16* qkv;
  __nv_bfloat16* o;
  __nv_bfloat16* kvb;    // bullet keys and values of one slice
  int kvb_envs;          // environments per slice
  int* env_off;          // compaction of the slice's active bullets (see compact_active)
  int* idx;
  int compacted_e0;      // first environment of the slice env_off / idx currently describe, -1 = none
  bool io_bf16 = false;  // x and y (and so the stream between launches) hold bfloat16
  int n_groups, t_loop;  // geometry of the pending program
  TrunkArgs a;
  int n;

  void begin(int groups, int tl) {
    a = TrunkArgs{};
    n = 0;
    n_groups = groups;
    t_loop = tl;
  }
  int flush() {
    if (n == 0) return BNB_OK;
    a.status = status;
    a.alive = split ? nullptr : alive;
    a.done = done;
    a.reset_env = reset_env;
    a.n_groups = n_groups;
    a.t_loop = t_loop;
    a.chunk = 0;
    a.steps = t_loop;
    if (t_loop > 1) {
      a.chunk = steps_per_tile(b, split, t_loop);
      if (a.chunk) a.t_loop = (t_loop + a.chunk - 1) / a.chunk;
    }
    a.n_sub = n;
    a.flat_rows = split ? 1 : 0;
    a.io_bf16 = io_bf16 ? 1 : 0;
    a.x = cur;
    a.y = y;
    int rc = launch(a, b, st);
    cur = y;
    const int g = n_groups, tl = t_loop;
    begin(g, tl);
    return rc;
  }
  int ensure(int groups, int tl) {
    if (n > 0 && (groups != n_groups || tl != t_loop)) {
      int rc = flush();
      if (rc) return rc;
    }
    n_groups = groups;
    t_loop = tl;
    return BNB_OK;
  }
  int add_spatial(const BnbSpatialWeights& w, int groups) {
    int rc = ensure(groups, 1);
    if (rc) return rc;
    if (n == MAX_SUBLAYERS && (rc = flush())) return rc;
    const bool reads = bullets && w.kv_bullet_w;
    fill_spatial(a.sub[n], w);
    if (!split && !reads) { ++n; return BNB_OK; }
    a.sub[n].type = SUB_SPATIAL_PRE;
    a.sub[n].qkv_out = qkv;
    ++n;
    if ((rc = flush())) return rc;
    const int total_envs = groups * b.n_envs;
    if (reads) {
      const int nb = bullets->per_env;
      for (int e0 = 0; e0 < total_envs; e0 += kvb_envs) {
        const int ne = total_envs - e0 < kvb_envs ? total_envs - e0 : kvb_envs;
        const bool masked = bullets->active != nullptr;
        if (masked && compacted_e0 != e0) {
          // the mask is the same for every reading sublayer of the call: one slice -> compact once
          if ((rc = compact_active(bullets->active + (size_t)e0 * nb, ne, nb, env_off, idx, st))) return rc;
          compacted_e0 = e0;
        }
        const bool rows_bf16 = bullets->tokens_bf16 != 0;
        const uint8_t* rows = reinterpret_cast<const uint8_t*>(bullets->tokens) + (size_t)e0 * nb * D * (rows_bf16 ? 2 : 4);
        const uint8_t* image = static_cast<const uint8_t*>(w.packed) + (size_t)N_SPATIAL_CHUNKS * CHUNK_BYTES;
        if ((rc = bullet_kv(rows, rows_bf16, ne * nb, masked ? idx : nullptr, masked ? env_off + ne : nullptr, image, kvb, status, st)))
          return rc;
        if ((rc = launch_attention(qkv, alive, o, b, e0, ne, kvb, masked ? env_off : nullptr, nb, st))) return rc;
      }
    } else if ((rc = launch_attention(qkv, alive, o, b, 0, total_envs, nullptr, nullptr, 0, st))) {
      return rc;
    }
    fill_spatial(a.sub[n], w);
    a.sub[n].type = SUB_SPATIAL_POST;
    a.sub[n].o_in = o;
    ++n;
    return BNB_OK;
  }
  int add_temporal(const BnbTemporalWeights& w, const float* hin, float* hout, int tl) {
    int rc = ensure(tl > 1 ? 1 : n_groups, tl);
    if (rc) return rc;
    if (tl > 1 && n > 0 && (rc = flush())) return rc;   // a time walk runs alone
    if (n == MAX_SUBLAYERS && (rc = flush())) return rc;
    fill_temporal(a.sub[n++], w, hin, hout);
    if (tl > 1) return flush();
    return BNB_OK;
  }
};

static int make_plan(Plan& p, void* scratch, size_t scratch_bytes, int T, bool clear_status = true) {
  int rc = prepare_status(scratch, scratch_bytes, p.st, clear_status, &p.status);
  if (rc) return rc;
  p.split = !fits_tile(p.b);
  p.qkv = nullptr;
  p.o = nullptr;
  p.kvb = nullptr;
  p.kvb_envs = 0;
  const int nb = p.bullets ? p.bullets->per_env : 0;
  if (nb > 0 && !supported_bullets(p.b, nb)) return BNB_ERR_UNSUPPORTED_DIMS;
  if (scratch_bytes < tensor::scratch_bytes(D, p.b, T, nb)) return BNB_ERR_SCRATCH_TOO_SMALL;
  uint8_t* base = static_cast<uint8_t*>(scratch) + 65536;
  if (p.split || nb > 0) {
    const size_t rows = (size_t)T * p.b.total_tokens;
    p.qkv = reinterpret_cast<__nv_bfloat16*>(base);
    p.o = p.qkv + rows * 3 * D;
    base += round256(rows * 4 * D * sizeof(__nv_bfloat16));
  }
  p.env_off = nullptr;
  p.idx = nullptr;
  p.compacted_e0 = -1;
  if (nb > 0) {
    p.kvb = reinterpret_cast<__nv_bfloat16*>(base);
    p.kvb_envs = bullet_slice_envs((long long)T * p.b.n_envs, nb, D, sizeof(__nv_bfloat16));
    base += round256(bullet_slice_bytes((long long)T * p.b.n_envs, nb, D, sizeof(__nv_bfloat16)));
    p.env_off = reinterpret_cast<int*>(base);
    base += round256(((size_t)p.kvb_envs + 1) * sizeof(int));
    p.idx = reinterpret_cast<int*>(base);
  }
  p.begin(1, 1);
  return BNB_OK;
}

int spatial_block(const BnbSpatialWeights& w, int d_model, int n_heads, const float* x, const uint8_t* alive,
                  const BnbBullets* bullets, float* y, const BnbBatch& b, int n_groups, void* scratch,
                  size_t scratch_bytes, cudaStream_t st) {
  if (!supported_batch(d_model, n_heads, b) || !w.packed) return BNB_ERR_UNSUPPORTED_DIMS;
  Plan p{b, st, nullptr, false, alive, nullptr, nullptr, x, y, bullets};
  int rc = make_plan(p, scratch, scratch_bytes, n_groups);
  if (rc) return rc;
  if ((rc = p.add_spatial(w, n_groups))) return rc;
  return p.flush();
}

int temporal_block(const BnbTemporalWeights& w, int d_model, const float* x, float* y, const float* hidden_in,
                   float* hidden_out, const uint8_t* done, const uint8_t* reset_env, const BnbBatch& b, int T,
                   void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (!supported_batch(d_model, HEADS, b) || !w.packed) return BNB_ERR_UNSUPPORTED_DIMS;
  Plan p{b, st, nullptr, false, nullptr, done, reset_env, x, y, nullptr};
  int rc = make_plan(p, scratch, scratch_bytes, T);
  if (rc) return rc;
  if ((rc = p.add_temporal(w, hidden_in, hidden_out, T))) return rc;
  return p.flush();
}

int trunk(const BnbSpatialWeights* spatial, const BnbTemporalWeights* temporal, int n_blocks, int n_spatial,
          int n_temporal, int d_model, int n_heads, const float* x, const uint8_t* alive, const BnbBullets* bullets,
          float* y, const float* hidden_in, float* hidden_out, const uint8_t* done, const uint8_t* reset_env,
          const BnbBatch& b, int T, void* scratch, size_t scratch_bytes, cudaStream_t st, bool io_bf16, bool pack_images) {
  if (!supported_batch(d_model, n_heads, b)) return BNB_ERR_UNSUPPORTED_DIMS;
  // bfloat16 x / y: every tile-kernel launch of the call reads and writes bfloat16 rows, so the
  // residual stream is rounded where one launch hands over to the next (the reference, given
  // bfloat16 tokens, rounds it after every sublayer)
  for (int i = 0; i < n_blocks * n_spatial; ++i) if (!spatial[i].packed) return BNB_ERR_UNSUPPORTED_DIMS;
  for (int i = 0; i < n_blocks * n_temporal; ++i) if (!temporal[i].packed) return BNB_ERR_UNSUPPORTED_DIMS;
  // a time walk carries its state through hidden_out between timesteps
  if (T > 1 && n_blocks * n_temporal > 0 && b.total_ships > 0 && !hidden_out) return BNB_ERR_NULL_POINTER;
  Plan p{b, st, nullptr, false, alive, done, reset_env, x, y, bullets};
  p.io_bf16 = io_bf16;
  const bool pack = pack_images && n_blocks * (n_spatial + n_temporal) > 0;
  int rc = make_plan(p, scratch, scratch_bytes, T, !pack);
  if (rc) return rc;
  if (pack && (rc = pack_trunk(spatial, n_blocks * n_spatial, temporal, n_blocks * n_temporal, d_model, n_heads, st, p.status))) return rc;
  const size_t slot_stride = (size_t)b.total_ships * 4 * D;
  for (int i = 0; i < n_blocks; ++i) {
    for (int j = 0; j < n_spatial; ++j)
      if ((rc = p.add_spatial(spatial[i * n_spatial + j], T))) return rc;
    for (int j = 0; j < n_temporal; ++j) {
      const int slot = i * n_temporal + j;
      if ((rc = p.add_temporal(temporal[slot], hidden_in ? hidden_in + slot * slot_stride : nullptr,
                               hidden_out ? hidden_out + slot * slot_stride : nullptr, T))) return rc;
    }
  }
  if ((rc = p.flush())) return rc;
  if (p.cur == x && y != x) {
    if (cudaMemcpyAsync(y, x, (size_t)T * b.total_tokens * D * (io_bf16 ? 2 : sizeof(float)), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
      return BNB_ERR_LAUNCH;
  }
  return BNB_OK;
}

}  // namespace tensor
}  // namespace bnb
