// Attention of the training path for environments of up to 32 tokens, float32, four heads of 32.
//
// One CTA per environment-step, one warp per head, every row staged once in shared memory with 16-byte
// asynchronous copies and written back as whole rows.  Its floor is the memory traffic of q|k|v (1.5 KB per
// token) and its gradient; what bounds it is shared-memory and load latency: 8192 environment-steps of 8
// tokens take 38 us forward (DRAM 36 % of peak, issue slots 53 % busy, 57 % of the warps) and 67 us for the gradient
// (64 registers without bullets hold 47 % of the warps, where 128 held 24 % and it took 95).  The kernels it replaces read rows element by element (one
// thread per query, or eight lanes per head), ran at 2.2 - 2.6 TB/s on environments of 8 tokens and took 425 /
// 575 us (forward / gradient) for 1536 environment-steps of 12 tokens with 80 bullet slots, most of it
// on slots that are not in use (39 / 73 us here, averaged over the sublayers that read them and those that do not).  Here only the slots in use are read.
//
// Gradient contract: probabilities recomputed as exp(s - lse) with lse = max + log(sum) in float32, row
// term <d out, out>, as the fused attention kernels behind F.scaled_dot_product_attention
// (models/yemong/attention.py:131-166).
#include "train_attention.h"

#include "common.cuh"
#include "launch_after.h"
#include "tensor_common.cuh"

namespace bnb {
namespace train_attn {

namespace {

constexpr int D = 128, H = 4, DH = 32, THREADS = 32 * H;
// row strides in floats, 4 mod 32: sixteen-byte reads of eight consecutive rows hit every bank once
constexpr int LDQ = 3 * D + 4, LDO = D + 4, LDB = 2 * D + 4;
constexpr int BLOCK = 32;    // bullet keys staged at a time
constexpr float SCALE = 0.17677669529663687f;   // 1 / sqrt(32)

__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}
// `rows` rows of W floats between global memory (dense) and shared memory (stride ld)
template <int W>
__device__ __forceinline__ void rows_in(float* dst, int ld, const float* src, int rows) {
  for (int i = threadIdx.x; i < rows * (W / 4); i += THREADS) copy16(dst + (i / (W / 4)) * ld + (i % (W / 4)) * 4, src + (size_t)i * 4);
}
// The q-th (mod PARTS * 32) four columns of a row of PARTS parts of D columns.
template <int PARTS>
__device__ __forceinline__ float4* parts_at(float* base, int ld, size_t off, size_t row, int q) {
  q %= PARTS * (D / 4);
  return reinterpret_cast<float4*>(base + row * ld + (q / (D / 4)) * off) + q % (D / 4);
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float s) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s)))); }
// One chain: its order is part of the results (in four chains they differ by 1e-7, and by 1e-3 behind the bfloat16 products that
// follow), and four took no less time, with 40 and 176 bytes spilled in the gradient for 16 tokens and for 32 with bullets (0 and 124).
__device__ __forceinline__ float dot32(const float* a, const float* b) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < DH / 4; ++i) s = dot4(ld4(a + 4 * i), ld4(b + 4 * i), s);
  return s;
}
__device__ __forceinline__ void load32(float* to, const float* from) {
#pragma unroll
  for (int i = 0; i < DH / 4; ++i) *reinterpret_cast<float4*>(to + 4 * i) = ld4(from + 4 * i);
}
template <int W>
__device__ __forceinline__ float seg_sum(float v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int W>
__device__ __forceinline__ float seg_max(float v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The bullet slots that are keys, in order (every thread calls; list and count in shared memory).
__device__ __forceinline__ int key_list(const uint8_t* active, int nb, uint16_t* list, int* count) {
  if (threadIdx.x < 32) {
    int n = 0;
    for (int j0 = 0; j0 < nb; j0 += 32) {
      const int j = j0 + threadIdx.x;
      const bool on = j < nb && (!active || active[j]);
      const uint32_t m = __ballot_sync(0xffffffffu, on);
      if (on) list[n + __popc(m & ((1u << threadIdx.x) - 1u))] = (uint16_t)j;
      n += __popc(m);
    }
    if (threadIdx.x == 0) *count = n;
  }
  __syncthreads();
  return *count;
}
// Where the k-th key of group g has its row: the first of its rows, or those of its list.
struct KeyRows {
  size_t first;
  const uint16_t* list;   // null: one behind the other
  __device__ __forceinline__ size_t operator()(int k) const { return first + (list ? list[k] : k); }
};
__device__ __forceinline__ KeyRows key_rows(const Call& c, size_t g, uint16_t* list, int* count, int* keys) {
  if (c.boff) {
    const int first = c.boff[g];
    *keys = c.boff[g + 1] - first;
    return {(size_t)first, nullptr};
  }
  *keys = key_list(c.bactive ? c.bactive + g * c.nb : nullptr, c.nb, list, count);
  return {g * c.nb, list};
}
__device__ __forceinline__ void stage_keys(float* kv, const float* kvb, const KeyRows& row, int k0, int n) {
  for (int i = threadIdx.x; i < n * (2 * D / 4); i += THREADS) {
    const int r = i / (2 * D / 4), q = i % (2 * D / 4);
    copy16(kv + r * LDB + q * 4, kvb + row(k0 + r) * 2 * D + q * 4);
  }
  copies_done();
}

struct Smem {
  float *rows, *d_o, *dq, *kv, *acc, *m, *l, *s;
  uint16_t* list;
  int* count;
};
__host__ __device__ inline size_t carve(char* base, int n, int nb, bool grad, Smem* out) {
  size_t off = 0;
  auto take = [&](size_t floats) { float* p = reinterpret_cast<float*>(base + off); off += (floats * 4 + 15) / 16 * 16; return p; };
  Smem s{};
  s.rows = take((size_t)n * LDQ);
  if (grad) s.d_o = take((size_t)n * LDO);
  if (nb > 0) {
    if (grad) s.dq = take((size_t)n * LDO);
    else s.acc = take((size_t)2 * n * D);      // self output, bullet output
    s.kv = take((size_t)BLOCK * LDB);
    s.m = take((size_t)n * H);
    s.l = take((size_t)n * H);
    if (grad) s.s = take((size_t)n * H);
    s.list = reinterpret_cast<uint16_t*>(take((size_t)(nb + 1) / 2));
    s.count = reinterpret_cast<int*>(take(4));
  }
  if (out) *out = s;
  return off;
}

// LPP lanes per query (8, 16 or 32: the smallest that holds the keys), so a warp serves 32 / LPP queries
// of its head at once; lane `sub` scores key `sub`, then owns CPL channels of the output.
template <int LPP, bool BULLETS>
__global__ void __launch_bounds__(THREADS) k_env_attn_fwd(const Call c) {
  extern __shared__ __align__(16) char raw[];
  tensor::let_next_start();
  tensor::wait_for_previous();
  constexpr int QPW = 32 / LPP, CPL = DH / LPP;
  Smem s;
  carve(raw, c.n, BULLETS ? c.nb : 0, false, &s);
  const int h = threadIdx.x >> 5, lane = threadIdx.x & 31, qs = lane / LPP, sub = lane % LPP;
  const int n = c.n;
  const size_t g = blockIdx.x, tok0 = g * n;
  rows_in<3 * D>(s.rows, LDQ, c.qkv + tok0 * 3 * D, n);
  int keys = 0;
  KeyRows row{};
  if constexpr (BULLETS) {
    row = key_rows(c, g, s.list, s.count, &keys);
    for (int i = threadIdx.x; i < n * H; i += THREADS) { s.m[i] = -INFINITY; s.l[i] = 0.f; }
    for (int i = threadIdx.x; i < n * D; i += THREADS) s.acc[n * D + i] = 0.f;
  }
  copies_done();
  const float* q = s.rows + h * DH;
  const float* k = q + D;
  const float* v = q + 2 * D;
  const bool key = sub < n;
  const bool dead = key && c.alive && !c.alive[tok0 + sub];
  // More than 16 tokens: a warp takes one query at a time and a lane one key for all of them, in registers.  1184 environment-steps of 20 tokens
  // 54 -> 45 us, 1280 of 32 106 -> 89; with bullets the same below, 80 for 20 tokens 282 -> 239, 40 for 32 604 -> 511.  (Read from shared memory for
  // each query the instances with and without bullets were slower than the one kernel for both had been: 51, 100, 260 and 531.)
  constexpr bool ONE = LPP == 32;
  float own[ONE ? DH : 1];
  if constexpr (ONE) load32(own, k + min(sub, n - 1) * LDQ);
  for (int q0 = 0; q0 < n; q0 += QPW) {
    const int i = q0 + qs, ic = min(i, n - 1);
    float sc = -INFINITY;
    if (key) sc = dead ? kMaskedScore : dot32(q + ic * LDQ, ONE ? own : k + sub * LDQ) * SCALE;
    const float mx = seg_max<LPP>(sc);
    const float e = key ? expf(sc - mx) : 0.f;
    const float p = e / seg_sum<LPP>(e);
    float acc[CPL];
#pragma unroll
    for (int j = 0; j < CPL; ++j) acc[j] = 0.f;
    for (int j = 0; j < n; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, qs * LPP + j);
      const float* vj = v + j * LDQ + sub * CPL;
#pragma unroll
      for (int d = 0; d < CPL; ++d) acc[d] = fmaf(pj, vj[d], acc[d]);
    }
    if (i < n) {
      float* out = keys ? s.acc + i * D + h * DH + sub * CPL : c.o + (tok0 + i) * D + h * DH + sub * CPL;
#pragma unroll
      for (int d = 0; d < CPL; ++d) out[d] = acc[d];
    }
  }
  if constexpr (!BULLETS) return;
  if (keys == 0) return;   // no bullet in use: the branch is gated off
  for (int k0 = 0; k0 < keys; k0 += BLOCK) {
    const int kn = min(BLOCK, keys - k0);
    __syncthreads();       // the previous block has been read
    stage_keys(s.kv, c.kvb, row, k0, kn);
    float* kb = s.kv + h * DH;
    if constexpr (LPP < 32) {
      // Lane = key: its key in registers, the weights of every query, which then take the key's place; lane = channel: every value
      // once for all queries, their weights by fours.  (A query at a time read all keys, values and a weight by shuffle for each
      // query: 66 -> 58 us for the environment-steps above.)
      float k32[DH];
      load32(k32, kb + min(lane, kn - 1) * LDB);
      __syncwarp();
#pragma unroll 1
      for (int i0 = 0; i0 < n; i0 += 4) {   // four queries side by side, the last ones perhaps the last query again
        float m0[4], mx[4], sum[4], p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = min(i0 + u, n - 1);
          const float sc = lane < kn ? dot32(q + i * LDQ, k32) * SCALE : -INFINITY;
          m0[u] = s.m[i * H + h];
          mx[u] = fmaxf(m0[u], seg_max<32>(sc));
          p[u] = lane < kn ? expf(sc - mx[u]) : 0.f;
          sum[u] = seg_sum<32>(p[u]);
        }
        if (lane < kn) *reinterpret_cast<float4*>(kb + lane * LDB + i0) = make_float4(p[0], p[1], p[2], p[3]);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u;
          if (i >= n) break;
          const float corr = expf(m0[u] - mx[u]);     // exp(-inf) = 0 on the first block
          s.acc[(n + i) * D + h * DH + lane] *= corr;
          if (lane == 0) {
            s.m[i * H + h] = mx[u];
            s.l[i * H + h] = s.l[i * H + h] * corr + sum[u];
          }
        }
      }
      __syncwarp();
      float a[LPP];
#pragma unroll
      for (int i = 0; i < LPP; ++i) a[i] = i < n ? s.acc[(n + i) * D + h * DH + lane] : 0.f;
#pragma unroll 4
      for (int j = 0; j < kn; ++j) {
        const float v1 = kb[j * LDB + D + lane];
#pragma unroll
        for (int i = 0; i < LPP; i += 4) {
          const float4 w = ld4(kb + j * LDB + i);
          a[i] = fmaf(w.x, v1, a[i]); a[i + 1] = fmaf(w.y, v1, a[i + 1]); a[i + 2] = fmaf(w.z, v1, a[i + 2]); a[i + 3] = fmaf(w.w, v1, a[i + 3]);
        }
      }
#pragma unroll
      for (int i = 0; i < LPP; ++i)
        if (i < n) s.acc[(n + i) * D + h * DH + lane] = a[i];
    } else {
      load32(own, kb + min(lane, kn - 1) * LDB);
      for (int i = 0; i < n; ++i) {
        const float sc = lane < kn ? dot32(q + i * LDQ, own) * SCALE : -INFINITY;
        const float m0 = s.m[i * H + h];
        const float mx = fmaxf(m0, seg_max<32>(sc));
        const float e = lane < kn ? expf(sc - mx) : 0.f;
        const float corr = expf(m0 - mx);     // exp(-inf) = 0 on the first block
        float a = s.acc[(n + i) * D + h * DH + lane] * corr;
        for (int j = 0; j < kn; ++j) a = fmaf(__shfl_sync(0xffffffffu, e, j), kb[j * LDB + D + lane], a);
        s.acc[(n + i) * D + h * DH + lane] = a;
        const float sum = seg_sum<32>(e);
        __syncwarp();
        if (lane == 0) {
          s.m[i * H + h] = mx;
          s.l[i * H + h] = s.l[i * H + h] * corr + sum;
        }
        __syncwarp();
      }
    }
  }
  for (int i = 0; i < n; ++i) {
    const int at = i * D + h * DH + lane;
    c.o[tok0 * D + at] = s.acc[at] + s.acc[n * D + at] / s.l[i * H + h];
  }
}

// Gradient.
// (Without bullets the sums of 32 channels a lane that their keys need would only cost registers, and so CTAs.)
template <int LPP, bool BULLETS>
__global__ void __launch_bounds__(THREADS, LPP == 32 ? 4 : BULLETS ? 3 : LPP == 16 ? 6 : 8) k_env_attn_bwd(const Call c) {
  extern __shared__ __align__(16) char raw[];
  tensor::let_next_start();
  tensor::wait_for_previous();
  constexpr int QPW = 32 / LPP, CPL = DH / LPP;
  Smem s;
  carve(raw, c.n, BULLETS ? c.nb : 0, true, &s);
  const int h = threadIdx.x >> 5, lane = threadIdx.x & 31, qs = lane / LPP, sub = lane % LPP;
  const int n = c.n;
  const size_t g = blockIdx.x, tok0 = g * n;
  rows_in<3 * D>(s.rows, LDQ, c.qkv + tok0 * 3 * D, n);
  rows_in<D>(s.d_o, LDO, c.d_o + tok0 * D, n);
  int keys = 0;
  KeyRows row{};
  if constexpr (BULLETS) {
    row = key_rows(c, g, s.list, s.count, &keys);
    for (int i = threadIdx.x; i < n * LDO; i += THREADS) s.dq[i] = 0.f;
    for (int i = threadIdx.x; i < n * H; i += THREADS) { s.m[i] = -INFINITY; s.l[i] = s.s[i] = 0.f; }
    // slots that are no keys have no gradient
    const uint8_t* on = c.bactive && !c.boff ? c.bactive + g * c.nb : nullptr;
    for (int i = threadIdx.x; on && i < c.nb * (2 * D / 4); i += THREADS)
      if (const int r = i / (2 * D / 4); !on[r]) *parts_at<2>(c.dkvb, c.ld_dkvb, c.off_dkvb, g * c.nb + r, i) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  copies_done();
  float* q = s.rows + h * DH;
  float* k = q + D;
  float* v = q + 2 * D;
  const float* go = s.d_o + h * DH;
  if (BULLETS && keys) {
    float dk[DH], dv[DH];
    // one sweep for the softmax statistics of every query, one for the gradients (up to a block of keys both in one)
    constexpr bool FEW = LPP < 32;
    if (FEW && keys <= BLOCK) {
      __syncthreads();
      stage_keys(s.kv, c.kvb, row, 0, keys);
    }
    for (int k0 = 0; k0 < keys && !(FEW && keys <= BLOCK); k0 += BLOCK) {
      const int kn = min(BLOCK, keys - k0);
      __syncthreads();
      stage_keys(s.kv, c.kvb, row, k0, kn);
      const float* kb = s.kv + h * DH;
      for (int i = 0; i < n; ++i) {
        const float sc = lane < kn ? dot32(q + i * LDQ, kb + lane * LDB) * SCALE : -INFINITY;
        const float dp = lane < kn ? dot32(go + i * LDO, kb + lane * LDB + D) : 0.f;
        const float m0 = s.m[i * H + h];
        const float mx = fmaxf(m0, seg_max<32>(sc));
        const float e = lane < kn ? expf(sc - mx) : 0.f;
        const float corr = expf(m0 - mx), sum = seg_sum<32>(e), sdp = seg_sum<32>(e * dp);
        __syncwarp();
        if (lane == 0) {
          s.m[i * H + h] = mx;
          s.l[i * H + h] = s.l[i * H + h] * corr + sum;
          s.s[i * H + h] = s.s[i * H + h] * corr + sdp;
        }
        __syncwarp();
      }
    }
    for (int k0 = 0; k0 < keys; k0 += BLOCK) {
      const int kn = min(BLOCK, keys - k0);
      if (keys > BLOCK) {    // a single block is still there
        __syncthreads();
        stage_keys(s.kv, c.kvb, row, k0, kn);
      }
      float* kb = s.kv + h * DH;
      if constexpr (FEW) {
        // Lane = key, its key and value in registers while every query's weight and score gradient are computed, which take the
        // value's place; lane = channel sums d q of all queries over the keys, each read once; lane = key again its own
        // gradients.  Loops over four queries stay loops: unrolled over all of them a quarter of the stalls were instruction
        // fetches.  1536 environment-steps of 12 tokens with 18 of 80 bullets 153 -> 108 us; a query at a time read every key and value
        // twice and each score gradient by shuffle, and the slots not in use got their zeros here.
        const int mine = min(lane, kn - 1);
#pragma unroll
        for (int d4 = 0; d4 < DH / 4; ++d4) {
          *reinterpret_cast<float4*>(&dk[4 * d4]) = ld4(kb + mine * LDB + 4 * d4);
          *reinterpret_cast<float4*>(&dv[4 * d4]) = ld4(kb + mine * LDB + D + 4 * d4);
        }
        __syncwarp();
        float* own = kb + mine * LDB + D;   // in place of the value: score gradients of the queries, then their weights
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += 4) {   // four queries side by side, the last ones perhaps the last query again
          float sc[4], dp[4], m[4], l[4], sdp[4], p[4], ds[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = min(i0 + u, n - 1);
            const float qk = dot32(q + i * LDQ, dk);
            sc[u] = lane < kn ? qk * SCALE : -INFINITY;
            dp[u] = lane < kn ? dot32(go + i * LDO, dv) : 0.f;
            if (keys <= BLOCK) {
              m[u] = seg_max<32>(sc[u]);
              const float e = lane < kn ? expf(sc[u] - m[u]) : 0.f;
              l[u] = seg_sum<32>(e);
              sdp[u] = seg_sum<32>(e * dp[u]);
            } else {
              m[u] = s.m[i * H + h];
              l[u] = s.l[i * H + h];
              sdp[u] = s.s[i * H + h];
            }
            p[u] = lane < kn && i0 + u < n ? expf(fmaf(qk, SCALE, -(m[u] + logf(l[u])))) : 0.f;   // rounded once, as where a query comes at a time
            ds[u] = p[u] * (dp[u] - sdp[u] / l[u]) * SCALE;
          }
          if (lane < kn) {
            *reinterpret_cast<float4*>(own + i0) = make_float4(ds[0], ds[1], ds[2], ds[3]);
            *reinterpret_cast<float4*>(own + 16 + i0) = make_float4(p[0], p[1], p[2], p[3]);
          }
        }
        __syncwarp();
        {
          float a[LPP];
#pragma unroll
          for (int i = 0; i < LPP; ++i) a[i] = i < n ? s.dq[i * LDO + h * DH + lane] : 0.f;
#pragma unroll 4
          for (int j = 0; j < kn; ++j) {
            const float k1 = kb[j * LDB + lane];
#pragma unroll
            for (int i = 0; i < LPP; i += 4) {
              const float4 w = ld4(kb + j * LDB + D + i);
              a[i] = fmaf(w.x, k1, a[i]); a[i + 1] = fmaf(w.y, k1, a[i + 1]); a[i + 2] = fmaf(w.z, k1, a[i + 2]); a[i + 3] = fmaf(w.w, k1, a[i + 3]);
            }
          }
#pragma unroll
          for (int i = 0; i < LPP; ++i)
            if (i < n) s.dq[i * LDO + h * DH + lane] = a[i];
        }
#pragma unroll
        for (int d = 0; d < DH; ++d) dk[d] = dv[d] = 0.f;
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += 4) {
          const float4 ds4 = ld4(own + i0), p4 = ld4(own + 16 + i0);
          const float ds[4] = {ds4.x, ds4.y, ds4.z, ds4.w}, p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {   // past the last query both are 0
            const int i = min(i0 + u, n - 1);
            const float* qi = q + i * LDQ;
            const float* gi = go + i * LDO;
#pragma unroll
            for (int d4 = 0; d4 < DH / 4; ++d4) {
              const float4 a = ld4(qi + 4 * d4), b = ld4(gi + 4 * d4);
              dk[4 * d4] = fmaf(ds[u], a.x, dk[4 * d4]); dk[4 * d4 + 1] = fmaf(ds[u], a.y, dk[4 * d4 + 1]);
              dk[4 * d4 + 2] = fmaf(ds[u], a.z, dk[4 * d4 + 2]); dk[4 * d4 + 3] = fmaf(ds[u], a.w, dk[4 * d4 + 3]);
              dv[4 * d4] = fmaf(p[u], b.x, dv[4 * d4]); dv[4 * d4 + 1] = fmaf(p[u], b.y, dv[4 * d4 + 1]);
              dv[4 * d4 + 2] = fmaf(p[u], b.z, dv[4 * d4 + 2]); dv[4 * d4 + 3] = fmaf(p[u], b.w, dv[4 * d4 + 3]);
            }
          }
        }
      } else {
#pragma unroll
        for (int d = 0; d < DH; ++d) dk[d] = dv[d] = 0.f;
        for (int i = 0; i < n; ++i) {
          const float l = s.l[i * H + h], lse = s.m[i * H + h] + logf(l), delta = s.s[i * H + h] / l;
          const float* qi = q + i * LDQ;
          const float* gi = go + i * LDO;
          float p = 0.f, ds = 0.f;
          if (lane < kn) {
            p = expf(dot32(qi, kb + lane * LDB) * SCALE - lse);
            ds = p * (dot32(gi, kb + lane * LDB + D) - delta) * SCALE;
          }
#pragma unroll
          for (int d4 = 0; d4 < DH / 4; ++d4) {
            const float4 a = ld4(qi + 4 * d4), b = ld4(gi + 4 * d4);
            dk[4 * d4] = fmaf(ds, a.x, dk[4 * d4]); dk[4 * d4 + 1] = fmaf(ds, a.y, dk[4 * d4 + 1]);
            dk[4 * d4 + 2] = fmaf(ds, a.z, dk[4 * d4 + 2]); dk[4 * d4 + 3] = fmaf(ds, a.w, dk[4 * d4 + 3]);
            dv[4 * d4] = fmaf(p, b.x, dv[4 * d4]); dv[4 * d4 + 1] = fmaf(p, b.y, dv[4 * d4 + 1]);
            dv[4 * d4 + 2] = fmaf(p, b.z, dv[4 * d4 + 2]); dv[4 * d4 + 3] = fmaf(p, b.w, dv[4 * d4 + 3]);
          }
          float dq = s.dq[i * LDO + h * DH + lane];
          for (int j = 0; j < kn; ++j) dq = fmaf(__shfl_sync(0xffffffffu, ds, j), kb[j * LDB + lane], dq);
          s.dq[i * LDO + h * DH + lane] = dq;
        }
      }
      __syncwarp();          // the head's keys and values of this block are done: their gradients take their place
      if (lane < kn)
#pragma unroll
        for (int d4 = 0; d4 < DH / 4; ++d4) {
          *reinterpret_cast<float4*>(kb + lane * LDB + 4 * d4) = make_float4(dk[4 * d4], dk[4 * d4 + 1], dk[4 * d4 + 2], dk[4 * d4 + 3]);
          *reinterpret_cast<float4*>(kb + lane * LDB + D + 4 * d4) = make_float4(dv[4 * d4], dv[4 * d4 + 1], dv[4 * d4 + 2], dv[4 * d4 + 3]);
        }
      __syncthreads();
      for (int i = threadIdx.x; i < kn * (2 * D / 4); i += THREADS) {
        const int r = i / (2 * D / 4), qq = i % (2 * D / 4);
        *parts_at<2>(c.dkvb, c.ld_dkvb, c.off_dkvb, row(k0 + r), qq) = ld4(s.kv + r * LDB + qq * 4);
      }
    }
  }

  const bool key = sub < n;
  const bool dead = key && c.alive && !c.alive[tok0 + sub];
  // probability and score gradient of (query, key sub)
  const auto weights = [&](int i, float& p, float& ds) {
    const int ic = min(i, n - 1);
    const float* qi = q + ic * LDQ;
    const float* gi = go + ic * LDO;
    float sc = -INFINITY, dp = 0.f;
    if (key) {
      sc = dead ? kMaskedScore : dot32(qi, k + sub * LDQ) * SCALE;
      dp = dot32(gi, v + sub * LDQ);
    }
    const float mx = seg_max<LPP>(sc);
    const float e = key ? expf(sc - mx) : 0.f;
    const float l = seg_sum<LPP>(e);
    const float lse = mx + logf(l);
    const float delta = seg_sum<LPP>(e / l * dp);   // <d out, out>
    p = key && i < n ? expf(sc - lse) : 0.f;
    ds = p * (dp - delta) * SCALE;
  };
  // d q of query i from its score gradients, one per lane; it takes the place of q
  const auto query_gradient = [&](int i, float ds) {
    float dq[CPL];
#pragma unroll
    for (int d = 0; d < CPL; ++d) dq[d] = BULLETS && keys && i < n ? s.dq[i * LDO + h * DH + sub * CPL + d] : 0.f;
    for (int j = 0; j < n; ++j) {
      const float dsj = __shfl_sync(0xffffffffu, ds, qs * LPP + j);
      const float* kj = k + j * LDQ + sub * CPL;
#pragma unroll
      for (int d = 0; d < CPL; ++d) dq[d] = fmaf(dsj, kj[d], dq[d]);
    }
    __syncwarp();            // this head's q of these queries is done with
    if (i < n)
#pragma unroll
      for (int d = 0; d < CPL; ++d) q[i * LDQ + sub * CPL + d] = dq[d];
  };
  if constexpr (LPP < 32) {
    // Every query's weights first (ROUNDS a lane), then lane (qs, sub) sums CH = LPP channels of d k and d v of key sub over all
    // queries: 2 CH accumulators and a broadcast per query, where shares of 32 channels each over the group's queries took 64
    // accumulators and as many sums over the groups at the end: 32 768 environment-steps of 8 tokens 343 -> 237 us.
    constexpr int ROUNDS = LPP / QPW, CH = LPP;
    float p[ROUNDS], ds[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      p[r] = ds[r] = 0.f;
      if (r * QPW < n) weights(r * QPW + qs, p[r], ds[r]);
    }
    float gk[CH], gv[CH];
#pragma unroll
    for (int d = 0; d < CH; ++d) gk[d] = gv[d] = 0.f;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
#pragma unroll
      for (int g2 = 0; g2 < QPW; ++g2) {
        const int i = r * QPW + g2;
        if (i >= n) break;
        const float pi = __shfl_sync(0xffffffffu, p[r], g2 * LPP + sub), di = __shfl_sync(0xffffffffu, ds[r], g2 * LPP + sub);
        const float* qi = q + i * LDQ + qs * CH;
        const float* gi = go + i * LDO + qs * CH;
#pragma unroll
        for (int d4 = 0; d4 < CH / 4; ++d4) {
          const float4 a = ld4(qi + 4 * d4), b = ld4(gi + 4 * d4);
          gk[4 * d4] = fmaf(di, a.x, gk[4 * d4]); gk[4 * d4 + 1] = fmaf(di, a.y, gk[4 * d4 + 1]);
          gk[4 * d4 + 2] = fmaf(di, a.z, gk[4 * d4 + 2]); gk[4 * d4 + 3] = fmaf(di, a.w, gk[4 * d4 + 3]);
          gv[4 * d4] = fmaf(pi, b.x, gv[4 * d4]); gv[4 * d4 + 1] = fmaf(pi, b.y, gv[4 * d4 + 1]);
          gv[4 * d4 + 2] = fmaf(pi, b.z, gv[4 * d4 + 2]); gv[4 * d4 + 3] = fmaf(pi, b.w, gv[4 * d4 + 3]);
        }
      }
    __syncwarp();            // this head's q has been read
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
      if (r * QPW < n) query_gradient(r * QPW + qs, ds[r]);
    __syncwarp();            // and so have its k and v
    if (key)
#pragma unroll
      for (int d4 = 0; d4 < CH / 4; ++d4) {
        *reinterpret_cast<float4*>(k + sub * LDQ + qs * CH + 4 * d4) = make_float4(gk[4 * d4], gk[4 * d4 + 1], gk[4 * d4 + 2], gk[4 * d4 + 3]);
        *reinterpret_cast<float4*>(v + sub * LDQ + qs * CH + 4 * d4) = make_float4(gv[4 * d4], gv[4 * d4 + 1], gv[4 * d4 + 2], gv[4 * d4 + 3]);
      }
  } else {
    float dk[DH], dv[DH];
#pragma unroll
    for (int d = 0; d < DH; ++d) dk[d] = dv[d] = 0.f;
    for (int i = 0; i < n; ++i) {
      float p, ds;
      weights(i, p, ds);
      const float* qi = q + i * LDQ;
      const float* gi = go + i * LDO;
#pragma unroll
      for (int d4 = 0; d4 < DH / 4; ++d4) {
        const float4 a = ld4(qi + 4 * d4), b = ld4(gi + 4 * d4);
        dk[4 * d4] = fmaf(ds, a.x, dk[4 * d4]); dk[4 * d4 + 1] = fmaf(ds, a.y, dk[4 * d4 + 1]);
        dk[4 * d4 + 2] = fmaf(ds, a.z, dk[4 * d4 + 2]); dk[4 * d4 + 3] = fmaf(ds, a.w, dk[4 * d4 + 3]);
        dv[4 * d4] = fmaf(p, b.x, dv[4 * d4]); dv[4 * d4 + 1] = fmaf(p, b.y, dv[4 * d4 + 1]);
        dv[4 * d4 + 2] = fmaf(p, b.z, dv[4 * d4 + 2]); dv[4 * d4 + 3] = fmaf(p, b.w, dv[4 * d4 + 3]);
      }
      query_gradient(i, ds);
    }
    __syncwarp();
    if (key)
#pragma unroll
      for (int d4 = 0; d4 < DH / 4; ++d4) {
        *reinterpret_cast<float4*>(k + sub * LDQ + 4 * d4) = make_float4(dk[4 * d4], dk[4 * d4 + 1], dk[4 * d4 + 2], dk[4 * d4 + 3]);
        *reinterpret_cast<float4*>(v + sub * LDQ + 4 * d4) = make_float4(dv[4 * d4], dv[4 * d4 + 1], dv[4 * d4 + 2], dv[4 * d4 + 3]);
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * (3 * D / 4); i += THREADS) {
    const int r = i / (3 * D / 4), qq = i % (3 * D / 4);
    *parts_at<3>(c.dqkv, c.ld_dqkv, c.off_dqkv, tok0 + r, qq) = ld4(s.rows + r * LDQ + qq * 4);
  }
}

constexpr size_t SMEM_MAX = 200 * 1024;

template <typename K>
int launch(K kernel, const Call& c, bool grad, cudaStream_t st) {
  const size_t smem = carve(nullptr, c.n, c.kvb ? c.nb : 0, grad, nullptr);
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX) != cudaSuccess) return 7;
  return launch_after(kernel, dim3(c.G), THREADS, smem, st, c);
}

}  // namespace

bool supported(int d_model, int n_heads, int n, int nb) {
  return d_model == D && n_heads == H && n >= 1 && n <= 32 && nb >= 0 && nb <= 65535 && carve(nullptr, n, nb, true, nullptr) <= SMEM_MAX;
}
int forward(const Call& c, cudaStream_t st) {
  if (c.G <= 0) return 0;
  if (c.kvb) return c.n <= 8 ? launch(k_env_attn_fwd<8, true>, c, false, st) : c.n <= 16 ? launch(k_env_attn_fwd<16, true>, c, false, st) : launch(k_env_attn_fwd<32, true>, c, false, st);
  return c.n <= 8 ? launch(k_env_attn_fwd<8, false>, c, false, st) : c.n <= 16 ? launch(k_env_attn_fwd<16, false>, c, false, st) : launch(k_env_attn_fwd<32, false>, c, false, st);
}
int backward(const Call& c, cudaStream_t st) {
  if (c.G <= 0) return 0;
  if (c.kvb) return c.n <= 8 ? launch(k_env_attn_bwd<8, true>, c, true, st) : c.n <= 16 ? launch(k_env_attn_bwd<16, true>, c, true, st) : launch(k_env_attn_bwd<32, true>, c, true, st);
  return c.n <= 8 ? launch(k_env_attn_bwd<8, false>, c, true, st) : c.n <= 16 ? launch(k_env_attn_bwd<16, false>, c, true, st) : launch(k_env_attn_bwd<32, false>, c, true, st);
}

}  // namespace train_attn
}  // namespace bnb
