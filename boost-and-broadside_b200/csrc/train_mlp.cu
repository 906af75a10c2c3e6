// The GatedMLP of the training path: y = x + down(gelu(gate n) * up n) with n = rmsnorm(x) * gain, and its
// gradient, under the bfloat16 contract (every product's operands bfloat16, float32 accumulation; what lies
// between two products is float32 and rounded once, where it becomes an operand), d_model 128, hidden 512.
// models/yemong/attention.py:21-37 under autocast; norms and residual stream float32.
//
// Nothing 4 d_model wide leaves the chip.  As separate products, gate, up, their product and its
// gradients were five (rows, 512) tensors, written once and read up to three times: 12.5 of the 23.5 ms of
// a training step of 262 144 rows.  Three kernels instead, each with the gate|up product recomputed where
// it is needed (K = 128: cheaper than reading its result back):
//
//   k_mlp_fwd   row tiles of 128: residual in tensor memory, gate|up of 64 hidden columns at a time, the
//               gated product as the A operand of the down projection in tensor memory.
//   k_mlp_dx    row tiles again: gate|up from n and d h from dy side by side, d gate | d up as the A operand
//               of dn = d gate Wg + d up Wu in tensor memory, then the norm's gradient.  Writes n and dy as
//               bfloat16 tile images for the third kernel.
//   k_mlp_dw    a CTA keeps one chunk of 64 hidden columns and walks row tiles: gate|up and d h of the
//               chunk again, then d Wg, d Wu, d Wd of the chunk accumulated in tensor memory over all its
//               tiles.  Row tiles serve as operands in both directions as they are: K-major for the
//               products over the width, MN-major (same bytes, another descriptor) for those over the rows.
//
// All three: sixteen epilogue warps, one issuing and one fetching warp that meet at mbarriers; weights
// stream from pre-tiled images through a ring (L2 to shared memory), every wait is bounded.
// What bounds them is the latency of that hand-off, at 18 warps per SM.  262 144 rows: k_mlp_fwd 186 us, 22 000 cycles a tile of which
// 9 800 are gelu, 2 400 waits for gate|up, 9 500 its start (rows, norm) and end, which overlap with no other tile's chunks (196 with each
// request right in front of its use); k_mlp_dx 287, 36 000 cycles a tile, 9 100 gelu and its gradient, 7 400 waits for products,
// 20 000 start and end (301 with dy row by row between the stores); k_mlp_dw 241, 2 900 cycles a tile and chunk, 1 600 gelu, 430 waits for
// products (273 and 1 100 with n and dy in one copy that waited for both products, from HBM).
#include "train_mlp.h"

#include "launch_after.h"
#include "tensor_kernels.h"
#include "tile_rows.cuh"

namespace bnb {
namespace train_mlp {

using namespace tensor;

namespace {

constexpr int F = 512, NCHUNK = 8;                 // hidden width, chunks of 64 hidden columns
// one chunk of a weight image: gate|up (two K atoms of 128 rows), down transposed (two K atoms of 64 rows),
// gate and up transposed (128 rows x 64 k each), down (128 rows x 64 k)
constexpr uint32_t IMG_GU = 0, IMG_DH = 32768, IMG_DN = 49152, IMG_D = 81920, IMG_CHUNK = 98304;
constexpr uint32_t IMAGE = NCHUNK * IMG_CHUNK;

// ------------------------------------------------------------------ weight images

struct PackJobs { Weights w[MAX_JOBS]; };
// One thread per 16-byte group (eight k of one row); rows run along the threads where the source is
// transposed, so that its reads are contiguous too.
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackJobs jobs, uint8_t* image) {
  const Weights& w = jobs.w[blockIdx.y];
  uint8_t* out = image + (size_t)blockIdx.y * IMAGE;
  const int per_chunk = IMG_CHUNK / 16;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NCHUNK * per_chunk; i += gridDim.x * blockDim.x) {
    const int c = i / per_chunk, j = i - c * per_chunk;
    uint8_t* base = out + (size_t)c * IMG_CHUNK;
    float v[8];
    uint32_t at;
    if (j < (int)(IMG_DH / 16) || j >= (int)(IMG_D / 16)) {   // rows as stored
      const float* src;
      if (j < (int)(IMG_DH / 16)) {
        const int atom = j >> 10, r = (j >> 3) & 127, g = j & 7;
        src = (r < 64 ? w.gate + (size_t)(64 * c + r) * D : w.up + (size_t)(64 * c + r - 64) * D) + atom * 64 + g * 8;
        at = IMG_GU + atom * CHUNK_BYTES + swz(r, g);
      } else {
        const int k = j - IMG_D / 16, r = k >> 3, g = k & 7;
        src = w.down + (size_t)r * F + 64 * c + g * 8;
        at = IMG_D + swz(r, g);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 f = *reinterpret_cast<const float4*>(src + 4 * q);
        v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
      }
    } else if (j < (int)(IMG_DN / 16)) {          // d h = dy Wd: row = hidden column, k = model dimension
      const int k = j - IMG_DH / 16, r = k & 63, g = (k >> 6) & 7, atom = k >> 9;
      const float* src = w.down + (size_t)(atom * 64 + g * 8) * F + 64 * c + r;
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = src[(size_t)q * F];
      at = IMG_DH + atom * (CHUNK_BYTES / 2) + swz(r, g);
    } else {                                       // dn = d gate Wg + d up Wu: row = model dimension, k = hidden column
      const int k = j - IMG_DN / 16, r = k & 127, g = (k >> 7) & 7, atom = k >> 10;
      const float* src = (atom ? w.up : w.gate) + (size_t)(64 * c + g * 8) * D + r;
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = src[(size_t)q * D];
      at = IMG_DN + atom * CHUNK_BYTES + swz(r, g);
    }
    *reinterpret_cast<uint4*>(base + at) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  }
}

// ------------------------------------------------------------------ shared pieces

struct Args {
  const float* x1;
  const float* dy;
  float* out;              // y or dx1
  const float* gain;
  float* d_gain;
  const uint8_t* image;    // weight image
  uint8_t* n_image;
  uint8_t* dy_image;
  float *d_gate, *d_up, *d_down;
  int rows, tiles;
  int* status;
  int* host_status;
};

// Phi(x) and exp(-x^2 / 2) for two x: erf by formula 7.1.26 of Abramowitz and Stegun (absolute error 1.5e-7),
// whose exponential is the density's too.
__device__ __forceinline__ F2 normal_cdf(F2 x, F2& e) {
  const float2 xs = halves(x);
  const float2 d = halves(fma(f2(fabsf(xs.x), fabsf(xs.y)), f2(0.3275911f * 0.70710678f), f2(1.0f)));
  const F2 t = f2(rcp_fast(d.x), rcp_fast(d.y));
  const float2 q = halves(mul(mul(x, x), f2(-0.72134752f)));   // log2(e) / 2
  e = f2(ex2_fast(q.x), ex2_fast(q.y));
  F2 p = fma(t, f2(0.5f * 1.061405429f), f2(0.5f * -1.453152027f));
  p = fma(t, p, f2(0.5f * 1.421413741f));
  p = fma(t, p, f2(0.5f * -0.284496736f));
  p = fma(t, p, f2(0.5f * 0.254829592f));
  const float2 half = halves(mul(mul(p, t), e));               // (1 - erf(|x| / sqrt 2)) / 2
  return f2(xs.x >= 0.f ? 1.0f - half.x : half.x, xs.y >= 0.f ? 1.0f - half.y : half.y);
}
__device__ __forceinline__ uint32_t pack_f2(F2 a) { const float2 v = halves(a); return pack_bf16(v.x, v.y); }
__device__ __forceinline__ F2 acc_pair(const uint32_t* v) { return f2(__uint_as_float(v[0]), __uint_as_float(v[1])); }
// n = bf16(x inv gain) into an operand tile; inv[i] of this lane's rows on the way
__device__ __forceinline__ void norm_rows(uint8_t* tile, const float4 (&x)[8], float (&inv)[8], const float4& gain, float* part_sums, const RowMap& m) {
#pragma unroll
  for (int i = 0; i < 8; ++i) inv[i] = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, fmaf(x[i].z, x[i].z, x[i].w * x[i].w)));
  row_sums(inv, part_sums, m);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    inv[i] = rsqrtf(inv[i] * (1.0f / D) + kRmsEps);
    put_row4(tile, m, i, make_float4(x[i].x * inv[i] * gain.x, x[i].y * inv[i] * gain.y, x[i].z * inv[i] * gain.z, x[i].w * inv[i] * gain.w));
  }
}
// One fetch by the fetching warp: wait for the slot, copy, signal.  Stops after a wait has run out.
__device__ __forceinline__ bool fetch(const Sync& s, int full, int done, uint32_t free_parity, uint32_t dst, const uint8_t* src, uint32_t bytes,
                                      bool elected) {
  s.wait(done, free_parity, TIMEOUT_FREE);
  if (__any_sync(0xffffffffu, s.aborted[0])) return false;
  if (elected) {
    mbar_expect_tx(s.bars + 8 * full, bytes);
    bulk_g2s(dst, src, bytes, s.bars + 8 * full);
  }
  __syncwarp();
  return true;
}
// ------------------------------------------------------------------ forward

// Shared memory: n (32 KB), three gate|up slots (32 KB), three down slots (16 KB), row sums, frame.
constexpr uint32_t FW_PAIR = 32768, FW_SINGLE = FW_PAIR + 3 * 32768, FW_SUMS = FW_SINGLE + 3 * 16384, FW_FRAME = FW_SUMS + 2048,
                   FW_BYTES = FW_FRAME + FRAME_BYTES;
enum : int { FB_OP = 0, FB_FFN0, FB_ACC = FB_FFN0 + 3, FB_DRAIN, FB_FULL0, FB_DONE0 = FB_FULL0 + 6, FB_COUNT = FB_DONE0 + 6 };

__device__ __forceinline__ uint32_t fw_slot(uint32_t i) { return i < 3 ? FW_PAIR + i * 32768 : FW_SINGLE + (i - 3) * 16384; }

// Tensor memory: down projection [0, 128), three gate|up accumulators.  The output transpose stages in the
// operand area, free once a tile's products are complete (the ring behind it may be refilling): 4 KB per warp,
// eight warps at a time.
__global__ void __launch_bounds__(THREADS, 1) k_mlp_fwd(const __grid_constant__ Args a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int counts[FB_COUNT] = {EPI_WARPS, EPI_WARPS / 2, EPI_WARPS / 2, EPI_WARPS / 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};
  const int tid = threadIdx.x, warp = tid >> 5;
  const Frame f = open_frame(smem + FW_FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot;
  const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

  if (warp == LOAD_WARP) {
    const uint32_t base = smem_u32(smem);
    const bool elected = elect_one() != 0;
    uint32_t pair = 0, single = 3, par = 0x3F;   // a fresh barrier passes a wait on parity 1
    bool go = true;
    for (int t = 0; t < my_tiles && go; ++t) {
      if (elected) prefetch_rows(a.x1, blockIdx.x + (t + 1) * gridDim.x, a.rows, D * 4);
#pragma unroll 1
      for (int i = 0; i < 16 && go; ++i) {
        // GU0 GU1 GU2 D0 GU3 D1 ... GU7 D5 D6 D7
        const bool down = i >= 3 && ((i & 1) || i > 13);
        const int c = i < 3 ? i : i > 13 ? i - 8 : down ? (i - 3) / 2 : (i + 2) / 2;
        const uint32_t slot = down ? single : pair;
        if (down) single = single == 5 ? 3 : single + 1;
        else pair = pair == 2 ? 0 : pair + 1;
        go = fetch(s, FB_FULL0 + slot, FB_DONE0 + slot, par >> slot, base + fw_slot(slot), a.image + (size_t)c * IMG_CHUNK + (down ? IMG_D : IMG_GU),
                   down ? 16384 : 32768, elected);
        par ^= 1u << slot;
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t base = smem_u32(smem), el = elect_one(), tm = uniform(tmem);
    const uint32_t n_lo = desc_lo(base), idesc = instr_desc(128);
    uint32_t pair = 0, single = 3, full = 0, op = 0, ffn = 0;
    auto gate_up = [&](uint32_t acc) {
      s.wait(FB_FULL0 + pair, full >> pair, TIMEOUT_FULL);
      full ^= 1u << pair;
      product128(el, tm + 128 + 128 * acc, n_lo, uniform(desc_lo(base + FW_PAIR + pair * 32768)), 1024, idesc);
      tc_commit_if(el, s.bars + 8 * (FB_DONE0 + pair));
      pair = pair == 2 ? 0 : pair + 1;
    };
    for (int t = 0; t < my_tiles; ++t) {
      s.wait(FB_OP, op, TIMEOUT_OPERAND);
      op ^= 1u;
      tc_fence_after();
#pragma unroll 1
      for (uint32_t c = 0; c < 3; ++c) gate_up(c);
      uint32_t acc = 0;
#pragma unroll 1
      for (uint32_t c = 0; c < 8; ++c) {
        s.wait(FB_FFN0 + acc, ffn >> acc, TIMEOUT_OPERAND);
        ffn ^= 1u << acc;
        tc_fence_after();
        s.wait(FB_FULL0 + single, full >> single, TIMEOUT_FULL);
        full ^= 1u << single;
        const uint32_t b = uniform(desc_lo(base + FW_SINGLE + (single - 3) * 16384));
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) mma_one<true>(el, tm, tm + 128 + 128 * acc + 16 * k, b + 2 * k, idesc, (c | k) ? 1u : 0u);
        tc_commit_if(el, s.bars + 8 * (FB_DONE0 + single));
        single = single == 5 ? 3 : single + 1;
        if (c + 3 < 8) gate_up(acc);
        acc = acc == 2 ? 0 : acc + 1;
      }
      tc_commit_if(el, s.bars + 8 * FB_ACC);
    }
    tc_commit_if(el, s.bars + 8 * FB_DRAIN);
    for (int i = 0; i < DEFAULT_POLL_LIMIT && !mbar_try_wait(s.bars + 8 * FB_DRAIN, 0); ++i) {
    }
  } else {
    const int part = tid >> 7, group = part >> 1, half = part & 1;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t pair = 0, par = 0, acc_par = 0;
    const RowMap m = row_map();
    const float4 gain = *reinterpret_cast<const float4*>(a.gain + m.col);
    // Rows are on their way before the waits in front of their use: the next tile's as this tile's leave, the residual's
    // as the last chunk does.
    float4 x[8];
    rows_in(x, a.x1, m, blockIdx.x * TILE, a.rows);
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
      epi_sync();   // every warp is done with the operand area of the previous tile
      {
        float inv[8];
        norm_rows(smem, x, inv, gain, reinterpret_cast<float*>(smem + FW_SUMS), m);
      }
      post(s, FB_OP);
#pragma unroll 1
      for (int c = 0; c < NCHUNK; ++c) {
        if ((c & 1) == group) {   // two groups of eight warps take turns
          s.wait(FB_DONE0 + pair, par >> pair, TIMEOUT_ACC);
          tc_fence_after();
          const uint32_t acc = lane_addr + 128 + (c % 3) * 128 + half * 32;
#pragma unroll 1
          for (int p = 0; p < 2; ++p) {
            uint32_t g[16], u[16], w[8];
            tmem_ld16_nowait(acc + 16 * p, g);
            tmem_ld16_nowait(acc + 64 + 16 * p, u);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const F2 x = acc_pair(&g[2 * j]);
              F2 e;
              w[j] = pack_f2(mul(mul(x, normal_cdf(x, e)), acc_pair(&u[2 * j])));
            }
            tmem_st8_nowait(acc + 16 * p, w);
          }
          tmem_wait_st();
          post(s, FB_FFN0 + c % 3);
        }
        par ^= 1u << pair;
        pair = pair == 2 ? 0 : pair + 1;
      }
      rows_in(x, a.x1, m, tile * TILE, a.rows);
      s.wait(FB_ACC, acc_par, TIMEOUT_ACC);
      acc_par ^= 1u;
      tc_fence_after();
      // y = x + down, row layout; the first eight warps stage in the operand area, then the others
      float4 d[8];
      if (group == 0) transpose_rows(d, lane_addr + part * 32, smem + (warp & 7) * 4096, m);
      epi_sync();
      if (group == 1) transpose_rows(d, lane_addr + part * 32, smem + (warp & 7) * 4096, m);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = tile * TILE + m.row(i);
        if (r < a.rows)
          *reinterpret_cast<float4*>(a.out + (size_t)r * D + m.col) = make_float4(x[i].x + d[i].x, x[i].y + d[i].y, x[i].z + d[i].z, x[i].w + d[i].w);
      }
      rows_in(x, a.x1, m, (tile + gridDim.x) * TILE, a.rows);
      tc_fence_before();
    }
  }
  close_frame(f, tmem);
}

// ------------------------------------------------------------------ gradient of the input

// Shared memory: n and dy (32 KB each), two slots of gate|up and transposed down (48 KB), two of transposed
// gate and up (32 KB), row sums, frame.
constexpr uint32_t DX_DY = 32768, DX_W1 = 65536, DX_W2 = DX_W1 + 2 * 49152, DX_SUMS = DX_W2 + 2 * 32768, DX_INV = DX_SUMS + 2048, DX_FRAME = DX_INV + 512,
                   DX_BYTES = DX_FRAME + FRAME_BYTES;
enum : int { XB_OP = 0, XB_FF0, XB_ACC = XB_FF0 + 2, XB_DRAIN, XB_FULL1, XB_DONE1 = XB_FULL1 + 2, XB_FULL2 = XB_DONE1 + 2, XB_DONE2 = XB_FULL2 + 2, XB_COUNT = XB_DONE2 + 2 };
// Tensor memory: dn [0, 128), two accumulator sets of gate|up (128 columns) and d h (64).
__device__ __forceinline__ uint32_t dx_acc(uint32_t i) { return 128 + 192 * i; }

__global__ void __launch_bounds__(THREADS, 1) k_mlp_dx(const __grid_constant__ Args a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int counts[XB_COUNT] = {EPI_WARPS, EPI_WARPS / 2, EPI_WARPS / 2, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};
  const int tid = threadIdx.x, warp = tid >> 5;
  const Frame f = open_frame(smem + DX_FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot;
  const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

  if (warp == LOAD_WARP) {
    const uint32_t base = smem_u32(smem);
    const bool elected = elect_one() != 0;
    uint32_t par1 = 3, par2 = 3;
    bool go = true;
    // W1(0) W1(1) then W2(c), W1(c + 2)
    for (int t = 0; t < my_tiles && go; ++t) {
      if (elected) {
        prefetch_rows(a.x1, blockIdx.x + (t + 1) * gridDim.x, a.rows, D * 4);
        prefetch_rows(a.dy, blockIdx.x + (t + 1) * gridDim.x, a.rows, D * 4);
      }
#pragma unroll 1
      for (int i = 0; i < 16 && go; ++i) {
        const bool second = i >= 2 && (!(i & 1) || i > 13);
        const int c = i < 2 ? i : i > 13 ? i - 8 : second ? (i - 2) / 2 : (i + 1) / 2;
        const uint32_t slot = c & 1;
        const uint8_t* src = a.image + (size_t)c * IMG_CHUNK;
        if (second) {
          go = fetch(s, XB_FULL2 + slot, XB_DONE2 + slot, par2 >> slot, base + DX_W2 + slot * 32768, src + IMG_DN, 32768, elected);
          par2 ^= 1u << slot;
        } else {
          go = fetch(s, XB_FULL1 + slot, XB_DONE1 + slot, par1 >> slot, base + DX_W1 + slot * 49152, src + IMG_GU, 49152, elected);
          par1 ^= 1u << slot;
        }
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t base = smem_u32(smem), el = elect_one(), tm = uniform(tmem);
    const uint32_t n_lo = desc_lo(base), dy_lo = desc_lo(base + DX_DY), id128 = instr_desc(128), id64 = instr_desc(64);
    uint32_t full1 = 0, full2 = 0, op = 0, ff = 0;
    auto first = [&](uint32_t slot) {   // gate|up and d h of a chunk
      s.wait(XB_FULL1 + slot, full1 >> slot, TIMEOUT_FULL);
      full1 ^= 1u << slot;
      const uint32_t w = uniform(desc_lo(base + DX_W1 + slot * 49152)), acc = tm + dx_acc(slot);
      product128(el, acc, n_lo, w, 1024, id128);
      product128(el, acc + 128, dy_lo, w + 2048, 512, id64);
      tc_commit_if(el, s.bars + 8 * (XB_DONE1 + slot));
    };
    for (int t = 0; t < my_tiles; ++t) {
      s.wait(XB_OP, op, TIMEOUT_OPERAND);
      op ^= 1u;
      tc_fence_after();
#pragma unroll 1
      for (uint32_t c = 0; c < 2; ++c) first(c);
#pragma unroll 1
      for (uint32_t c = 0; c < 8; ++c) {
        const uint32_t slot = c & 1, acc = tm + dx_acc(slot);
        s.wait(XB_FF0 + slot, ff >> slot, TIMEOUT_OPERAND);
        ff ^= 1u << slot;
        tc_fence_after();
        s.wait(XB_FULL2 + slot, full2 >> slot, TIMEOUT_FULL);
        full2 ^= 1u << slot;
        const uint32_t w = uniform(desc_lo(base + DX_W2 + slot * 32768));
        // dn += d gate Wg + d up Wu: both halves of the operand in tensor memory, 16 columns per k step
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) mma_one<true>(el, tm, acc + 16 * k, w + 2 * k, id128, (c | k) ? 1u : 0u);
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) mma_one<true>(el, tm, acc + 64 + 16 * k, w + 1024 + 2 * k, id128, 1u);
        tc_commit_if(el, s.bars + 8 * (XB_DONE2 + slot));
        if (c + 2 < 8) first(slot);
      }
      tc_commit_if(el, s.bars + 8 * XB_ACC);
    }
    tc_commit_if(el, s.bars + 8 * XB_DRAIN);
    for (int i = 0; i < DEFAULT_POLL_LIMIT && !mbar_try_wait(s.bars + 8 * XB_DRAIN, 0); ++i) {
    }
  } else {
    const int part = tid >> 7, group = part >> 1, half = part & 1;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float *sums = reinterpret_cast<float*>(smem + DX_SUMS), *row_inv = reinterpret_cast<float*>(smem + DX_INV);
    uint32_t par = 0, acc_par = 0;
    const RowMap m = row_map();
    const float4 gain = *reinterpret_cast<const float4*>(a.gain + m.col);
    float4 gsum = make_float4(0.f, 0.f, 0.f, 0.f);   // gain gradient of this lane's columns
    float4 x[8], dn[8];
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
      // the operand area: its tiles on their way to global memory are read, the transposes of the previous
      // round done
      if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      rows_in(x, a.x1, m, tile * TILE, a.rows);
      rows_in(dn, a.dy, m, tile * TILE, a.rows);
      epi_sync();
      {
        float inv[8];
        norm_rows(smem, x, inv, gain, sums, m);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          put_row4(smem + DX_DY, m, i, dn[i]);
          if (m.col == 0) row_inv[m.row(i)] = inv[i];
        }
      }
      post(s, XB_OP);
      epi_sync();
      if (tid == 0) {   // every thread has fenced its part
        const size_t at = (size_t)tile * 32768;
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(a.n_image + at), "r"(smem_u32(smem)), "r"(32768) : "memory");
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(a.dy_image + at), "r"(smem_u32(smem) + DX_DY), "r"(32768) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
#pragma unroll 1
      for (int c = group; c < NCHUNK; c += 2) {   // accumulator set = group
        s.wait(XB_DONE1 + group, par, TIMEOUT_ACC);
        par ^= 1u;
        tc_fence_after();
        const uint32_t acc = lane_addr + dx_acc(group) + half * 32;
#pragma unroll 1
        for (int p = 0; p < 2; ++p) {
          uint32_t g[16], u[16], h[16], wg[8], wu[8];
          tmem_ld16_nowait(acc + 16 * p, g);
          tmem_ld16_nowait(acc + 64 + 16 * p, u);
          tmem_ld16_nowait(acc + 128 + 16 * p, h);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const F2 x = acc_pair(&g[2 * j]), dh = acc_pair(&h[2 * j]);
            F2 e;
            const F2 cdf = normal_cdf(x, e);
            // gelu' = Phi + x phi
            wg[j] = pack_f2(mul(mul(dh, acc_pair(&u[2 * j])), fma(mul(x, f2(0.39894228f)), e, cdf)));
            wu[j] = pack_f2(mul(dh, mul(x, cdf)));
          }
          tmem_st8_nowait(acc + 16 * p, wg);
          tmem_st8_nowait(acc + 64 + 16 * p, wu);
        }
        tmem_wait_st();
        post(s, XB_FF0 + group);
      }
      rows_in(x, a.x1, m, tile * TILE, a.rows);
      s.wait(XB_ACC, acc_par, TIMEOUT_ACC);
      acc_par ^= 1u;
      tc_fence_after();
      // the norm: dx = dy + inv gain dn - x inv^3 mean(x gain dn);  d gain += sum over rows of dn x inv.  The operand
      // area (64 KB, 4 KB per warp) stages the transpose once its copies to global memory have read it.
      if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      epi_sync();
      transpose_rows(dn, lane_addr + part * 32, smem + warp * 4096, m);
      tc_fence_before();
#pragma unroll
      for (int i = 0; i < 8; ++i) {   // sums of x gain dn over a row: eight lanes here, the four warps of the row through shared memory
        float c = fmaf(x[i].x * gain.x, dn[i].x, fmaf(x[i].y * gain.y, dn[i].y, fmaf(x[i].z * gain.z, dn[i].z, x[i].w * gain.w * dn[i].w)));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if ((m.lane & 7) == 0) sums[part * TILE + m.row(i)] = c;
      }
      asm volatile("bar.sync %0, 128;" ::"r"(3 + (warp & 3)) : "memory");   // their next use is behind the next tile's first barrier
      // four rows of dy at a time: behind a store the next load would wait for it
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        float4 dy[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = tile * TILE + m.row(i0 + i);
          dy[i] = r < a.rows ? *reinterpret_cast<const float4*>(a.dy + (size_t)r * D + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = i0; i < i0 + 4; ++i) {
          const int r = tile * TILE + m.row(i);
          if (r >= a.rows) continue;
          const float* p = sums + m.row(i);
          const float iv = row_inv[m.row(i)], k = ((p[0] + p[TILE]) + (p[2 * TILE] + p[3 * TILE])) * iv * iv * iv * (1.0f / D);
          const float4 d = dy[i - i0];
          *reinterpret_cast<float4*>(a.out + (size_t)r * D + m.col) =
              make_float4(d.x + iv * gain.x * dn[i].x - x[i].x * k, d.y + iv * gain.y * dn[i].y - x[i].y * k,
                          d.z + iv * gain.z * dn[i].z - x[i].z * k, d.w + iv * gain.w * dn[i].w - x[i].w * k);
          gsum.x = fmaf(dn[i].x * x[i].x, iv, gsum.x); gsum.y = fmaf(dn[i].y * x[i].y, iv, gsum.y);
          gsum.z = fmaf(dn[i].z * x[i].z, iv, gsum.z); gsum.w = fmaf(dn[i].w * x[i].w, iv, gsum.w);
        }
      }
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      gsum.x += __shfl_xor_sync(0xffffffffu, gsum.x, o);
      gsum.y += __shfl_xor_sync(0xffffffffu, gsum.y, o);
      gsum.z += __shfl_xor_sync(0xffffffffu, gsum.z, o);
      gsum.w += __shfl_xor_sync(0xffffffffu, gsum.w, o);
    }
    if (m.lane < 8 && my_tiles > 0) atomicAdd(reinterpret_cast<float4*>(a.d_gain + m.col), gsum);
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  close_frame(f, tmem);
}

// ------------------------------------------------------------------ gradient of the weights

// Shared memory: the chunk's gate|up and transposed down (48 KB), two stages of n and dy tiles (64 KB),
// d gate | d up (32 KB) and h (16 KB) of a tile as operands, frame.
constexpr uint32_t DW_TILE = 49152, DW_G = DW_TILE + 2 * 65536, DW_H = DW_G + 32768, DW_FRAME = DW_H + 16384, DW_BYTES = DW_FRAME + FRAME_BYTES;
enum : int { WB_WEIGHTS = 0, WB_READY, WB_READ, WB_STAGED, WB_DRAIN, WB_FULL0, WB_DONE0 = WB_FULL0 + 4, WB_COUNT = WB_DONE0 + 4 };   // slots of n, then of dy
// Tensor memory: gate|up [0, 128), d h [128, 192), d Wg | d Wu (lane = hidden column) [192, 320), d Wd (lane =
// model dimension) [320, 384).
constexpr uint32_t DW_ACC1 = 192, DW_ACC2 = 320;

__global__ void __launch_bounds__(THREADS, 1) k_mlp_dw(const __grid_constant__ Args a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int counts[WB_COUNT] = {1, 1, EPI_WARPS, EPI_WARPS, 1, 1, 1, 1, 1, 1, 1, 1, 1};
  const int tid = threadIdx.x, warp = tid >> 5;
  const Frame f = open_frame(smem + DW_FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot;
  // CTAs of eight neighbouring indices share their row tiles (one chunk each): a tile comes from HBM once
  const int chunk = blockIdx.x & 7, first = blockIdx.x >> 3, stride = gridDim.x >> 3;
  const int my_tiles = first < a.tiles ? (a.tiles - first + stride - 1) / stride : 0;

  if (warp == LOAD_WARP) {
    const uint32_t base = smem_u32(smem);
    const bool elected = elect_one() != 0;
    if (elected) {
      mbar_expect_tx(s.bars + 8 * WB_WEIGHTS, 49152);
      bulk_g2s(base, a.image + (size_t)chunk * IMG_CHUNK + IMG_GU, 49152, s.bars + 8 * WB_WEIGHTS);
    }
    __syncwarp();
    uint32_t par = 3;
    // A tile's copies start when the products of the tile two before are complete and are waited for a period later: it is in
    // L2 by then, an eighth asked for by each CTA that reads it.
    auto ask = [&](int i) {
      if (i < my_tiles && elected) {
        const size_t at = (size_t)(first + i * stride) * 32768 + chunk * 4096;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.n_image + at), "r"(4096) : "memory");
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.dy_image + at), "r"(4096) : "memory");
      }
    };
    ask(2);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const uint32_t slot = i & 1;
      const size_t at = (size_t)(first + i * stride) * 32768;
      ask(i + 3);
      bool go = true;
#pragma unroll
      for (int p = 0; p < 2 && go; ++p)   // n, whose products are the first and the last that are waited for, then dy
        go = fetch(s, WB_FULL0 + 2 * p + slot, WB_DONE0 + 2 * p + slot, par >> slot, base + DW_TILE + slot * 65536 + p * 32768, (p ? a.dy_image : a.n_image) + at, 32768, elected);
      if (!go) break;
      par ^= 1u << slot;
    }
  } else if (warp == MMA_WARP) {
    const uint32_t base = smem_u32(smem), el = elect_one(), tm = uniform(tmem), w_lo = desc_lo(base);
    const uint32_t id128 = instr_desc(128), id64 = instr_desc(64);
    uint32_t full = 0;
    s.wait(WB_WEIGHTS, 0, TIMEOUT_FULL);
    auto recompute = [&](uint32_t slot) {
      s.wait(WB_FULL0 + slot, full >> slot, TIMEOUT_FULL);
      const uint32_t n_lo = uniform(desc_lo(base + DW_TILE + slot * 65536));
      product128(el, tm, n_lo, w_lo, 1024, id128);
      s.wait(WB_FULL0 + 2 + slot, full >> slot, TIMEOUT_FULL);
      full ^= 1u << slot;
      product128(el, tm + 128, n_lo + 2048, w_lo + 2048, 512, id64);
      tc_commit_if(el, s.bars + 8 * WB_READY);
    };
    if (my_tiles > 0) recompute(0);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const uint32_t slot = i & 1;
      s.wait(WB_READ, i, TIMEOUT_OPERAND);       // the epilogue has the accumulators in registers
      tc_fence_after();
      if (i + 1 < my_tiles) recompute(slot ^ 1);
      s.wait(WB_STAGED, i, TIMEOUT_OPERAND);
      tc_fence_after();
      const uint32_t n_mn = uniform(desc_mn(base + DW_TILE + slot * 65536)), g_mn = desc_mn(base + DW_G), h_mn = desc_mn(base + DW_H);
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k)           // 16 rows = 2048 bytes per k step
        mma_one<false>(el, tm + DW_ACC1, g_mn + 128 * k, n_mn + 128 * k, id128 | BOTH_MN, (i | (int)k) ? 1u : 0u);
      tc_commit_if(el, s.bars + 8 * (WB_DONE0 + slot));
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k)
        mma_one<false>(el, tm + DW_ACC2, n_mn + 2048 + 128 * k, h_mn + 128 * k, id64 | BOTH_MN, (i | (int)k) ? 1u : 0u);
      tc_commit_if(el, s.bars + 8 * (WB_DONE0 + 2 + slot));
    }
    tc_commit_if(el, s.bars + 8 * WB_DRAIN);
    for (int i = 0; i < DEFAULT_POLL_LIMIT && !mbar_try_wait(s.bars + 8 * WB_DRAIN, 0); ++i) {
    }
  } else {
    const int row = tid & (TILE - 1), part = tid >> 7;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t done = 0;
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      s.wait(WB_READY, i, TIMEOUT_ACC);
      tc_fence_after();
      uint32_t g[16], u[16], h[16];
      tmem_ld16_nowait(lane_addr + 16 * part, g);
      tmem_ld16_nowait(lane_addr + 64 + 16 * part, u);
      tmem_ld16_nowait(lane_addr + 128 + 16 * part, h);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(s.bars + 8 * WB_READ);
      uint32_t wg[8], wu[8], wh[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const F2 x = acc_pair(&g[2 * j]), up = acc_pair(&u[2 * j]), dh = acc_pair(&h[2 * j]);
        F2 e;
        const F2 cdf = normal_cdf(x, e), y = mul(x, cdf);
        wg[j] = pack_f2(mul(mul(dh, up), fma(mul(x, f2(0.39894228f)), e, cdf)));
        wu[j] = pack_f2(mul(dh, y));
        wh[j] = pack_f2(mul(y, up));
      }
      if (i > 0) {   // the previous tile's operands have been read
        s.wait(WB_DONE0 + 2 + ((i - 1) & 1), done >> ((i - 1) & 1), TIMEOUT_ACC);
        done ^= 1u << ((i - 1) & 1);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t at = swz(row, part * 2 + q);
        *reinterpret_cast<uint4*>(smem + DW_G + at) = make_uint4(wg[4 * q], wg[4 * q + 1], wg[4 * q + 2], wg[4 * q + 3]);
        *reinterpret_cast<uint4*>(smem + DW_G + CHUNK_BYTES + at) = make_uint4(wu[4 * q], wu[4 * q + 1], wu[4 * q + 2], wu[4 * q + 3]);
        *reinterpret_cast<uint4*>(smem + DW_H + at) = make_uint4(wh[4 * q], wh[4 * q + 1], wh[4 * q + 2], wh[4 * q + 3]);
      }
      post(s, WB_STAGED);
    }
    if (my_tiles > 0) {
      s.wait(WB_DONE0 + 2 + ((my_tiles - 1) & 1), done >> ((my_tiles - 1) & 1), TIMEOUT_ACC);
      tc_fence_after();
      // lanes 0 - 63: d Wg rows, 64 - 127: d Wu rows of the chunk; this thread: 32 of the 128 columns
      float* dst = (row < 64 ? a.d_gate + (size_t)(64 * chunk + row) * D : a.d_up + (size_t)(64 * chunk + row - 64) * D) + part * 32;
      uint32_t v[32];
      tmem_ld32(lane_addr + DW_ACC1 + part * 32, v);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        atomicAdd(reinterpret_cast<float4*>(dst + 4 * q), make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                                     __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3])));
      uint32_t w[16];
      tmem_ld16_nowait(lane_addr + DW_ACC2 + part * 16, w);
      tmem_wait_ld();
      float* dd = a.d_down + (size_t)row * F + 64 * chunk + part * 16;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        atomicAdd(reinterpret_cast<float4*>(dd + 4 * q), make_float4(__uint_as_float(w[4 * q]), __uint_as_float(w[4 * q + 1]),
                                                                    __uint_as_float(w[4 * q + 2]), __uint_as_float(w[4 * q + 3])));
    }
  }
  close_frame(f, tmem);
}

// ------------------------------------------------------------------ host side

template <typename K>
bool opt_in(K kernel, uint32_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}
bool configure() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!done[dev]) done[dev] = opt_in(k_mlp_fwd, FW_BYTES) && opt_in(k_mlp_dx, DX_BYTES) && opt_in(k_mlp_dw, DW_BYTES);
  return done[dev];
}
int launched() { return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH; }

}  // namespace

size_t image_bytes() { return IMAGE; }
size_t rows_image_bytes(size_t rows) { return (rows + TILE - 1) / TILE * 32768; }

int pack(const Weights* w, int n, uint8_t* image, cudaStream_t st) {
  for (int i0 = 0; i0 < n; i0 += MAX_JOBS) {
    PackJobs jobs{};
    const int m = n - i0 < MAX_JOBS ? n - i0 : MAX_JOBS;
    for (int i = 0; i < m; ++i) jobs.w[i] = w[i0 + i];
    count_launch();
    k_pack<<<dim3(48, m), 256, 0, st>>>(jobs, image + (size_t)i0 * IMAGE);
  }
  return launched();
}

int forward(const float* x1, const float* gain, const uint8_t* image, float* y, size_t rows, int* status, cudaStream_t st) {
  if (rows == 0) return BNB_OK;
  if (!configure()) return BNB_ERR_LAUNCH;
  Args a{};
  a.x1 = x1; a.gain = gain; a.image = image; a.out = y;
  a.rows = (int)rows;
  a.tiles = (int)((rows + TILE - 1) / TILE);
  a.status = status;
  a.host_status = tensor::host_status_word(st);
  return launch_after(k_mlp_fwd, dim3(a.tiles < 148 ? a.tiles : 148), THREADS, FW_BYTES, st, a);
}

int backward(const float* x1, const float* gain, const uint8_t* image, const float* dy, float* dx1, float* d_gain, float* d_gate,
             float* d_up, float* d_down, uint8_t* n_image, uint8_t* dy_image, size_t rows, int* status, cudaStream_t st) {
  if (rows == 0) return BNB_OK;
  if (!configure()) return BNB_ERR_LAUNCH;
  Args a{};
  a.x1 = x1; a.dy = dy; a.gain = gain; a.d_gain = d_gain; a.image = image; a.out = dx1;
  a.n_image = n_image; a.dy_image = dy_image;
  a.d_gate = d_gate; a.d_up = d_up; a.d_down = d_down;
  a.rows = (int)rows;
  a.tiles = (int)((rows + TILE - 1) / TILE);
  a.status = status;
  a.host_status = tensor::host_status_word(st);
  if (const int rc = launch_after(k_mlp_dx, dim3(a.tiles < 148 ? a.tiles : 148), THREADS, DX_BYTES, st, a)) return rc;
  const int groups = a.tiles < 18 ? a.tiles : 18;   // 18 CTAs per chunk: 144 of the 148 SMs
  return launch_after(k_mlp_dw, dim3(8 * groups), THREADS, DW_BYTES, st, a);
}

}  // namespace train_mlp
}  // namespace bnb
