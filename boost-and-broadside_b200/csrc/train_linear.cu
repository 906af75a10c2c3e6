// Linear layers of the training path, d_model 128, bfloat16 operands and float32 accumulation (what autocast does
// to the reference's Linears and their backward; models/yemong/attention.py:76-169, griffin.py:249-317).
//
// With 128-wide rows the floor of these layers is memory: a row tile costs 64 KB per float32 tensor it touches and half
// a thousand cycles of tensor pipe per product.  So what shares rows shares a pass:
//
//   k_linear_fwd   norm (its result written once, as bfloat16) and up to three layers of it
//   k_linear_bwd   gradient with respect to the input and the weights of up to three layers from one reading of
//                  their dy, bias gradients as column sums on the way, and the norm's gradient as the epilogue
//
// Persistent CTAs, one per SM: the weights stay in shared memory, row tiles of 128 pass by.  Rows are on their way in
// registers (64 KB per SM) while the tile before is worked on.  The weight images are plain K-major tiles; backward
// reads them as MN-major operands (dn = dy W needs W's other direction), and dy and n as MN-major operands for
// d W = dy^T n, whose accumulator stays in tensor memory over all tiles of a CTA.
//
// 262 144 rows: forward and backward of a temporal sublayer's Linears and norm took 13 launches of mma.sync
// products, each reading and writing its operands for itself.
//
// What bounds them now is the latency of the row loads, not the copy rate: for 65 536 rows the forward of three layers
// takes 38 us at 30 % of DRAM's peak and of one layer 24 us at 36 %, the backward of one layer 36 us at 24 %, of two gates
// 59 us at 31 %, of two layers with their norm 83 us at 26 %; 14 to 20 of 25 to 30 cycles between two issues of a warp are
// waits for global and tensor memory, because a tile's tensors are requested one after the other into registers.
#include "train_linear.h"

#include "launch_after.h"
#include "tensor_kernels.h"
#include "tile_rows.cuh"

namespace bnb {
namespace train_linear {

using namespace tensor;

namespace {

constexpr uint32_t TILE_BYTES = 32768;   // 128 x 128 bfloat16

constexpr int MAX_PACK = 64;
struct PackJobs { const float* src[MAX_PACK]; };
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackJobs jobs, uint8_t* image) {
  const float* src = jobs.src[blockIdx.y];
  uint8_t* out = image + (size_t)blockIdx.y * BLOCK_IMAGE;
  const int i = blockIdx.x * blockDim.x + threadIdx.x, r = i >> 4, g = i & 15;   // eight columns per thread
  const float4 a = *reinterpret_cast<const float4*>(src + r * D + 8 * g), b = *reinterpret_cast<const float4*>(src + r * D + 8 * g + 4);
  *reinterpret_cast<uint4*>(out + (g >> 3) * CHUNK_BYTES + swz(r, g & 7)) =
      make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void store4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void put_row4(uint8_t* tile, int row, int col, const float4& v) { put4(tile, row, col, v.x, v.y, v.z, v.w); }
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// ------------------------------------------------------------------ forward

struct FwdArgs {
  Forward f;
  int rows, tiles;
  int* status;
  int* host_status;
};
// Shared memory: weights, two operand tiles, transposing stages (4 KB per warp), row sums, frame.
template <int NB> struct FwdMap {
  static constexpr uint32_t A = NB * TILE_BYTES, STAGE = A + (NB == 3 ? 1 : 2) * TILE_BYTES, SUMS = STAGE + 65536, FRAME = SUMS + 2048,
                            BYTES = FRAME + FRAME_BYTES;
};
// An operand and an accumulator barrier per accumulator set: the epilogue runs a tile behind, and a phase must not be
// overtaken before it has been waited for.
enum : int { F_W = 0, F_OP0, F_ACC0 = F_OP0 + 2, F_COUNT = F_ACC0 + 2 };

// Up to two blocks, the products of a tile run while the tile before is written out (two accumulator sets); three
// blocks fill tensor memory with one set.
template <int NB>
__global__ void __launch_bounds__(THREADS, 1) k_linear_fwd(const __grid_constant__ FwdArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using Map = FwdMap<NB>;
  constexpr bool LAG = NB < 3;
  const int counts[F_COUNT] = {1, EPI_WARPS, EPI_WARPS, 1, 1};
  const Frame f = open_frame(smem + Map::FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot, base = smem_u32(smem);
  const int warp = threadIdx.x >> 5;
  auto set_of = [](int i) { return LAG ? i & 1 : 0; };
  auto phase_of = [](int i) { return (uint32_t)(LAG ? i >> 1 : i); };
  const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  if (warp == LOAD_WARP) {
    if (elect_one()) {
      mbar_expect_tx(s.bars + 8 * F_W, NB * TILE_BYTES);
      for (int b = 0; b < NB; ++b) bulk_g2s(base + b * TILE_BYTES, a.f.image + (size_t)b * BLOCK_IMAGE, TILE_BYTES, s.bars + 8 * F_W);
    }
    __syncwarp();
    s.wait(F_W, 0, TIMEOUT_FULL);
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(tmem), w_lo = desc_lo(base), idesc = instr_desc(128);
    s.wait(F_W, 0, TIMEOUT_FULL);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const uint32_t set = set_of(i);
      s.wait(F_OP0 + set, phase_of(i), TIMEOUT_OPERAND);
      tc_fence_after();
      const uint32_t a_lo = uniform(desc_lo(base + Map::A + set * TILE_BYTES));
#pragma unroll
      for (uint32_t b = 0; b < NB; ++b) product128(el, tm + set * (NB * 128) + 128 * b, a_lo, w_lo + (TILE_BYTES >> 4) * b, 1024, idesc);
      tc_commit_if(el, s.bars + 8 * (F_ACC0 + set));
    }
    if (my_tiles > 0) s.wait(F_ACC0 + set_of(my_tiles - 1), phase_of(my_tiles - 1), TIMEOUT_ACC);
  } else {
    const RowMap m = row_map();
    const int part = warp >> 2;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* stage = smem + Map::STAGE + warp * 4096;
    const bool normed = a.f.gain != nullptr;
    const float4 gain = normed ? load4(a.f.gain + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
    auto finish = [&](int i) {   // the accumulators of the i-th tile to memory
      const int first = (blockIdx.x + i * gridDim.x) * TILE;
      s.wait(F_ACC0 + set_of(i), phase_of(i), TIMEOUT_ACC);
      tc_fence_after();
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float4 extra[8];
        const float4 bias = a.f.bias[b] ? load4(a.f.bias[b] + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (NB == 1 && a.f.residual) rows_in(extra, a.f.residual, m, first, a.rows);
        __syncwarp();
        stage_rows(lane_addr + set_of(i) * (NB * 128) + 128 * b + part * 32, stage, m.lane);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = first + m.row(k);
          if (r >= a.rows) continue;
          float4 v = add4(staged_row(stage, k, m.lane), bias);
          if (NB == 1 && a.f.residual) v = add4(v, extra[k]);
          store4(a.f.out[b] + (size_t)r * a.f.ld_out + m.col, v);
        }
      }
      tc_fence_before();
    };
    float4 x[8];
    if (my_tiles > 0) rows_in(x, a.f.x, m, blockIdx.x * TILE, a.rows);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const int first = (blockIdx.x + i * gridDim.x) * TILE;
      uint8_t* tile = smem + Map::A + set_of(i) * TILE_BYTES;
      if (normed) {
        float inv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) inv[k] = fmaf(x[k].x, x[k].x, fmaf(x[k].y, x[k].y, fmaf(x[k].z, x[k].z, x[k].w * x[k].w)));
        row_sums(inv, reinterpret_cast<float*>(smem + Map::SUMS), m);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          inv[k] = rsqrtf(inv[k] / (float)D + kRmsEps);
          const uint2 n = make_uint2(pack_bf16(x[k].x * inv[k] * gain.x, x[k].y * inv[k] * gain.y), pack_bf16(x[k].z * inv[k] * gain.z, x[k].w * inv[k] * gain.w));
          *reinterpret_cast<uint2*>(tile + (m.col >> 6) * CHUNK_BYTES + swz(m.row(k), (m.col & 63) >> 3) + ((m.col >> 2) & 1) * 8) = n;
          const int r = first + m.row(k);
          if (r >= a.rows) continue;
          *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.f.n_out) + (size_t)r * D + m.col) = n;
          if (m.col == 0) a.f.inv[r] = inv[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) put_row4(tile, m.row(k), m.col, x[k]);
      }
      post(s, F_OP0 + set_of(i));
      if (i + 1 < my_tiles) rows_in(x, a.f.x, m, (blockIdx.x + (i + 1) * gridDim.x) * TILE, a.rows);
      if (!LAG) finish(i);
      else if (i > 0) finish(i - 1);
    }
    if (LAG && my_tiles > 0) finish(my_tiles - 1);
  }
  close_frame(f, tmem);
}

// ------------------------------------------------------------------ backward

struct BwdArgs {
  Backward b;
  int rows, tiles;
  int* status;
  int* host_status;
};
// Shared memory: weights, two dy tiles, one n tile, transposing stages (2 KB per warp: 16 columns), row sums, frame.
template <int NB> struct BwdMap {
  static constexpr uint32_t DY = NB * TILE_BYTES, N = DY + 2 * TILE_BYTES, STAGE = N + TILE_BYTES, SUMS = STAGE + 32768, FRAME = SUMS + 2048,
                            BYTES = FRAME + FRAME_BYTES;
};
enum : int { G_W = 0, G_OP0, G_ACC = G_OP0 + 2, G_FREE0, G_COUNT = G_FREE0 + 2 };   // operand and slot barriers per dy tile

// Sixteen accumulator columns of 32 rows into the row layout: lane l of the i-th request (i < 8) holds columns
// 4 (l % 8) .. of row 4 i + l / 8, so each half fills the lanes of its four column groups.
__device__ __forceinline__ void unstage(float4 (&v)[8], uint32_t taddr, uint8_t* stage, const RowMap& m) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t t[16];
    tmem_ld16_nowait(taddr + 16 * h, t);
    tmem_wait_ld();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(stage + m.lane * 64 + ((q ^ ((m.lane >> 1) & 3)) << 4)) = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
    __syncwarp();
    if (((m.lane >> 2) & 1) == h)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (m.lane >> 3);
        v[i] = *reinterpret_cast<const float4*>(stage + r * 64 + (((m.lane & 3) ^ ((r >> 1) & 3)) << 4));
      }
  }
}

// NB blocks; NORM: n is bfloat16 and dn goes through the norm's gradient; otherwise n is float32.
template <int NB, bool NORM>
__global__ void __launch_bounds__(THREADS, 1) k_linear_bwd(const __grid_constant__ BwdArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using Map = BwdMap<NB>;
  const int counts[G_COUNT] = {1, EPI_WARPS, EPI_WARPS, 1, 1, 1};
  const Frame f = open_frame(smem + Map::FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot, base = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  // tensor memory: d W of block b at 128 b, dn at 384
  if (warp == LOAD_WARP) {
    if (elect_one()) {
      mbar_expect_tx(s.bars + 8 * G_W, NB * TILE_BYTES);
      for (int b = 0; b < NB; ++b) bulk_g2s(base + b * TILE_BYTES, a.b.image + (size_t)b * BLOCK_IMAGE, TILE_BYTES, s.bars + 8 * G_W);
    }
    __syncwarp();
    s.wait(G_W, 0, TIMEOUT_FULL);
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(tmem), idesc = instr_desc(128);
    const uint32_t n_mn = desc_mn(base + Map::N);
    s.wait(G_W, 0, TIMEOUT_FULL);
    int item = 0;
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i)
#pragma unroll 1
      for (uint32_t b = 0; b < NB; ++b, ++item) {
        const uint32_t dy = base + Map::DY + (item & 1) * TILE_BYTES;
        s.wait(G_OP0 + (item & 1), item >> 1, TIMEOUT_OPERAND);
        tc_fence_after();
        const uint32_t dy_lo = uniform(desc_lo(dy)), dy_mn = uniform(desc_mn(dy)), w_mn = uniform(desc_mn(base + b * TILE_BYTES));
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)   // dn += dy W: K = the block's output features
          mma_one<false>(el, tm + 384, dy_lo + (k >> 2) * 1024 + 2 * (k & 3), w_mn + 128 * k, idesc | (1u << 16), (b | k) ? 1u : 0u);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)   // d W += dy^T n: K = rows
          mma_one<false>(el, tm + 128 * b, dy_mn + 128 * k, n_mn + 128 * k, idesc | BOTH_MN, (i | (int)k) ? 1u : 0u);
        tc_commit_if(el, s.bars + 8 * (G_FREE0 + (item & 1)));
        if (b == NB - 1) tc_commit_if(el, s.bars + 8 * G_ACC);
      }
    if (my_tiles > 0) s.wait(G_ACC, my_tiles - 1, TIMEOUT_ACC);
  } else {
    const RowMap m = row_map();
    const int part = warp >> 2;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* stage = smem + Map::STAGE + warp * 2048;
    float* sums = reinterpret_cast<float*>(smem + Map::SUMS);
    float4 gsum = make_float4(0.f, 0.f, 0.f, 0.f), bsum[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) bsum[b] = gsum;
    float4 dy[8];
    auto request = [&](int tile, const float* src) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = tile * TILE + m.row(k);
        dy[k] = r < a.rows ? load4(src + (size_t)r * a.b.ld_dy + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    if (my_tiles > 0) request(blockIdx.x, a.b.dy[0]);
    int item = 0;
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, first = tile * TILE;
      // One layer: the next tile's rows on their way to L2 (98 -> 90 us; the kernels with more registers in use lost 10 %).
      if (NB == 1 && tid == 0) {
        prefetch_rows(a.b.dy[0], tile + gridDim.x, a.rows, D * 4);
        prefetch_rows(a.b.n, tile + gridDim.x, a.rows, D * 4);
        if (a.b.accumulate) prefetch_rows(a.b.dx, tile + gridDim.x, a.rows, D * 4);
      }
#pragma unroll
      for (int b = 0; b < NB; ++b, ++item) {
        if (b == 0) {   // n of the tile; the products of the tile before are complete
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int r = first + m.row(k);
            if constexpr (NORM) {
              const uint2 v = r < a.rows ? *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(a.b.n) + (size_t)r * D + m.col) : make_uint2(0u, 0u);
              *reinterpret_cast<uint2*>(smem + Map::N + (m.col >> 6) * CHUNK_BYTES + swz(m.row(k), (m.col & 63) >> 3) + ((m.col >> 2) & 1) * 8) = v;
            } else {
              put_row4(smem + Map::N, m.row(k), m.col,
                       r < a.rows ? load4(static_cast<const float*>(a.b.n) + (size_t)r * D + m.col) : make_float4(0.f, 0.f, 0.f, 0.f));
            }
          }
        }
        if (item >= 2) s.wait(G_FREE0 + (item & 1), (item >> 1) - 1, TIMEOUT_FREE);
        uint8_t* at = smem + Map::DY + (item & 1) * TILE_BYTES;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          put_row4(at, m.row(k), m.col, dy[k]);
          if (!NORM) bsum[b] = add4(bsum[b], dy[k]);
        }
        post(s, G_OP0 + (item & 1));
        if (b + 1 < NB) request(tile, a.b.dy[b + 1]);
        else if (!NORM && i + 1 < my_tiles) request(tile + gridDim.x, a.b.dy[0]);
      }
      float4 x[8], dn[8];
      float iv[8];
      if constexpr (NORM) {
        rows_in(x, a.b.x, m, first, a.rows);
#pragma unroll
        for (int k = 0; k < 8; ++k) iv[k] = first + m.row(k) < a.rows ? a.b.inv[first + m.row(k)] : 0.f;
      }
      s.wait(G_ACC, i, TIMEOUT_ACC);
      tc_fence_after();
      unstage(dn, lane_addr + 384 + part * 32, stage, m);
      tc_fence_before();
      if constexpr (NORM) {
        const float4 gain = load4(a.b.gain + m.col);
        float coef[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          coef[k] = fmaf(x[k].x * gain.x, dn[k].x, fmaf(x[k].y * gain.y, dn[k].y, fmaf(x[k].z * gain.z, dn[k].z, x[k].w * gain.w * dn[k].w)));
        row_sums(coef, sums, m);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = first + m.row(k);
          if (r >= a.rows) continue;
          const float v = iv[k], c = coef[k] * v * v * v * (1.0f / D);
          float4 d = a.b.dres ? load4(a.b.dres + (size_t)r * D + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
          d.x += v * gain.x * dn[k].x - x[k].x * c; d.y += v * gain.y * dn[k].y - x[k].y * c;
          d.z += v * gain.z * dn[k].z - x[k].z * c; d.w += v * gain.w * dn[k].w - x[k].w * c;
          store4(a.b.dx + (size_t)r * D + m.col, d);
          gsum.x = fmaf(dn[k].x * x[k].x, v, gsum.x); gsum.y = fmaf(dn[k].y * x[k].y, v, gsum.y);
          gsum.z = fmaf(dn[k].z * x[k].z, v, gsum.z); gsum.w = fmaf(dn[k].w * x[k].w, v, gsum.w);
        }
        if (i + 1 < my_tiles) request(tile + gridDim.x, a.b.dy[0]);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = first + m.row(k);
          if (r >= a.rows) continue;
          float* p = a.b.dx + (size_t)r * D + m.col;
          store4(p, a.b.accumulate ? add4(load4(p), dn[k]) : dn[k]);
        }
      }
    }
    if (my_tiles > 0) {
      // d W: lane = output feature, this thread 32 of its 128 columns
      const int row = tid & (TILE - 1);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        uint32_t v[32];
        tmem_ld32(lane_addr + 128 * b + part * 32, v);
        float* dst = a.b.d_weight[b] + (size_t)row * D + part * 32;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          atomicAdd(reinterpret_cast<float4*>(dst + 4 * q), make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                                       __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3])));
      }
      auto column_sum = [&](float4 v, float* dst) {   // over the rows of the warp, then of the grid
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
          v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
          v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
          v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
          v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
        }
        if (m.lane < 8) atomicAdd(reinterpret_cast<float4*>(dst + m.col), v);
      };
      if (NORM) column_sum(gsum, a.b.d_gain);
#pragma unroll
      for (int b = 0; b < NB; ++b)
        if (!NORM && a.b.d_bias[b]) column_sum(bsum[b], a.b.d_bias[b]);
    }
  }
  close_frame(f, tmem);
}

// ------------------------------------------------------------------ host side

int launched() { return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH; }
int grid_of(int tiles) { return tiles < 148 ? tiles : 148; }

template <class K>
bool opt_in(K kernel, uint32_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}
bool configure() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!done[dev])
    done[dev] = opt_in(k_linear_fwd<1>, FwdMap<1>::BYTES) && opt_in(k_linear_fwd<2>, FwdMap<2>::BYTES) && opt_in(k_linear_fwd<3>, FwdMap<3>::BYTES) &&
                opt_in(k_linear_bwd<1, false>, BwdMap<1>::BYTES) && opt_in(k_linear_bwd<2, false>, BwdMap<2>::BYTES) &&
                opt_in(k_linear_bwd<2, true>, BwdMap<2>::BYTES) && opt_in(k_linear_bwd<3, true>, BwdMap<3>::BYTES);
  return done[dev];
}

}  // namespace

int pack(const float* const* blocks, int n, uint8_t* image, cudaStream_t st) {
  for (int i0 = 0; i0 < n; i0 += MAX_PACK) {
    PackJobs jobs{};
    const int m = n - i0 < MAX_PACK ? n - i0 : MAX_PACK;
    for (int i = 0; i < m; ++i) jobs.src[i] = blocks[i0 + i];
    count_launch();
    k_pack<<<dim3(8, m), 256, 0, st>>>(jobs, image + (size_t)i0 * BLOCK_IMAGE);
  }
  return launched();
}

int forward(const Forward& f, int* status, cudaStream_t st) {
  if (f.rows == 0) return BNB_OK;
  if (!configure()) return BNB_ERR_LAUNCH;
  const int tiles = (int)((f.rows + TILE - 1) / TILE);
  const FwdArgs a{f, (int)f.rows, tiles, status, tensor::host_status_word(st)};
  const dim3 grid(grid_of(tiles));
  return f.blocks == 1   ? launch_after(k_linear_fwd<1>, grid, THREADS, FwdMap<1>::BYTES, st, a)
         : f.blocks == 2 ? launch_after(k_linear_fwd<2>, grid, THREADS, FwdMap<2>::BYTES, st, a)
                         : launch_after(k_linear_fwd<3>, grid, THREADS, FwdMap<3>::BYTES, st, a);
}

int backward(const Backward& b, int* status, cudaStream_t st) {
  if (b.rows == 0) return BNB_OK;
  if (!configure()) return BNB_ERR_LAUNCH;
  const int tiles = (int)((b.rows + TILE - 1) / TILE);
  const BwdArgs a{b, (int)b.rows, tiles, status, tensor::host_status_word(st)};
  const dim3 grid(grid_of(tiles));
  if (b.gain && b.blocks == 3) return launch_after(k_linear_bwd<3, true>, grid, THREADS, BwdMap<3>::BYTES, st, a);
  if (b.gain && b.blocks == 2) return launch_after(k_linear_bwd<2, true>, grid, THREADS, BwdMap<2>::BYTES, st, a);
  if (!b.gain && b.blocks == 2) return launch_after(k_linear_bwd<2, false>, grid, THREADS, BwdMap<2>::BYTES, st, a);
  if (!b.gain && b.blocks == 1) return launch_after(k_linear_bwd<1, false>, grid, THREADS, BwdMap<1>::BYTES, st, a);
  return BNB_ERR_BAD_ARGUMENT;
}

}  // namespace train_linear
}  // namespace bnb
