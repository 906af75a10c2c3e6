// Keys and values of the bullet tokens under the bfloat16 contract: norm_bullet and kv_bullet of the rows in use,
// models/yemong/attention.py:149-166.
//
// Row tiles of 128 pass by persistent CTAs, one per SM, that keep the 64 KB of weights; the rows of the next tile are
// on their way while this one is normed and multiplied, and the result of the tile before is written out while the
// tensor cores work.  Bound by the rows' way through the SM: 256 or 512 bytes in (eight lines a request), 512 out: 33 us for
// the 147 000 active rows of 8192 environments of 80 bullets, with DRAM at 23 % of its peak, issue slots 27 % busy, the tensor
// pipe 16 %, and the stalls shared out between loads, the shared-memory port and its queue.
// As a program of a general tile kernel, with weights streamed per tile and a thread per row on the way in and out,
// it took 73 us for the active rows of 8192 environments of 80 bullets.
#include "bullet_kv.h"

#include "launch_after.h"
#include "tensor_kernels.h"
#include "tile_rows.cuh"

namespace bnb {
namespace tensor {

namespace {

struct KvArgs {
  const void* rows;        // (n_rows or more, 128), bfloat16 or float32
  const int* index;        // tile row r reads input row index[r], or null: r
  const int* n_rows_dev;   // number of rows on the device, or null: n_rows
  int n_rows;
  const uint8_t* image;    // keys, then values: 32 KB each
  __nv_bfloat16* out;      // (rows, 256)
  int* status;
  int* host_status;
};
constexpr uint32_t KV_A = 65536, KV_STAGE = KV_A + 65536, KV_SUMS = KV_STAGE + 32768, KV_FRAME = KV_SUMS + 4096, KV_BYTES = KV_FRAME + FRAME_BYTES;
// Operand and accumulator barriers per tile parity, so that no phase is overtaken before it has been waited for.
enum : int { V_W = 0, V_OP0, V_ACC0 = V_OP0 + 2, V_COUNT = V_ACC0 + 2 };

template <bool BF16>
__global__ void __launch_bounds__(THREADS, 1) k_bullet_kv(const __grid_constant__ KvArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int counts[V_COUNT] = {1, EPI_WARPS, EPI_WARPS, 1, 1};
  const Frame f = open_frame(smem + KV_FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot, base = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = a.n_rows_dev ? min(*a.n_rows_dev, a.n_rows) : a.n_rows, tiles = (rows + TILE - 1) / TILE;
  const int my_tiles = (int)blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  if (warp == LOAD_WARP) {
    if (elect_one()) {
      mbar_expect_tx(s.bars + 8 * V_W, 65536);
      bulk_g2s(base, a.image, 65536, s.bars + 8 * V_W);
    }
    __syncwarp();
    s.wait(V_W, 0, TIMEOUT_FULL);
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(tmem), w_lo = desc_lo(base), idesc = instr_desc(128);
    s.wait(V_W, 0, TIMEOUT_FULL);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const uint32_t set = i & 1;
      s.wait(V_OP0 + set, i >> 1, TIMEOUT_OPERAND);
      tc_fence_after();
      const uint32_t a_lo = uniform(desc_lo(base + KV_A + set * 32768));
      product128(el, tm + set * 256, a_lo, w_lo, 1024, idesc);
      product128(el, tm + set * 256 + 128, a_lo, w_lo + 2048, 1024, idesc);
      tc_commit_if(el, s.bars + 8 * (V_ACC0 + set));
    }
    for (int i = my_tiles - 2; i < my_tiles; ++i)
      if (i >= 0) s.wait(V_ACC0 + (i & 1), i >> 1, TIMEOUT_ACC);
  } else {
    const int part = warp >> 2, quarter = warp & 3;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const int row0 = 32 * quarter + (lane >> 2), col = 32 * part + 8 * (lane & 3);   // rows row0 + 8 k, eight columns
    uint8_t* stage = smem + KV_STAGE + warp * 2048;
    auto place = [&](int i, int k) {   // input row of the k-th row in the i-th tile, -1 past the end
      const int r = (blockIdx.x + i * gridDim.x) * TILE + row0 + 8 * k;
      return i < my_tiles && r < rows ? (a.index ? a.index[r] : r) : -1;
    };
    uint4 in[BF16 ? 4 : 8];
    auto request = [&](const int (&at)[4]) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (BF16) {
          in[k] = at[k] >= 0 ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.rows) + (size_t)at[k] * D + col) : make_uint4(0u, 0u, 0u, 0u);
        } else {
          const uint4* p = reinterpret_cast<const uint4*>(static_cast<const float*>(a.rows) + (size_t)at[k] * D + col);
          in[2 * k] = at[k] >= 0 ? p[0] : make_uint4(0u, 0u, 0u, 0u);
          in[2 * k + 1] = at[k] >= 0 ? p[1] : make_uint4(0u, 0u, 0u, 0u);
        }
      }
    };
    auto finish = [&](int i) {
      const int first = (blockIdx.x + i * gridDim.x) * TILE;
      s.wait(V_ACC0 + (i & 1), i >> 1, TIMEOUT_ACC);
      tc_fence_after();
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        uint32_t t[32];
        tmem_ld32(lane_addr + (i & 1) * 256 + 128 * b + 32 * part, t);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = pack_bf16(__uint_as_float(t[8 * q + 2 * j]), __uint_as_float(t[8 * q + 2 * j + 1]));
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int rr = (lane >> 2) + 8 * k, r = first + 32 * quarter + rr;
          if (r < rows)
            *reinterpret_cast<uint4*>(a.out + (size_t)r * 256 + 128 * b + col) =
                *reinterpret_cast<const uint4*>(stage + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
        }
      }
      tc_fence_before();
    };
    int at[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) at[k] = place(0, k);
    request(at);
#pragma unroll
    for (int k = 0; k < 4; ++k) at[k] = place(1, k);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      uint8_t* tile = smem + KV_A + (i & 1) * 32768;
      float* sums = reinterpret_cast<float*>(smem + KV_SUMS) + (i & 1) * 512 + row0;   // two buffers: one barrier a tile
      float x[4][8], ss[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (BF16) {
          const uint32_t w[4] = {in[k].x, in[k].y, in[k].z, in[k].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) { x[k][2 * j] = bf16_lo(w[j]); x[k][2 * j + 1] = bf16_hi(w[j]); }
        } else {
          const uint32_t w[8] = {in[2 * k].x, in[2 * k].y, in[2 * k].z, in[2 * k].w, in[2 * k + 1].x, in[2 * k + 1].y, in[2 * k + 1].z, in[2 * k + 1].w};
#pragma unroll
          for (int j = 0; j < 8; ++j) x[k][j] = __uint_as_float(w[j]);
        }
        ss[k] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[k] = fmaf(x[k][j], x[k][j], ss[k]);
        ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], 1);
        ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], 2);
        if ((lane & 3) == 0) sums[part * TILE + 8 * k] = ss[k];
      }
      asm volatile("bar.sync %0, 128;" ::"r"(3 + quarter) : "memory");
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float* p = sums + 8 * k;
        const float inv = rsqrtf(((p[0] + p[TILE]) + (p[2 * TILE] + p[3 * TILE])) * (1.0f / D) + kRmsEps);   // the gain is in the weights
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = pack_bf16(x[k][2 * j] * inv, x[k][2 * j + 1] * inv);
        *reinterpret_cast<uint4*>(tile + (col >> 6) * CHUNK_BYTES + swz(row0 + 8 * k, (col & 63) >> 3)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      post(s, V_OP0 + (i & 1));
      request(at);
#pragma unroll
      for (int k = 0; k < 4; ++k) at[k] = place(i + 2, k);
      if (i > 0) finish(i - 1);
    }
    if (my_tiles > 0) finish(my_tiles - 1);
  }
  close_frame(f, tmem);
}

}  // namespace

int bullet_kv(const void* rows, bool rows_bf16, int n_rows, const int* index, const int* n_rows_dev, const uint8_t* image, __nv_bfloat16* kvb,
              int* status, cudaStream_t st) {
  if (n_rows <= 0) return BNB_OK;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BNB_ERR_NO_DEVICE;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(k_bullet_kv<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KV_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(k_bullet_kv<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KV_BYTES) != cudaSuccess)
      return BNB_ERR_LAUNCH;
    configured[dev] = true;
  }
  const KvArgs a{rows, index, n_rows_dev, n_rows, image, kvb, status, host_status_word(st)};
  const int tiles = (n_rows + TILE - 1) / TILE, grid = tiles < 148 ? tiles : 148;
  return launch_after(rows_bf16 ? k_bullet_kv<true> : k_bullet_kv<false>, dim3(grid), THREADS, KV_BYTES, st, a);
}

}  // namespace tensor
}  // namespace bnb
