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
// Persistent CTAs, one per SM: the weights stay in shared memory, row tiles of 128 pass by.  The weight images are plain
// K-major tiles; backward reads them as MN-major operands (dn = dy W needs W's other direction), and dy and n as MN-major
// operands for d W = dy^T n, whose accumulator stays in tensor memory over all tiles of a CTA.
//
// 262 144 rows: forward and backward of a temporal sublayer's Linears and norm took 13 launches of mma.sync
// products, each reading and writing its operands for itself.
//
// What bounds them is memory: for 262 144 rows the forward of three layers takes 117 us (603 MB, 5.2 TB/s) and of one 71 (403 MB, 5.7),
// the backward of one layer 80 us (403 MB, 5.0), of two gates 111 (671 MB, 6.0), of two layers with their norm 157 (738 MB, 4.7), of
// three with theirs 191 (872 MB, 4.6).  Backward through registers, a tensor of a tile behind the other, took 91, 178, 263 and 326.
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
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// ------------------------------------------------------------------ forward

struct FwdArgs {
  Forward f;
  int rows;
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
  const int rows = a.f.count ? min(*a.f.count, a.rows) : a.rows, tiles = (rows + TILE - 1) / TILE;
  const int my_tiles = (int)blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
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
        if (NB == 1 && a.f.residual) rows_in(extra, a.f.residual, m, first, rows);
        __syncwarp();
        stage_rows(lane_addr + set_of(i) * (NB * 128) + 128 * b + part * 32, stage, m.lane);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = first + m.row(k);
          if (r >= rows) continue;
          float4 v = add4(staged_row(stage, k, m.lane), bias);
          if (NB == 1 && a.f.residual) v = add4(v, extra[k]);
          store4(a.f.out[b] + (size_t)r * a.f.ld_out + m.col, v);
        }
      }
      tc_fence_before();
    };
    float4 x[8];
    if (my_tiles > 0) rows_in(x, a.f.x, m, blockIdx.x * TILE, rows);
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
          *reinterpret_cast<uint2*>(tile + (m.col >> 6) * CHUNK_BYTES + row_swz(m, k, (m.col & 63) >> 3) + ((m.col >> 2) & 1) * 8) = n;
          const int r = first + m.row(k);
          if (r >= rows) continue;
          *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.f.n_out) + (size_t)r * D + m.col) = n;
          if (m.col == 0) a.f.inv[r] = inv[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) put_row4(tile, m, k, x[k]);
      }
      post(s, F_OP0 + set_of(i));
      if (i + 1 < my_tiles) rows_in(x, a.f.x, m, (blockIdx.x + (i + 1) * gridDim.x) * TILE, rows);
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
  int rows;
  int* status;
  int* host_status;
};
// Shared memory: weights, the operand tiles of dy and n, float32 rows on their way, row sums, frame.  The rows: pieces of
// 16 rows (8 KB), SLOTS of them for each group of four warps, which reads 32 rows of a tile.
constexpr int PIECE_ROWS = 16, PIECE_BYTES = PIECE_ROWS * D * 4;
template <int NB> struct BwdMap {
  static constexpr int SLOTS = NB == 3 ? 2 : 3;
  static constexpr uint32_t DY = NB * TILE_BYTES, N = DY + TILE_BYTES, RAW = N + TILE_BYTES, SUMS = RAW + 4 * SLOTS * PIECE_BYTES, FRAME = SUMS + 2048,
                            BYTES = FRAME + FRAME_BYTES;
  static constexpr int FREE = 3 + 4 * SLOTS, COUNT = FREE + 4 * SLOTS;   // barriers behind G_FULL
};
enum : int { G_W = 0, G_OP, G_DONE, G_FULL };   // weights, dy tile written, its products complete, pieces

// Sixteen accumulator columns of 32 rows at a time into the row layout: lane l of the i-th request (i < 8) holds columns
// 4 (l % 8) .. of row 4 i + l / 8, so each half fills the lanes of its four column groups.  Through the memory that only
// this warp writes of the dy tile (64 bytes of its 32 rows).  ADD: onto what v holds.
template <bool ADD>
__device__ __forceinline__ void unstage(float4 (&v)[8], uint32_t taddr, uint8_t* dy_tile, const RowMap& m) {
  const int part = threadIdx.x >> 7;
  uint8_t* stage = dy_tile + (part >> 1) * CHUNK_BYTES;
  const int g0 = 4 * (part & 1);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t t[16];
    tmem_ld16_nowait(taddr + 16 * h, t);
    tmem_wait_ld();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(stage + swz(m.row0 + m.lane, g0 + q)) = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
    __syncwarp();
    if (((m.lane >> 2) & 1) == h)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 t4 = *reinterpret_cast<const float4*>(stage + row_swz(m, i, g0 + (m.lane & 3)));
        v[i] = ADD ? add4(v[i], t4) : t4;
      }
  }
  __syncwarp();
}

// NB blocks; NORM: n is bfloat16 and dn goes through the norm's gradient; otherwise n is float32.
//
// The fetching warp keeps the float32 rows of everything a tile reads on their way through shared memory, piece by piece, in the
// order of their use: of dy0 .. dy(NB - 1), x, d residual with norm, of n, dy0 .. , dx before without.  A tile of three layers
// with norm took 41 000 cycles with its loads one behind the other (d residual row by row between the stores), 31 000 with
// loads into registers two tensors ahead, and takes 27 000 of which 17 000 are waits for pieces (416 KB: 19 000 at the copy
// rate).  Every tensor is rows of 128 floats one behind the other: d q | d k | d v side by side in rows of 384 came as 512-byte
// copies, 45 cycles each (39 000 cycles a tile).
template <int NB, bool NORM>
__global__ void __launch_bounds__(THREADS, 1) k_linear_bwd(const __grid_constant__ BwdArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using Map = BwdMap<NB>;
  int counts[Map::COUNT];
#pragma unroll
  for (int i = 0; i < Map::COUNT; ++i) counts[i] = i == G_OP ? EPI_WARPS : i >= Map::FREE ? 4 : 1;
  const Frame f = open_frame(smem + Map::FRAME, a.status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), a.status, f.aborted};
  const uint32_t tmem = *f.tmem_slot, base = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int rows = a.b.count ? min(*a.b.count, a.rows) : a.rows, tiles = (rows + TILE - 1) / TILE;
  const int my_tiles = (int)blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  // tensor memory: d W of block b at 128 b, dn at 384
  if (warp == LOAD_WARP) {
    if (elect_one()) {
      mbar_expect_tx(s.bars + 8 * G_W, NB * TILE_BYTES);
      for (int b = 0; b < NB; ++b) bulk_g2s(base + b * TILE_BYTES, a.b.image + (size_t)b * BLOCK_IMAGE, TILE_BYTES, s.bars + 8 * G_W);
    }
    __syncwarp();
    // eight lanes for each group's pieces
    const int group = (tid & 31) >> 3, sub = tid & 7;
    int slot = 0;
    uint32_t free_parity = 1;   // a fresh barrier passes a wait on parity 1
    auto stream = [&](int tile, const float* src) {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const int bar = group * Map::SLOTS + slot, row = tile * TILE + 32 * group + PIECE_ROWS * h;
        const int n = min(max(rows - row, 0), PIECE_ROWS);
        const uint32_t full = s.bars + 8 * (G_FULL + bar);
        s.wait(Map::FREE + bar, free_parity, TIMEOUT_FREE);
        if (__any_sync(0xffffffffu, s.aborted[0])) return false;
        if (sub == 0) {
          mbar_expect_tx(full, n * D * 4);
          if (n > 0) bulk_g2s(base + Map::RAW + bar * PIECE_BYTES, src + (size_t)row * D, n * D * 4, full);
        }
        __syncwarp();
        if (++slot == Map::SLOTS) { slot = 0; free_parity ^= 1u; }
      }
      return true;
    };
    bool go = true;
#pragma unroll 1
    for (int i = 0; i < my_tiles && go; ++i) {
      const int tile = blockIdx.x + i * gridDim.x;
      if (!NORM) go = stream(tile, static_cast<const float*>(a.b.n));
#pragma unroll 1
      for (int b = 0; b < NB && go; ++b) go = stream(tile, a.b.dy[b]);
      if (NORM && go) go = stream(tile, a.b.x);
      const float* last = NORM ? a.b.dres : a.b.accumulate ? a.b.dx : nullptr;
      if (last && go) go = stream(tile, last);
    }
    s.wait(G_W, 0, TIMEOUT_FULL);
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(tmem), idesc = instr_desc(128);
    const uint32_t n_mn = desc_mn(base + Map::N), dy_lo = desc_lo(base + Map::DY), dy_mn = desc_mn(base + Map::DY);
    s.wait(G_W, 0, TIMEOUT_FULL);
    uint32_t item = 0;
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i)
#pragma unroll 1
      for (uint32_t b = 0; b < NB; ++b, ++item) {
        s.wait(G_OP, item, TIMEOUT_OPERAND);
        tc_fence_after();
        const uint32_t w_mn = uniform(desc_mn(base + b * TILE_BYTES));
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)   // dn += dy W: K = the block's output features
          mma_one<false>(el, tm + 384, dy_lo + (k >> 2) * 1024 + 2 * (k & 3), w_mn + 128 * k, idesc | (1u << 16), (b | k) ? 1u : 0u);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)   // d W += dy^T n: K = rows
          mma_one<false>(el, tm + 128 * b, dy_mn + 128 * k, n_mn + 128 * k, idesc | BOTH_MN, (i | (int)k) ? 1u : 0u);
        tc_commit_if(el, s.bars + 8 * G_DONE);
      }
    if (item > 0) s.wait(G_DONE, item - 1, TIMEOUT_ACC);
  } else {
    const RowMap m = row_map();
    const int part = warp >> 2, group = warp & 3;
    const uint32_t lane_addr = tmem + ((uint32_t)(group * 32) << 16);
    float* sums = reinterpret_cast<float*>(smem + Map::SUMS);
    float4 gsum = make_float4(0.f, 0.f, 0.f, 0.f), bsum[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) bsum[b] = gsum;
    int slot = 0;
    uint32_t parity = 0, item = 0;
    // The next piece of this group, used by four calls of `row` with its place in the tile and this lane's columns there.
    auto piece = [&](int first, int h, auto row) {
      const int bar = group * Map::SLOTS + slot;
      s.wait(G_FULL + bar, parity, TIMEOUT_FULL);
      const uint8_t* at = smem + Map::RAW + bar * PIECE_BYTES + (m.lane >> 3) * (D * 4) + m.col * 4;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 v = *reinterpret_cast<const float4*>(at + 4 * k * (D * 4));
        row(4 * h + k, first + m.row(4 * h + k) < rows ? v : make_float4(0.f, 0.f, 0.f, 0.f));
      }
      __syncwarp();
      if (m.lane == 0) mbar_arrive(s.bars + 8 * (Map::FREE + bar));
      if (++slot == Map::SLOTS) { slot = 0; parity ^= 1u; }
    };
    auto take = [&](float4 (&to)[8], int first) {
#pragma unroll
      for (int h = 0; h < 2; ++h) piece(first, h, [&](int k, const float4& v) { to[k] = v; });
    };
    // dy of block b as an operand; the products that read the tile before are complete
    auto place = [&](const float4 (&from)[8], int b) {
      if (b > 0) s.wait(G_DONE, item - 1, TIMEOUT_FREE);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        put_row4(smem + Map::DY, m, k, from[k]);
        if (!NORM) bsum[b] = add4(bsum[b], from[k]);
      }
      post(s, G_OP);
      ++item;
    };
    // bfloat16 n of a tile: this warp's 32 rows of 64 bytes as they are, zeros past the last row
    auto copy_n = [&](int tile) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = m.row0 + 8 * k + (m.lane >> 2), r = tile * TILE + row, g = 4 * part + (m.lane & 3);
        const uint32_t dst = smem_u32(smem + Map::N + (part >> 1) * CHUNK_BYTES + swz(row, g & 7));
        const __nv_bfloat16* src = static_cast<const __nv_bfloat16*>(a.b.n) + (size_t)(r < rows ? r : 0) * D + 8 * g;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(r < rows ? 16 : 0) : "memory");
      }
    };
    const float4 gain = NORM ? load4(a.b.gain + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (NORM && my_tiles > 0) copy_n(blockIdx.x);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, first = tile * TILE;
      float4 u[8], v[8];
      float inv = 0.f;   // of the row that is this lane's among the warp's
      if (NORM && first + m.row0 + m.lane < rows) inv = a.b.inv[first + m.row0 + m.lane];
      take(u, first);
      if constexpr (NORM) {
        asm volatile("cp.async.wait_all;" ::: "memory");   // n
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) put_row4(smem + Map::N, m, k, u[k]);   // the products of the tile before are complete
        take(u, first);
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        place(u, b);
        if (b + 1 < NB) take(u, first);
      }
      if constexpr (NORM) {
        take(v, first);   // x
        s.wait(G_DONE, item - 1, TIMEOUT_ACC);
        tc_fence_after();
        if (i + 1 < my_tiles) copy_n(tile + gridDim.x);
        unstage<false>(u, lane_addr + 384 + part * 32, smem + Map::DY, m);
        tc_fence_before();
#pragma unroll
        for (int k = 0; k < 8; ++k) {   // sums of x gain dn over a row: eight lanes here, the four warps of the row through shared memory
          float c = fmaf(v[k].x * gain.x, u[k].x, fmaf(v[k].y * gain.y, u[k].y, fmaf(v[k].z * gain.z, u[k].z, v[k].w * gain.w * u[k].w)));
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
          if ((m.lane & 7) == 0) sums[part * TILE + m.row(k)] = c;
        }
        // its next use comes behind a wait for products that every warp of these rows has to post for
        asm volatile("bar.sync %0, 128;" ::"r"(3 + group) : "memory");
        auto out = [&](int k, float4 d) {   // d: residual
          const int r = first + m.row(k);
          const float* p = sums + m.row(k);
          const float w = __shfl_sync(0xffffffffu, inv, 4 * k + (m.lane >> 3)), c = ((p[0] + p[TILE]) + (p[2 * TILE] + p[3 * TILE])) * w * w * w * (1.0f / D);
          if (r >= rows) return;
          d.x += w * gain.x * u[k].x - v[k].x * c; d.y += w * gain.y * u[k].y - v[k].y * c;
          d.z += w * gain.z * u[k].z - v[k].z * c; d.w += w * gain.w * u[k].w - v[k].w * c;
          store4(a.b.dx + (size_t)r * D + m.col, d);
          gsum.x = fmaf(u[k].x * v[k].x, w, gsum.x); gsum.y = fmaf(u[k].y * v[k].y, w, gsum.y);
          gsum.z = fmaf(u[k].z * v[k].z, w, gsum.z); gsum.w = fmaf(u[k].w * v[k].w, w, gsum.w);
        };
        if (a.b.dres) {
#pragma unroll
          for (int h = 0; h < 2; ++h) piece(first, h, out);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) out(k, make_float4(0.f, 0.f, 0.f, 0.f));
        }
      } else {
        if (a.b.accumulate) take(v, first);
        else
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        s.wait(G_DONE, item - 1, TIMEOUT_ACC);
        tc_fence_after();
        unstage<true>(v, lane_addr + 384 + part * 32, smem + Map::DY, m);
        tc_fence_before();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = first + m.row(k);
          if (r < rows) store4(a.b.dx + (size_t)r * D + m.col, v[k]);
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
  const FwdArgs a{f, (int)f.rows, status, tensor::host_status_word(st)};
  const dim3 grid(grid_of(tiles));
  return f.blocks == 1   ? launch_after(k_linear_fwd<1>, grid, THREADS, FwdMap<1>::BYTES, st, a)
         : f.blocks == 2 ? launch_after(k_linear_fwd<2>, grid, THREADS, FwdMap<2>::BYTES, st, a)
                         : launch_after(k_linear_fwd<3>, grid, THREADS, FwdMap<3>::BYTES, st, a);
}

int backward(const Backward& b, int* status, cudaStream_t st) {
  if (b.rows == 0) return BNB_OK;
  if (!configure()) return BNB_ERR_LAUNCH;
  const int tiles = (int)((b.rows + TILE - 1) / TILE);
  const BwdArgs a{b, (int)b.rows, status, tensor::host_status_word(st)};
  const dim3 grid(grid_of(tiles));
  if (b.gain && b.blocks == 3) return launch_after(k_linear_bwd<3, true>, grid, THREADS, BwdMap<3>::BYTES, st, a);
  if (b.gain && b.blocks == 2) return launch_after(k_linear_bwd<2, true>, grid, THREADS, BwdMap<2>::BYTES, st, a);
  if (!b.gain && b.blocks == 2) return launch_after(k_linear_bwd<2, false>, grid, THREADS, BwdMap<2>::BYTES, st, a);
  if (!b.gain && b.blocks == 1) return launch_after(k_linear_bwd<1, false>, grid, THREADS, BwdMap<1>::BYTES, st, a);
  return BNB_ERR_BAD_ARGUMENT;
}

}  // namespace train_linear
}  // namespace bnb
