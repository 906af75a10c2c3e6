// The policy's MLPs with a hidden layer of 256 on tcgen05 tiles, bfloat16 contract, rounding where mlp_kernels.cu does (a
// Linear's output after its bias, a norm's result, the GELU's):
//
//   heads     Linear(128, 256) + b -> RMSNorm -> GELU -> Linear(256, out <= 32) + b          models/yemong/policy.py:185-214
//   encoder   Linear(in <= 128, 256) + b -> RMSNorm -> GELU -> Linear(256, 128) + b -> RMSNorm   models/yemong/encoder.py:45-102
//
// A CTA serves one chain and keeps its weights (80 or 128 KB as bfloat16 operands) in shared memory; row tiles of 128 pass by.
// The hidden layer never leaves tensor memory and registers: a thread takes 64 hidden columns of its row, four threads
// add up the row's squares, and the activations go back as the A operand of the second product over the columns they
// came from.  Tensor memory holds two tiles, so the first product of the next tile runs under this one's epilogue, which
// is the bound: about 12 instructions per hidden element, two elements at a time but for the row's squares (24 one by one: three heads of 65 536 rows
// and the win head's teams 78.2 -> 67.3 us, an encoder of 98 304 rows 66.3 -> 62.4; issue slots were 57 % busy, the tensor pipe 12 %, DRAM 3 % of
// peak, and the chain of a tile's phases is what is left; an encoder's rows come in element by element).  On mma.sync tiles of 16 rows, with
// the first product computed twice for the norm, three heads of 65 536 rows took 139 us, one of 16 384 rows 39 (14 here), one of 128 rows no less.
#include "head_tiles.h"

#include "launch_after.h"
#include "tensor_kernels.h"
#include "tile_rows.cuh"

namespace bnb {
namespace mlp {

using namespace tensor;

namespace {

constexpr int HIDDEN = 256;
// Shared memory: both weights in K atoms of 64, two operand tiles, b1 | g1 | b2 | g2, row sums of both norms, frame.
template <bool ENC> struct Map {
  static constexpr int OUT = ENC ? 128 : 32;
  static constexpr uint32_t W1_ATOM = HIDDEN * 128, W2_ATOM = OUT * 128, W2 = 2 * W1_ATOM, A = W2 + 4 * W2_ATOM, VEC = A + 65536,
                            SUMS = VEC + 4 * (2 * HIDDEN + 2 * OUT), FRAME = SUMS + 8192, STATUS = FRAME + FRAME_BYTES, BYTES = STATUS + 16;
  static_assert(A % 1024 == 0 && FRAME % 8 == 0, "operand and barrier alignment");
};
// Barriers per tile parity (operand, hidden accumulator, activations, output accumulator).
enum : int { HB_OP0 = 0, HB_ACC0 = 2, HB_ACT0 = 4, HB_OUT0 = 6, HB_COUNT = 8 };

struct Args {
  MlpCall calls[2];
  int n_first;                       // chains of the first call
  int first[2 * MAX_CHAINS + 1];     // first CTA of each chain, then the grid
  int* host_status;
};

__device__ __forceinline__ uint4 pack_row8(const float* src) {
  const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
  return make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
}

// A row's squares one after the other: in two chains the norm's root differs in its last bit, and roundings behind it with it, down to
// the action that is drawn.
__device__ __forceinline__ float add_squares(float sum, uint32_t two) { return fmaf(bf16_hi(two), bf16_hi(two), fmaf(bf16_lo(two), bf16_lo(two), sum)); }

template <bool ENC>
__global__ void __launch_bounds__(THREADS, 1) k_head_tiles(const __grid_constant__ Args a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using M = Map<ENC>;
  constexpr int OUT = M::OUT;
  int c = 0;
  while ((int)blockIdx.x >= a.first[c + 1]) ++c;
  const int block = blockIdx.x - a.first[c], blocks = a.first[c + 1] - a.first[c], in_call = c < a.n_first ? 0 : 1;
  const MlpCall& call = a.calls[in_call];
  const MlpChain& chain = call.chain[in_call ? c - a.n_first : c];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  wait_for_previous();
  // operands: eight k of a row per thread and turn, several turns' loads under way; rows of w2 past out_store are zero
#pragma unroll 4
  for (int i = tid; i < HIDDEN * 16; i += THREADS) {
    const int r = i >> 4, g = i & 15;
    uint4 v;
    if constexpr (ENC) {   // rows of any width, zero past it
      float w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = 8 * g + j < call.in_dim ? chain.w1[(size_t)r * call.w1_ld + 8 * g + j] : 0.f;
      v = make_uint4(pack_bf16(w[0], w[1]), pack_bf16(w[2], w[3]), pack_bf16(w[4], w[5]), pack_bf16(w[6], w[7]));
    } else {
      v = pack_row8(chain.w1 + r * D + 8 * g);
    }
    *reinterpret_cast<uint4*>(smem + (g >> 3) * M::W1_ATOM + swz(r, g & 7)) = v;
  }
#pragma unroll 4
  for (int i = tid; i < OUT * 32; i += THREADS) {
    const int r = i >> 5, g = i & 31;
    *reinterpret_cast<uint4*>(smem + M::W2 + (g >> 3) * M::W2_ATOM + swz(r, g & 7)) =
        r < chain.out_store ? pack_row8(chain.w2 + (size_t)r * HIDDEN + 8 * g) : make_uint4(0u, 0u, 0u, 0u);
  }
  float* b1 = reinterpret_cast<float*>(smem + M::VEC);
  float *g1 = b1 + HIDDEN, *b2 = g1 + HIDDEN, *g2 = b2 + OUT;
  for (int i = tid; i < HIDDEN; i += THREADS) {
    b1[i] = round_bf16(chain.b1[i]);
    g1[i] = 0.5f * chain.g1[i];   // see activation
  }
  if (tid < OUT) {
    b2[tid] = tid < chain.out_store ? round_bf16(chain.b2[tid]) : 0.f;
    if (ENC) g2[tid] = chain.g2[tid];
  }
  if (ENC)   // the columns past the input's width stay zero
    for (int i = tid; i < 65536 / 16; i += THREADS) reinterpret_cast<uint4*>(smem + M::A)[i] = make_uint4(0u, 0u, 0u, 0u);
  // no launch of this call shares a status word with the next: a wait that runs out stops its CTA and tells the host
  int* status = reinterpret_cast<int*>(smem + M::STATUS);
  if (tid == 0) *status = 0;
  fence_proxy_async();
  const int counts[HB_COUNT] = {EPI_WARPS, EPI_WARPS, 1, 1, EPI_WARPS, EPI_WARPS, 1, 1};
  const Frame f = open_frame(smem + M::FRAME, status, a.host_status, counts);
  const Sync s{smem_u32(f.bars), status, f.aborted};
  const uint32_t tmem = *f.tmem_slot, base = smem_u32(smem);
  const int rows = call.n_rows, tiles = (rows + TILE - 1) / TILE;
  const int my_tiles = block < tiles ? (tiles - block + blocks - 1) / blocks : 0;

  if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(tmem), w1 = desc_lo(base), w2 = desc_lo(base + M::W2);
    auto hidden = [&](int i) {
      const uint32_t set = i & 1;
      s.wait(HB_OP0 + set, i >> 1, TIMEOUT_OPERAND);
      tc_fence_after();
      const uint32_t x = uniform(desc_lo(base + M::A + set * 32768));
      if constexpr (ENC) {
        const int steps = (call.in_dim + 15) / 16;
#pragma unroll 1
        for (int k = 0; k < steps; ++k)
          mma_one<false>(el, tm + 256 * set, uniform(x + (k >> 2) * 1024 + 2 * (k & 3)), uniform(w1 + (k >> 2) * (M::W1_ATOM >> 4) + 2 * (k & 3)), instr_desc(256), k ? 1u : 0u);
      } else {
        product128(el, tm + 256 * set, x, w1, M::W1_ATOM >> 4, instr_desc(256));
      }
      tc_commit_if(el, s.bars + 8 * (HB_ACC0 + set));
    };
    if (my_tiles > 0) hidden(0);
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      const uint32_t set = i & 1;
      if (i + 1 < my_tiles) hidden(i + 1);
      s.wait(HB_ACT0 + set, i >> 1, TIMEOUT_OPERAND);
      tc_fence_after();
#pragma unroll
      for (uint32_t k = 0; k < 16; ++k)
        mma_one<true>(el, tm + 256 * set + 128, tm + 256 * set + 8 * k, w2 + (k >> 2) * (M::W2_ATOM >> 4) + 2 * (k & 3), instr_desc(OUT), k ? 1u : 0u);
      tc_commit_if(el, s.bars + 8 * (HB_OUT0 + set));
    }
    for (int i = my_tiles - 2; i < my_tiles; ++i)
      if (i >= 0) s.wait(HB_OUT0 + (i & 1), i >> 1, TIMEOUT_ACC);
  } else if (warp < EPI_WARPS) {
    const int part = warp >> 2, quarter = warp & 3;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const int row0 = 32 * quarter + (lane >> 2), col = 32 * part + 8 * (lane & 3);   // input: rows row0 + 8 k, eight columns
    const bool pairs = ((chain.out_store | chain.y_ld) & 1) == 0;                  // two columns share an aligned word
    // heads: sixteen bytes of four rows; encoder: pairs of the tile's values, which lie in one piece
    uint4 in[ENC ? 8 : 4];
    const int half = call.in_dim >> 1, n_pairs = ENC ? TILE * half : 0;
    const float inv_half = ENC ? 1.0f / (float)half : 0.f;
    auto request = [&](int i) {
      if constexpr (ENC) {
        const float2* src = static_cast<const float2*>(call.x) + (size_t)(block + (size_t)i * blocks) * TILE * half;
        const int left = i < my_tiles ? min(TILE, rows - (block + i * blocks) * TILE) * half : 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int at = tid + EPI_THREADS * k;
          float2 v = make_float2(0.f, 0.f);
          if (at < left) v = src[at];
          reinterpret_cast<uint32_t*>(in)[k] = pack_bf16(v.x, v.y);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = (block + i * blocks) * TILE + row0 + 8 * k;
          in[k] = make_uint4(0u, 0u, 0u, 0u);
          if (i < my_tiles && r < rows) {
            const int from = call.group_rows ? r / call.group_rows * call.group_stride + r % call.group_rows : r;
            in[k] = call.x_bf16 ? *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(call.x) + (size_t)from * D + col)
                                  : pack_row8(static_cast<const float*>(call.x) + (size_t)from * D + col);
          }
        }
      }
    };
    auto put = [&](int i) {
      if constexpr (ENC) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int at = tid + EPI_THREADS * k;
          if (at >= n_pairs) continue;
          int r = (int)((float)at * inv_half);   // at < 2^14: off by one at most
          r -= r * half > at;
          r += (r + 1) * half <= at;
          const int c = 2 * (at - r * half);
          *reinterpret_cast<uint32_t*>(smem + M::A + (i & 1) * 32768 + (c >> 6) * CHUNK_BYTES + swz(r, (c & 63) >> 3) + (c & 7) * 2) = reinterpret_cast<const uint32_t*>(in)[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          *reinterpret_cast<uint4*>(smem + M::A + (i & 1) * 32768 + (col >> 6) * CHUNK_BYTES + swz(row0 + 8 * k, (col & 63) >> 3)) = in[k];
      }
    };
    auto finish = [&](int i) {   // heads: eight output columns of this thread's row; encoder: 32, and the last norm
      if constexpr (ENC) {
        s.wait(HB_OUT0 + (i & 1), i >> 1, TIMEOUT_ACC);
        tc_fence_after();
        uint32_t v[32];
        tmem_ld32(lane_addr + 256 * (i & 1) + 128 + 32 * part, v);
        tc_fence_before();
        float ss = 0.f;
        const F2* bias = reinterpret_cast<const F2*>(b2 + 32 * part);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          v[j] = pack_bf16(add(f2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), bias[j]));
          ss = add_squares(ss, v[j]);
        }
        float* sums = reinterpret_cast<float*>(smem + M::SUMS) + 1024 + (i & 1) * 512 + (tid & (TILE - 1));
        sums[part * TILE] = ss;
        asm volatile("bar.sync %0, 128;" ::"r"(3 + quarter) : "memory");
        const float inv = rsqrtf(((sums[0] + sums[TILE]) + (sums[2 * TILE] + sums[3 * TILE])) / (float)OUT + kRmsEps);
        const int r = (block + i * blocks) * TILE + (tid & (TILE - 1));
        uint4* y = reinterpret_cast<uint4*>(chain.y + (size_t)r * OUT + 32 * part);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w[j] = pack_bf16(mul(mul(unpack_bf16(v[4 * q + j]), f2(inv)), reinterpret_cast<const F2*>(g2 + 32 * part)[4 * q + j]));
          if (r < rows) y[q] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      } else {     // eight output columns of this thread's row
        s.wait(HB_OUT0 + (i & 1), i >> 1, TIMEOUT_ACC);
        tc_fence_after();
        uint32_t v[8];
        tmem_ld8_nowait(lane_addr + 256 * (i & 1) + 128 + 8 * part, v);
        tmem_wait_ld();
        tc_fence_before();
        const int r = (block + i * blocks) * TILE + (tid & (TILE - 1));
        if (r >= rows) return;
        __nv_bfloat16* y = chain.y + (size_t)r * chain.y_ld;
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          const int c = 8 * part + j;
          const uint32_t w = pack_bf16(__uint_as_float(v[j]) + b2[c], __uint_as_float(v[j + 1]) + b2[c + 1]);
          const __nv_bfloat162 p = *reinterpret_cast<const __nv_bfloat162*>(&w);
          if (pairs) {
            if (c < chain.out_store) *reinterpret_cast<uint32_t*>(y + c) = w;
          } else {
            if (c < chain.out_store) y[c] = p.x;
            if (c + 1 < chain.out_store) y[c + 1] = p.y;
          }
        }
      }
    };
    if (my_tiles > 0) {
      request(0);
      put(0);
      post(s, HB_OP0);
      request(1);
    }
#pragma unroll 1
    for (int i = 0; i < my_tiles; ++i) {
      if (i + 1 < my_tiles) put(i + 1);
      if (i > 0) finish(i - 1);   // before the next tile's first product takes its columns
      if (i + 1 < my_tiles) post(s, HB_OP0 + ((i + 1) & 1));
      request(i + 2);
      s.wait(HB_ACC0 + (i & 1), i >> 1, TIMEOUT_ACC);
      tc_fence_after();
      const uint32_t acc = lane_addr + 256 * (i & 1);
      uint32_t v[32];   // the Linear's output, two bfloat16 a word
      float ss = 0.f;
      const float4* bias = reinterpret_cast<const float4*>(b1 + 64 * part);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[32];
        tmem_ld32(acc + 64 * part + 32 * c, t);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 b = bias[8 * c + q];
          uint32_t* w = v + 16 * c + 2 * q;
          w[0] = pack_bf16(add(f2(__uint_as_float(t[4 * q]), __uint_as_float(t[4 * q + 1])), f2(b.x, b.y)));
          w[1] = pack_bf16(add(f2(__uint_as_float(t[4 * q + 2]), __uint_as_float(t[4 * q + 3])), f2(b.z, b.w)));
          ss = add_squares(add_squares(ss, w[0]), w[1]);
        }
      }
      float* sums = reinterpret_cast<float*>(smem + M::SUMS) + (i & 1) * 512 + (tid & (TILE - 1));   // two buffers: one barrier a tile
      sums[part * TILE] = ss;
      tc_fence_before();
      asm volatile("bar.sync %0, 128;" ::"r"(3 + quarter) : "memory");   // and every column of these rows has been read
      tc_fence_after();
      const float inv = rsqrtf(((sums[0] + sums[TILE]) + (sums[2 * TILE] + sums[3 * TILE])) / (float)HIDDEN + kRmsEps);
      const float4* gain = reinterpret_cast<const float4*>(g1 + 64 * part);
      const F2 inv2 = f2(inv);
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        uint32_t w[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 g = gain[4 * o + q];
          w[2 * q] = activation(v[8 * o + 2 * q], inv2, f2(g.x, g.y));
          w[2 * q + 1] = activation(v[8 * o + 2 * q + 1], inv2, f2(g.z, g.w));
        }
        tmem_st8_nowait(acc + 32 * part + 8 * o, w);
      }
      tmem_wait_st();
      post(s, HB_ACT0 + (i & 1));
    }
    if (my_tiles > 0) finish(my_tiles - 1);
  }
  close_frame(f, tmem);
}

}  // namespace

bool head_tiles_serve(const MlpCall& call, int n_chains, int in_pad, int hidden, int out_dim) {
  if (hidden != HIDDEN || call.active) return false;
  const auto at = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  if (out_dim == 32) {   // heads
    if (call.in_dim != D || in_pad != D || call.w1_ld != D || at(call.x) % 16) return false;
    for (int i = 0; i < n_chains; ++i)
      if (call.chain[i].g2 || (at(call.chain[i].w1) | at(call.chain[i].w2)) % 16) return false;
    return true;
  }
  const MlpChain& c = call.chain[0];   // encoder
  return n_chains == 1 && !call.x_bf16 && c.g2 && out_dim == D && c.out_store == D && c.y_ld == D && call.in_dim % 2 == 0 && call.in_dim <= D && !call.group_rows &&
         at(call.x) % 8 == 0 && (at(c.w2) | at(c.y)) % 16 == 0;
}

int head_tiles(const MlpCall& call, int n_chains, int out_dim, cudaStream_t st, const MlpCall* more, int n_more) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BNB_ERR_NO_DEVICE;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(k_head_tiles<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Map<false>::BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(k_head_tiles<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Map<true>::BYTES) != cudaSuccess)
      return BNB_ERR_LAUNCH;
    configured[dev] = true;
  }
  Args a{};
  a.calls[0] = call;
  if (more) a.calls[1] = *more;
  a.n_first = n_chains;
  a.host_status = host_status_word(st);
  // a CTA fills an SM and stages its weights once: the chains share the SMs out so that none takes more rounds of tiles than it must
  const int n = n_chains + (more ? n_more : 0);
  int tiles[2 * MAX_CHAINS], longest = 0;
  for (int i = 0; i < n; ++i) {
    tiles[i] = ((i < n_chains ? call : *more).n_rows + TILE - 1) / TILE;
    longest = tiles[i] > longest ? tiles[i] : longest;
  }
  const auto ctas = [&](int rounds) {
    a.first[0] = 0;
    for (int i = 0; i < n; ++i) a.first[i + 1] = a.first[i] + (tiles[i] + rounds - 1) / rounds;
    return a.first[n];
  };
  int enough = longest;   // rounds: a CTA a chain
  for (int few = 0; few + 1 < enough;) {
    const int mid = few + (enough - few) / 2;
    if (ctas(mid) <= 148) enough = mid;
    else few = mid;
  }
  const dim3 grid((unsigned)ctas(enough));
  return out_dim == 32 ? launch_after(k_head_tiles<false>, grid, THREADS, Map<false>::BYTES, st, a)
                       : launch_after(k_head_tiles<true>, grid, THREADS, Map<true>::BYTES, st, a);
}

}  // namespace mlp
}  // namespace bnb
