// One step of the trunk under the float32 contract (d_model 128, 4 heads) on tcgen05 tiles.
//
// A float32 product on bfloat16 tensor cores: each operand is the sum of three bfloat16 numbers, v = h + m + l
// (8 significant bits each, 24 in all: the sum is exact), and of the nine products the six above 2^-26 relative
// are accumulated in float32, smallest first.  Against two tf32 numbers and three products that is the same
// tensor time, a smaller dropped term (2^-26 against 2^-22) and operands a TMA copy can bring as they are.
//
// The row-wise layers of a sublayer need whole rows of 128 only, so a tile is 128 rows and one CTA keeps its
// operand (three pieces, 96 KB) in shared memory while the weights stream past it.  A step of 3552 rows has 28
// tiles for 148 SMs: each kernel splits the columns of its products over several CTAs as well.
//
//   k_pack      weights to three-piece images (every call, from the live parameters)
//   k_project   norm -> q|k|v, and norm -> k|v of the bullets
//   k_attend    attention of an environment, bullets included, on the float32 pipes
//   k_front     temporal sublayer up to the recurrent branch's output: norm -> linear1 (all columns) | linear2
//               (own columns) -> conv -> gates (own columns) -> RG-LRU.  Field tokens: field_sub in place of the
//               last three.
//   k_post      output projection -> residual -> norm -> GatedMLP -> residual, the hidden columns split over a
//               cluster, whose partial sums meet in distributed shared memory.
//
// One step of 96 environments of 37 tokens took 1457 us with a CTA per 32 rows walking all layers on mma.sync
// (111 CTAs, each streaming every weight through registers), and takes 258 here.  What bounds these kernels is
// the chain inside a CTA: k_post's 24 us are rows in 2, output projection 2, norm 1.5, gate|up 4.5, GELU and down
// projection 3, exchange 4 and the start; the tensor cores work for a third of that.  Launches overlap by
// programmatic dependence (289 us without), clusters of two instead of four take 295.
#include "split_kernels.h"

#include "common.cuh"
#include "launch_count.h"
#include "tensor_kernels.h"
#include "tile_rows.cuh"

namespace bnb {
namespace split {

using namespace tensor;

namespace {

constexpr int F = 512;                              // hidden width of the GatedMLP
constexpr uint32_t PIECE = 32768, ATOM = 16384;     // operand tile: 3 pieces of 2 K atoms of 128 rows x 64
constexpr uint32_t S_RING = 3 * PIECE, RING_BYTES = 7 * 16384, S_SUMS = S_RING + RING_BYTES, S_ROWS = S_SUMS + 2048,
                   S_FRAME = S_ROWS + 1024, SMEM = S_FRAME + 512;

// ------------------------------------------------------------------ pieces and images

// Two floats as three pairs of bfloat16, exact sums.
__device__ __forceinline__ void split3(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(a, b);
  a -= bf16_lo(h);
  b -= bf16_hi(h);
  m = pack_bf16(a, b);
  l = pack_bf16(a - bf16_lo(m), b - bf16_hi(m));
}
// Four columns of a row into the operand tile.
__device__ __forceinline__ void put_pieces(uint8_t* tile, int row, int col, const float4& v) {
  uint32_t h[2], m[2], l[2];
  split3(v.x, v.y, h[0], m[0], l[0]);
  split3(v.z, v.w, h[1], m[1], l[1]);
  uint8_t* at = tile + (col >> 6) * ATOM + swz(row, (col & 63) >> 3) + ((col >> 2) & 1) * 8;
  *reinterpret_cast<uint2*>(at) = make_uint2(h[0], h[1]);
  *reinterpret_cast<uint2*>(at + PIECE) = make_uint2(m[0], m[1]);
  *reinterpret_cast<uint2*>(at + 2 * PIECE) = make_uint2(l[0], l[1]);
}
__device__ __forceinline__ float4 get_pieces(const uint8_t* tile, int row, int col) {
  const uint8_t* at = tile + (col >> 6) * ATOM + swz(row, (col & 63) >> 3) + ((col >> 2) & 1) * 8;
  const uint2 h = *reinterpret_cast<const uint2*>(at), m = *reinterpret_cast<const uint2*>(at + PIECE),
              l = *reinterpret_cast<const uint2*>(at + 2 * PIECE);
  return make_float4(bf16_lo(h.x) + (bf16_lo(m.x) + bf16_lo(l.x)), bf16_hi(h.x) + (bf16_hi(m.x) + bf16_hi(l.x)),
                     bf16_lo(h.y) + (bf16_lo(m.y) + bf16_lo(l.y)), bf16_hi(h.y) + (bf16_hi(m.y) + bf16_hi(l.y)));
}

// Image of a (rows, K) weight: for each 64 k and each piece, rows x 128 bytes in the operand's swizzle.
__host__ __device__ constexpr size_t image_bytes(int rows, int k) { return (size_t)rows * k * 6; }
struct Image { const uint8_t* at; int rows; };
// Places of a sublayer's images.
enum : int { IM_QKV = 0, IM_OUT, IM_GATE, IM_UP, IM_DOWN, IM_KVB };
enum : int { IM_LIN1 = 0, IM_LIN2, IM_A, IM_X, IM_OUT_T, IM_GATE_T, IM_UP_T, IM_DOWN_T, IM_FIELD, IM_DECAY };
__host__ __device__ constexpr size_t spatial_at(int i) {
  return image_bytes(128, 128) * (i == IM_QKV ? 0 : i == IM_OUT ? 3 : 4 + 4 * (i - IM_GATE));
}
__host__ __device__ constexpr size_t temporal_at(int i) {
  return image_bytes(128, 128) * (i <= IM_GATE_T ? i : i <= IM_DOWN_T ? 5 + 4 * (i - IM_GATE_T) : 17 + i - IM_FIELD);
}

constexpr int MAX_PACK = 96;
struct PackJobs {
  const float* src[MAX_PACK];
  uint8_t* dst[MAX_PACK];
  short rows[MAX_PACK], k[MAX_PACK];
  int* status;
};
// One thread per eight k of a row; a sublayer's matrices are 64 KB to 256 KB, read once and written as 1.5
// times that: bound by the launch.
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackJobs jobs) {
  if (jobs.status && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *jobs.status = 0;
  const int rows = jobs.rows[blockIdx.y], k = jobs.k[blockIdx.y], per_row = k / 8;   // k = 0: a vector
  const float* src = jobs.src[blockIdx.y];
  uint8_t* dst = jobs.dst[blockIdx.y];
  if (k == 0) {   // Lambda: the logarithm of its sigmoid as high and low part
    float* out = reinterpret_cast<float*>(dst);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
      const float base = sigmoidf_(src[i]);
      const double v = base == 0.f ? (double)kLogOfZero : log((double)base);
      out[i] = (float)v;
      out[rows + i] = (float)(v - (double)(float)v);
    }
    return;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows * per_row; i += gridDim.x * blockDim.x) {
    const int r = i / per_row, g = i - r * per_row;
    const float4 a = *reinterpret_cast<const float4*>(src + (size_t)r * k + 8 * g), b = *reinterpret_cast<const float4*>(src + (size_t)r * k + 8 * g + 4);
    uint32_t h[4], m[4], l[4];
    split3(a.x, a.y, h[0], m[0], l[0]);
    split3(a.z, a.w, h[1], m[1], l[1]);
    split3(b.x, b.y, h[2], m[2], l[2]);
    split3(b.z, b.w, h[3], m[3], l[3]);
    uint8_t* at = dst + (size_t)(g >> 3) * 3 * rows * 128 + swz(r, g & 7);
    *reinterpret_cast<uint4*>(at) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(at + rows * 128) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4*>(at + 2 * rows * 128) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// ------------------------------------------------------------------ shared pieces of the tile kernels

// Programmatic dependence: in this chain a kernel waits for the launch before it and triggers the one behind it after that (the
// kernels of launch_after.h the other way round), so a launch that has started knows that the one before the one before it is
// complete.  What is older than that is read before the wait: weight images from the chain's second launch on (weights_early;
// k_pack before the first is a plain launch), in k_front also the state.  A kernel that triggers first, put into this chain, would
// let its successor read both too early.
struct Waits { int* status; int* host_status; int weights_early; };

enum : int { B_FULL = 0, B_FREE = 7, B_OP0 = 14, B_OP1, B_ACC0, B_ACC1, B_GU0, B_H0 = B_GU0 + 8, B_COUNT = B_H0 + 8 };
static_assert(8 * B_COUNT <= 400, "frame area");

struct Frame { Sync s; uint32_t tmem; int* aborted; };
__device__ __forceinline__ Frame open_frame(uint8_t* smem, const Waits& w) {
  uint8_t* at = smem + S_FRAME;
  int* aborted = reinterpret_cast<int*>(at + 400);
  uint32_t* slot = reinterpret_cast<uint32_t*>(at + 416);
  const uint32_t bars = smem_u32(at);
  if (threadIdx.x == 0) {
    aborted[0] = 0;
    aborted[1] = DEFAULT_POLL_LIMIT;
    *reinterpret_cast<int**>(&aborted[2]) = w.host_status;
    for (int i = 0; i < B_COUNT; ++i)
      mbar_init(bars + 8 * i, i == B_OP0 || i == B_OP1 || i >= B_H0 ? EPI_WARPS : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    __syncwarp();
    tmem_alloc(smem_u32(slot), 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return {Sync{bars, w.status, aborted}, *slot, aborted};
}
// An earlier launch of the call whose wait ran out: this one drains too.
__device__ __forceinline__ void inherit_abort(const Frame& f) {
  if (*static_cast<volatile int*>(f.s.status) != 0) *static_cast<volatile int*>(f.aborted) = 1;
}
__device__ __forceinline__ void close_frame(const Frame& f) {
  tc_fence_before();
  __syncthreads();
  if (f.aborted[0] && threadIdx.x >= 32 * LOAD_WARP)   // copies may still be on their way here
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  __syncthreads();
  if (threadIdx.x < 32) {
    __syncwarp();
    tmem_dealloc(f.tmem, 512);
  }
}

// The ring of weight slots as one of its two sides sees it.
struct Ring {
  uint32_t bytes, n;       // of a slot, slots
  uint32_t slot, parity;   // next slot; bit per slot
  __device__ __forceinline__ uint32_t at() const { return S_RING + slot * bytes; }
  __device__ __forceinline__ void next() { parity ^= 1u << slot; slot = slot + 1 == n ? 0 : slot + 1; }
};
__device__ __forceinline__ Ring make_ring(uint32_t bytes, uint32_t parity) {
  const uint32_t n = RING_BYTES / bytes;
  return {bytes, n > 7 ? 7 : n, 0, parity};
}
// Rows [r0, r0 + n) of one block of an image.
struct Rows { Image im; int r0, n; };
// One slot by the fetching warp: block (atom, piece) of one or two row ranges, one behind the other.
__device__ __forceinline__ bool fetch(const Frame& f, Ring& ring, uint32_t base, bool elected, int atom, int piece, const Rows& a, const Rows& b) {
  f.s.wait(B_FREE + ring.slot, ring.parity >> ring.slot, TIMEOUT_FREE);
  if (__any_sync(0xffffffffu, *static_cast<volatile int*>(f.aborted))) return false;
  if (elected) {
    const uint32_t bar = f.s.bars + 8 * (B_FULL + ring.slot), dst = base + ring.at();
    const size_t block = (size_t)(atom * 3 + piece);
    mbar_expect_tx(bar, (a.n + b.n) * 128);
    bulk_g2s(dst, a.im.at + (block * a.im.rows + a.r0) * 128, a.n * 128, bar);
    if (b.n) bulk_g2s(dst + a.n * 128, b.im.at + (block * b.im.rows + b.r0) * 128, b.n * 128, bar);
  }
  __syncwarp();
  ring.next();
  return true;
}
// The six slots of a 128-deep product: per K atom the low, middle and high piece.
__device__ __forceinline__ bool fetch_product(const Frame& f, Ring& ring, uint32_t base, bool elected, const Rows& a, const Rows& b) {
  bool go = true;
#pragma unroll 1
  for (int i = 0; i < 6 && go; ++i) go = fetch(f, ring, base, elected, i >= 3, i >= 3 ? 5 - i : 2 - i, a, b);
  return go;
}
// d += operand tile x weights of the next six slots, by the issuing warp.
__device__ __forceinline__ void product(const Frame& f, Ring& ring, uint32_t base, uint32_t el, uint32_t d, uint32_t idesc) {
  const uint32_t a_lo = uniform(desc_lo(base));
#pragma unroll 1
  for (uint32_t atom = 0; atom < 2; ++atom) {
    const uint32_t a_at = uniform(a_lo + (ATOM >> 4) * atom);
#pragma unroll
    for (uint32_t weak = 0; weak < 3; ++weak) {   // weight piece 2 - weak meets operand pieces weak .. 0
      f.s.wait(B_FULL + ring.slot, ring.parity >> ring.slot, TIMEOUT_FULL);
      const uint32_t b = uniform(desc_lo(base + ring.at()));
#pragma unroll
      for (uint32_t j = 0; j <= weak; ++j)
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          mma_one<false>(el, d, a_at + (PIECE >> 4) * (weak - j) + 2 * k, b + 2 * k, idesc, (atom | weak | j | k) ? 1u : 0u);
      tc_commit_if(el, f.s.bars + 8 * (B_FREE + ring.slot));
      ring.next();
    }
  }
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void store4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// How rows come in: warp w takes rows 32 (w % 4) .. and columns 32 (w / 4) .., in its i-th request (i < 4) lane l
// eight columns of row 8 i + l / 4.  A request touches eight lines, and a piece of eight columns is sixteen
// bytes of the operand tile, stored with two lanes to a bank at most.
struct Rows8 {
  int row0, col;
  __device__ __forceinline__ int row(int i) const { return row0 + 8 * i + ((threadIdx.x & 31) >> 2); }
};
__device__ __forceinline__ Rows8 rows8() { return {32 * ((int)(threadIdx.x >> 5) & 3), 32 * (int)(threadIdx.x >> 7) + 8 * (int)(threadIdx.x & 3)}; }
__device__ __forceinline__ void rows_in8(float4 (&v)[8], const float* src, const Rows8& m, int first, int rows) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = first + m.row(i);
    const float* p = src + (size_t)r * D + m.col;
    v[2 * i] = r < rows ? load4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[2 * i + 1] = r < rows ? load4(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
// Eight columns of a row into the operand tile.
__device__ __forceinline__ void put_pieces8(uint8_t* tile, int row, int col, const float4& a, const float4& b) {
  uint32_t h[4], m[4], l[4];
  split3(a.x, a.y, h[0], m[0], l[0]);
  split3(a.z, a.w, h[1], m[1], l[1]);
  split3(b.x, b.y, h[2], m[2], l[2]);
  split3(b.z, b.w, h[3], m[3], l[3]);
  uint8_t* at = tile + (col >> 6) * ATOM + swz(row, (col & 63) >> 3);
  *reinterpret_cast<uint4*>(at) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(at + PIECE) = make_uint4(m[0], m[1], m[2], m[3]);
  *reinterpret_cast<uint4*>(at + 2 * PIECE) = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ float4 norm4(const float4& x, float inv, const float4& g) {
  return make_float4(x.x * inv * g.x, x.y * inv * g.y, x.z * inv * g.z, x.w * inv * g.w);
}
__device__ __forceinline__ float square4(const float4& x) { return fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w))); }
// Rows of the operand: n = x inv gain, as pieces.  The four lanes of a row, then the four warps of these rows,
// add up their squares.
__device__ __forceinline__ void norm_pieces(uint8_t* tile, const float4 (&x)[8], const float* gain, float* part_sums, const Rows8& m) {
  float ss[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ss[i] = square4(x[2 * i]) + square4(x[2 * i + 1]);
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
    if ((threadIdx.x & 3) == 0) part_sums[(threadIdx.x >> 7) * TILE + m.row(i)] = ss[i];
  }
  asm volatile("bar.sync %0, 128;" ::"r"(3 + ((threadIdx.x >> 5) & 3)) : "memory");
  const float4 g0 = load4(gain + m.col), g1 = load4(gain + m.col + 4);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* p = part_sums + m.row(i);
    const float inv = rsqrtf(((p[0] + p[TILE]) + (p[2 * TILE] + p[3 * TILE])) / (float)D + kRmsEps);
    put_pieces8(tile, m.row(i), m.col, norm4(x[2 * i], inv, g0), norm4(x[2 * i + 1], inv, g1));
  }
}

// ------------------------------------------------------------------ norm -> product -> rows

struct ProjectArgs {
  const float* x;
  const float* gain;
  Image w;
  float* out;              // (rows, w.rows)
  int rows, cols, splits;  // columns of a CTA, CTAs per row tile
  Waits waits;
};
__global__ void __launch_bounds__(THREADS, 1) k_project(const __grid_constant__ ProjectArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5;
  const Frame f = open_frame(smem, a.waits);
  const uint32_t base = smem_u32(smem);
  const int first = (blockIdx.x / a.splits) * TILE, n0 = (blockIdx.x % a.splits) * a.cols;
  if (warp != LOAD_WARP || !a.waits.weights_early) {
    wait_for_previous();
    let_next_start();
    inherit_abort(f);
  }
  if (warp == LOAD_WARP) {
    Ring ring = make_ring(a.cols * 128, 0x7F);
    fetch_product(f, ring, base, elect_one() != 0, {a.w, n0, a.cols}, {a.w, 0, 0});
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one();
    Ring ring = make_ring(a.cols * 128, 0);
    f.s.wait(B_OP0, 0, TIMEOUT_OPERAND);
    tc_fence_after();
    product(f, ring, base, el, uniform(f.tmem), instr_desc(a.cols));
    tc_commit_if(el, f.s.bars + 8 * B_ACC0);
    f.s.wait(B_ACC0, 0, TIMEOUT_ACC);
  } else {
    const RowMap m = row_map();
    float4 x[8];
    rows_in8(x, a.x, rows8(), first, a.rows);
    norm_pieces(smem, x, a.gain, reinterpret_cast<float*>(smem + S_SUMS), rows8());
    post(f.s, B_OP0);
    f.s.wait(B_ACC0, 0, TIMEOUT_ACC);
    tc_fence_after();
    const int part = warp >> 2;
    if (part * 32 < a.cols) {
      transpose_rows(x, f.tmem + ((uint32_t)((warp & 3) * 32) << 16) + part * 32, smem + warp * 4096, m);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = first + m.row(i);
        if (r < a.rows) store4(a.out + (size_t)r * a.w.rows + n0 + m.col, x[i]);
      }
    }
  }
  close_frame(f);
}

// ------------------------------------------------------------------ attention

// Running softmax of one query of one head, channels in pairs.
struct Soft {
  float m, l;
  F2 acc[DH / 2];
  __device__ __forceinline__ void clear() {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int d = 0; d < DH / 2; ++d) acc[d] = f2(0.f);
  }
};
constexpr int KEYS = 16;                        // of a staged chunk, for each of the two warps of a group of queries
constexpr int KV_HEAD = DH + 4, KV_V = 4 * KV_HEAD, KV_ROW = 2 * KV_V;   // staged key: four heads of k, of v, 4 floats of padding each
// kv: staged rows at this lane's head; live: bit per key, a key that is not live scores kMaskedScore, as
// attention.py:101-112 has it.  Four keys a turn, in a loop: the code runs a few times only, and unrolled over all
// keys its fetch took longer than its arithmetic.
__device__ __forceinline__ void absorb(Soft& t, const F2 (&q)[DH / 2], const float* kv, int n, uint32_t live, float scale) {
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += 4, kv += 4 * KV_ROW, live >>= 4) {
    float s[4], mx = t.m;
#pragma unroll
    for (int j = 0; j < 4; ++j) {   // rows past the n-th hold older keys: read, not used
      F2 a = f2(0.f), b = f2(0.f);
#pragma unroll
      for (int d = 0; d < DH; d += 4) {
        const float4 u = load4(kv + j * KV_ROW + d);
        a = fma(q[d / 2], f2(u.x, u.y), a);
        b = fma(q[d / 2 + 1], f2(u.z, u.w), b);
      }
      const float2 p = halves(a), r = halves(b);
      s[j] = j0 + j < n ? ((live >> j) & 1u ? ((p.x + p.y) + (r.x + r.y)) * scale : kMaskedScore) : -INFINITY;
      mx = fmaxf(mx, s[j]);
    }
    const float corr = expf(t.m - mx);   // exp(-inf) = 0 at the first keys
    t.m = mx;
    t.l *= corr;
    const F2 c2 = f2(corr);
#pragma unroll
    for (int d = 0; d < DH / 2; ++d) t.acc[d] = mul(t.acc[d], c2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j0 + j >= n) break;
      const float p = expf(s[j] - mx);
      const F2 p2 = f2(p);
      t.l += p;
#pragma unroll
      for (int d = 0; d < DH; d += 4) {
        const float4 v = load4(kv + j * KV_ROW + KV_V + d);
        t.acc[d / 2] = fma(p2, f2(v.x, v.y), t.acc[d / 2]);
        t.acc[d / 2 + 1] = fma(p2, f2(v.z, v.w), t.acc[d / 2 + 1]);
      }
    }
  }
}

// One environment and 128 of its (head, query) pairs per CTA, a lane per pair, head by head: the lanes of a warp
// read the same key of one head, or of the two that meet in it (broadcasts on different banks).  Two warps share
// 32 pairs, each takes half of a chunk of 32 keys; the halves meet at the end.  Bound by instructions, which is
// why lanes hold pairs (37 queries fill 5 warps, a warp per head and 32 queries would be 8) and channels go two at
// a time.  Keys and values pass through shared memory once per CTA in whole rows, the next chunk's on their way
// while one is worked on; of the bullets only the active slots do, since the others' weight is exactly zero (and
// the sum is, if none is active).
struct AttendArgs {
  const float* qkv;
  const uint8_t* alive;
  float* o;
  EnvMap map;
  int env0;                 // first environment of the launch
  const float* kvb;         // (environments of the launch * nb, 256), or null
  const uint8_t* active;    // (environments, nb), or null: all
  int nb;
};
constexpr int KV_BUF = (2 * KEYS + 4) * KV_ROW, ATT_SMEM = 2 * KV_BUF * 4;   // a turn of four may reach past a chunk's last key
constexpr int ATT_THREADS = 256, ATT_PAIRS = ATT_THREADS / 2, SLOTS = ATT_THREADS;
template <bool BULLETS>
__global__ void __launch_bounds__(ATT_THREADS, 2) k_attend(const __grid_constant__ AttendArgs a) {
  extern __shared__ __align__(16) float kv[];   // two chunks
  __shared__ int slots[SLOTS], counts[ATT_THREADS / 32];
  wait_for_previous();
  let_next_start();
  const int e = a.env0 + blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tok0 = a.map.env_tok_begin(e), n = a.map.env_tok_count(e), first = blockIdx.y * ATT_PAIRS + 32 * (warp & 3);
  if ((int)blockIdx.y * ATT_PAIRS >= HEADS * n) return;
  const bool working = first < HEADS * n;        // the same in the whole warp
  const int pair = min(first + lane, HEADS * n - 1), head = pair / n, row = tok0 + pair - head * n, half = warp >> 2;
  const float scale = rsqrtf((float)DH);
  F2 q[DH / 2];
#pragma unroll
  for (int d = 0; d < DH; d += 4) {
    const float4 v = load4(a.qkv + (size_t)row * 384 + head * DH + d);
    q[d / 2] = f2(v.x, v.y);
    q[d / 2 + 1] = f2(v.z, v.w);
  }
  Soft t;
  // count keys in chunks: row_of(k) is key k's [k | v] row, up(k) whether it is live
  auto walk = [&](int count, auto row_of, auto up) {
    auto request = [&](int k0) {
      const uint32_t dst = smem_u32(kv + ((k0 / (2 * KEYS)) & 1) * KV_BUF + ((tid >> 5) & 1) * KV_V + ((tid >> 3) & 3) * KV_HEAD + (tid & 7) * 4);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = (tid >> 6) + 4 * j;
        if (k0 + k < count) cp_async16(dst + k * KV_ROW * 4, row_of(k0 + k) + (tid & 63) * 4);
      }
    };
    __syncthreads();
    request(0);
    for (int k0 = 0; k0 < count; k0 += 2 * KEYS) {
      const int nk = min(2 * KEYS, count - k0);
      const bool lit = lane < nk && up(k0 + lane);
      asm volatile("cp.async.wait_all;" ::: "memory");
      const uint32_t live = __ballot_sync(0xffffffffu, lit);
      __syncthreads();   // this chunk is there for everyone, everyone is done with the one before
      if (k0 + 2 * KEYS < count) request(k0 + 2 * KEYS);
      const int mine = half ? nk / 2 : nk - nk / 2, begin = half ? nk - nk / 2 : 0;
      if (working) absorb(t, q, kv + ((k0 / (2 * KEYS)) & 1) * KV_BUF + begin * KV_ROW + head * KV_HEAD, mine, live >> begin, scale);
    }
  };
  // the two halves: the upper one's through shared memory into the lower one's result
  auto merge = [&](F2 (&out)[DH / 2], bool add) {
    float* share = kv + (warp & 3) * 32 * (DH + 2) + lane;
    __syncthreads();
    if (half) {
      share[0] = t.m;
      share[32] = t.l;
#pragma unroll
      for (int d = 0; d < DH / 2; ++d) {
        const float2 v = halves(t.acc[d]);
        share[(2 + 2 * d) * 32] = v.x;
        share[(3 + 2 * d) * 32] = v.y;
      }
    }
    __syncthreads();
    if (half || !working || (add && !(t.l + share[32] > 0.f))) return;
    const float m = fmaxf(t.m, share[0]), ea = expf(t.m - m), eb = expf(share[0] - m), inv = 1.0f / (t.l * ea + share[32] * eb);
    const F2 ca = f2(ea * inv), cb = f2(eb * inv);
#pragma unroll
    for (int d = 0; d < DH / 2; ++d)
      out[d] = fma(t.acc[d], ca, fma(f2(share[(2 + 2 * d) * 32], share[(3 + 2 * d) * 32]), cb, add ? out[d] : f2(0.f)));
  };
  F2 out[DH / 2];
  t.clear();
  walk(n, [&](int k) { return a.qkv + (size_t)(tok0 + k) * 384 + 128; }, [&](int k) { return !a.alive || a.alive[tok0 + k]; });
  merge(out, false);
  if constexpr (BULLETS) {
    t.clear();
    const float* rows = a.kvb + (size_t)blockIdx.x * a.nb * 256;
    for (int s0 = 0; s0 < a.nb; s0 += SLOTS) {
      const int slot = s0 + tid;
      const bool on = slot < a.nb && (!a.active || a.active[(size_t)e * a.nb + slot]);
      const uint32_t ballot = __ballot_sync(0xffffffffu, on);
      __syncthreads();   // the slots before are done with
      if (lane == 0) counts[warp] = __popc(ballot);
      __syncthreads();
      int at = __popc(ballot & ((1u << lane) - 1)), total = 0;
#pragma unroll
      for (int w = 0; w < ATT_THREADS / 32; ++w) {
        if (w < warp) at += counts[w];
        total += counts[w];
      }
      if (on) slots[at] = slot;
      __syncthreads();
      walk(total, [&](int k) { return rows + (size_t)slots[k] * 256; }, [](int) { return true; });
    }
    merge(out, true);
  }
  if (!half && first + lane < HEADS * n)
#pragma unroll
    for (int d = 0; d < DH; d += 4) {
      const float2 u = halves(out[d / 2]), v = halves(out[d / 2 + 1]);
      store4(a.o + (size_t)row * D + head * DH + d, make_float4(u.x, u.y, v.x, v.y));
    }
}

// ------------------------------------------------------------------ temporal sublayer, first half

struct FrontArgs {
  const float* x;
  float* o;                 // (tokens, 128): what the output projection takes
  const float* hidden_in;
  float* hidden_out;
  const uint8_t* reset_env;
  EnvMap map;
  int ship_tiles;           // row tiles of ships, then those of field tokens
  int cols, splits;         // columns of a CTA, CTAs per row tile
  BnbTemporalWeights w;
  Image lin1, lin2, gate_a, gate_x, field;
  const float* decay;       // log sigmoid(Lambda): high parts, low parts
  Waits waits;
};

// sigmoid(Lambda)^(8 r) from the logarithm of the sigmoid in two parts, so that the product with 8 r keeps the
// precision a powf has (which took half of the kernel's last phase).
__device__ __forceinline__ float rglru(float ga, float gx, float ba, float bx, float log_hi, float log_lo, float u, float h) {
  const float c = kRglruC * sigmoidf_(ga + ba), ig = sigmoidf_(gx + bx);
  const float e = c * log_hi, rest = fmaf(c, log_lo, fmaf(c, log_hi, -e)), ea = expf(e);
  const float a = fmaf(ea, rest, ea);
  return a * h + sqrtf(fmaxf((1.0f - a) * (1.0f + a), kGateFloor)) * (ig * u);
}

// Tensor memory: linear1 | linear2 of the own columns at 0, gates a | x (or field_sub) of the own columns at 256.
// The conv needs a token's own four values per column, the gates a whole row of its result: every CTA computes
// all 128 columns of linear1 and the conv (2 us for a tile, less than another launch and the way through memory)
// and keeps the columns it owns of the rest.
__global__ void __launch_bounds__(THREADS, 1) k_front(const __grid_constant__ FrontArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5;
  const Frame f = open_frame(smem, a.waits);
  const uint32_t base = smem_u32(smem);
  const int tile = blockIdx.x / a.splits, c0 = (blockIdx.x % a.splits) * a.cols;
  const bool ships = tile < a.ship_tiles;
  const uint32_t slot_bytes = (a.cols == 128 ? 256 : 128 + a.cols) * 128;
  // What comes from the caller is there before the wait: the rows' places, their incoming state.
  const int item0 = (ships ? tile : tile - a.ship_tiles) * TILE, n_items = ships ? a.map.total_ships : a.map.total_fields();
  int* token = reinterpret_cast<int*>(smem + S_ROWS);    // token row of each tile row, -1 past the end
  int* fresh = token + TILE;                             // its incoming state counts as zero
  const RowMap m = row_map();
  // Stored conv taps of four of this lane's rows at a time, all loads before the stores of
  // the new taps (behind them they would wait for each other)
  float4 taps[12];
  auto load_taps = [&](int i0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = m.row(i0 + i);
      const float* h = a.hidden_in + (size_t)(item0 + r) * 4 * D + m.col;
#pragma unroll
      for (int k = 0; k < 3; ++k) taps[3 * i + k] = fresh[r] ? make_float4(0.f, 0.f, 0.f, 0.f) : load4(h + (k + 1) * D);
    }
  };
  if (warp < EPI_WARPS) {
    if (tid < TILE) {
      const int it = item0 + tid;
      int row = -1, e = 0;
      if (it < n_items) row = ships ? a.map.ship_token_row(it, &e) : a.map.field_token_row(it);
      token[tid] = row;
      fresh[tid] = row < 0 || (ships && a.reset_env && a.reset_env[e]);
    }
    epi_sync();
    if (ships) load_taps(0);
  }
  if (warp != LOAD_WARP || !a.waits.weights_early) {
    wait_for_previous();
    let_next_start();
    inherit_abort(f);
  }
  if (warp == LOAD_WARP) {
    const bool elected = elect_one() != 0;
    Ring ring = make_ring(slot_bytes, 0x7F);
    if (fetch_product(f, ring, base, elected, {a.lin1, 0, 128}, {a.lin2, c0, a.cols})) {
      if (ships) fetch_product(f, ring, base, elected, {a.gate_a, c0, a.cols}, {a.gate_x, c0, a.cols});
      else fetch_product(f, ring, base, elected, {a.field, c0, a.cols}, {a.field, 0, 0});
    }
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(f.tmem);
    Ring ring = make_ring(slot_bytes, 0);
    f.s.wait(B_OP0, 0, TIMEOUT_OPERAND);
    tc_fence_after();
    product(f, ring, base, el, tm, instr_desc(128 + a.cols));
    tc_commit_if(el, f.s.bars + 8 * B_ACC0);
    f.s.wait(B_OP1, 0, TIMEOUT_OPERAND);
    tc_fence_after();
    product(f, ring, base, el, tm + 256, instr_desc(ships ? 2 * a.cols : a.cols));
    tc_commit_if(el, f.s.bars + 8 * B_ACC1);
    f.s.wait(B_ACC1, 0, TIMEOUT_ACC);
  } else {
    const uint32_t lane_addr = f.tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int part = warp >> 2;
    float4 v[8];
    {
      const Rows8 in = rows8();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = token[in.row(i)];
        const float* p = a.x + (size_t)row * D + in.col;
        v[2 * i] = row >= 0 ? load4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[2 * i + 1] = row >= 0 ? load4(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      norm_pieces(smem, v, a.w.norm1_w, reinterpret_cast<float*>(smem + S_SUMS), in);
    }
    post(f.s, B_OP0);
    f.s.wait(B_ACC0, 0, TIMEOUT_ACC);
    tc_fence_after();
    // linear1: through shared memory (the operand is done with) into the row layout
    uint8_t* own_stage = smem + warp * 4096;
    stage_rows(lane_addr + part * 32, own_stage, m.lane);
    __syncwarp();
    if (ships) {
      const bool own = (unsigned)(m.col - c0) < (unsigned)a.cols;
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        if (i0) load_taps(i0);
        float4 cw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) cw[j] = load4(a.w.conv_w + (m.col + j) * BNB_CONV_KERNEL);
        const float4 cb = load4(a.w.conv_b + m.col);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = m.row(i0 + i);
          const float4 t0 = taps[3 * i], t1 = taps[3 * i + 1], t2 = taps[3 * i + 2], b1 = staged_row(own_stage, i0 + i, m.lane);
          if (own && token[r] >= 0) {
            float* h = a.hidden_out + (size_t)(item0 + r) * 4 * D + m.col;
            store4(h + D, t1); store4(h + 2 * D, t2); store4(h + 3 * D, b1);
          }
          auto conv = [](float p0, float p1, float p2, float p3, const float4& w, float b) {
            return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p0, w.x), __fmul_rn(p1, w.y)), __fmul_rn(p2, w.z)), __fmul_rn(p3, w.w)), b);
          };
          v[i0 + i] = make_float4(conv(t0.x, t1.x, t2.x, b1.x, cw[0], cb.x), conv(t0.y, t1.y, t2.y, b1.y, cw[1], cb.y),
                                  conv(t0.z, t1.z, t2.z, b1.z, cw[2], cb.z), conv(t0.w, t1.w, t2.w, b1.w, cw[3], cb.w));
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = staged_row(own_stage, i, m.lane);
    }
    epi_sync();   // every warp has read its part of the stage
#pragma unroll
    for (int i = 0; i < 8; ++i) put_pieces(smem, m.row(i), m.col, v[i]);
    post(f.s, B_OP1);
    // per group of 32 own columns: this thread's four columns of biases and decay, two rows of state
    float4 ba, bx, lh, ll, state[2];
    const int q = tid & 7;
    auto load_group = [&](int g) {
      const int col = c0 + g + 4 * q;
      ba = load4(a.w.a_b + col); bx = load4(a.w.x_b + col);
      lh = load4(a.decay + col); ll = load4(a.decay + D + col);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int r = (tid + 512 * k) >> 3;
        state[k] = fresh[r] ? make_float4(0.f, 0.f, 0.f, 0.f) : load4(a.hidden_in + (size_t)(item0 + r) * 4 * D + col);
      }
    };
    if (ships) load_group(0);
    f.s.wait(B_ACC1, 0, TIMEOUT_ACC);
    tc_fence_after();
    // 32 own columns at a time: the accumulators through the ring's memory (every slot has been read) to 1024
    // float4 over all 512 threads
    uint8_t* stage = smem + S_RING;
#pragma unroll 1
    for (int g = 0; g < a.cols; g += 32) {
      if (part < 3 && (ships || part != 1)) {   // a (or field_sub), x, linear2
        uint32_t t[32];
        tmem_ld32(lane_addr + (part == 2 ? 128 + g : 256 + part * a.cols + g), t);
        uint8_t* at = stage + part * 16384 + (warp & 3) * 4096 + m.lane * 128;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(at + ((q ^ (m.lane & 7)) << 4)) = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
      }
      if (g > 0 && ships) load_group(g);
      epi_sync();
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int r = (tid + 512 * k) >> 3, col = c0 + g + 4 * q;
        if (token[r] < 0) continue;
        const uint8_t* at = stage + (r >> 5) * 4096 + (r & 31) * 128 + ((q ^ (r & 7)) << 4);
        const float4 p = *reinterpret_cast<const float4*>(at), l2 = *reinterpret_cast<const float4*>(at + 2 * 16384);
        float4 out = make_float4(gelu_erf(l2.x), gelu_erf(l2.y), gelu_erf(l2.z), gelu_erf(l2.w));
        if (ships) {
          const float4 gx = *reinterpret_cast<const float4*>(at + 16384), u = get_pieces(smem, r, col);
          const size_t at_h = (size_t)(item0 + r) * 4 * D + col;
          float4 h = state[k];
          h = make_float4(rglru(p.x, gx.x, ba.x, bx.x, lh.x, ll.x, u.x, h.x), rglru(p.y, gx.y, ba.y, bx.y, lh.y, ll.y, u.y, h.y),
                          rglru(p.z, gx.z, ba.z, bx.z, lh.z, ll.z, u.z, h.z), rglru(p.w, gx.w, ba.w, bx.w, lh.w, ll.w, u.w, h.w));
          store4(a.hidden_out + at_h, h);
          out = make_float4(out.x * h.x, out.y * h.y, out.z * h.z, out.w * h.w);
        } else {
          out = make_float4(out.x * p.x, out.y * p.y, out.z * p.z, out.w * p.w);
        }
        store4(a.o + (size_t)token[r] * D + col, out);
      }
      epi_sync();
    }
  }
  close_frame(f);
}

// ------------------------------------------------------------------ output projection, GatedMLP

struct PostArgs {
  const float* o;
  const float* x;
  float* y;                // may be x
  const float* gain;
  Image out, gate, up, down;
  int rows, cluster;       // CTAs of a row tile
  Waits waits;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 peer_load4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .b32 p;\n\tmapa.shared::cluster.u32 p, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [p];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank));   // between two cluster barriers
  return v;
}

// A hidden chunk is 64 gate and 64 up columns in one accumulator of 128.  Its gated product goes back into the
// columns it came from, as the operand of the down projection: a thread's 16 hidden columns of a row, packed to eight words, the high piece there, the middle one 8 further, the low one in the up
// half.  Tensor memory: down 0, output projection 128, two chunks at 256 and 384.
__device__ __forceinline__ uint32_t hidden_piece(uint32_t p) { return p == 2 ? 64 : 8 * p; }

// A cluster of `cluster` CTAs shares a row tile: each computes the output projection and the norm for itself
// (1.6 us against an exchange of rows), then 8 / cluster hidden chunks and their part of the down projection.
__global__ void __launch_bounds__(THREADS, 1) k_post(const __grid_constant__ PostArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5;
  const Frame f = open_frame(smem, a.waits);
  const uint32_t base = smem_u32(smem);
  const int rank = blockIdx.x % a.cluster, first = (blockIdx.x / a.cluster) * TILE;
  const int chunks = 8 / a.cluster, chunk0 = rank * chunks;
  if (warp != LOAD_WARP || !a.waits.weights_early) {
    wait_for_previous();
    let_next_start();
    inherit_abort(f);
  }
  if (warp == LOAD_WARP) {
    const bool elected = elect_one() != 0;
    Ring ring = make_ring(16384, 0x7F);
    bool go = fetch_product(f, ring, base, elected, {a.out, 0, 128}, {a.out, 0, 0});
#pragma unroll 1
    for (int i = 0; i < chunks + 2 && go; ++i) {
      if (i >= 2)
#pragma unroll 1
        for (int piece = 2; piece >= 0 && go; --piece)
          go = fetch(f, ring, base, elected, chunk0 + i - 2, piece, {a.down, 0, 128}, {a.down, 0, 0});
      if (i < chunks && go) {
        const int r0 = (chunk0 + i) * 64;
        go = fetch_product(f, ring, base, elected, {a.gate, r0, 64}, {a.up, r0, 64});
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t el = elect_one(), tm = uniform(f.tmem), idesc = instr_desc(128);
    Ring ring = make_ring(16384, 0);
    f.s.wait(B_OP0, 0, TIMEOUT_OPERAND);
    tc_fence_after();
    product(f, ring, base, el, tm + 128, idesc);
    tc_commit_if(el, f.s.bars + 8 * B_ACC0);
    f.s.wait(B_OP1, 0, TIMEOUT_OPERAND);
    tc_fence_after();
#pragma unroll 1
    for (uint32_t i = 0; i < (uint32_t)chunks + 2; ++i) {
      const uint32_t acc = tm + 256 + 128 * (i & 1);
      if (i >= 2) {
        f.s.wait(B_H0 + i - 2, 0, TIMEOUT_OPERAND);
        tc_fence_after();
#pragma unroll 1
        for (uint32_t weak = 0; weak < 3; ++weak) {
          f.s.wait(B_FULL + ring.slot, ring.parity >> ring.slot, TIMEOUT_FULL);
          const uint32_t b = uniform(desc_lo(base + ring.at()));
#pragma unroll 1
          for (uint32_t j = 0; j <= weak; ++j) {
            const uint32_t h = uniform(acc + hidden_piece(weak - j));
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) mma_one<true>(el, tm, h + 16 * k, b + 2 * k, idesc, ((i - 2) | weak | j | k) ? 1u : 0u);
          }
          tc_commit_if(el, f.s.bars + 8 * (B_FREE + ring.slot));
          ring.next();
        }
      }
      if (i < (uint32_t)chunks) {
        product(f, ring, base, el, acc, idesc);
        tc_commit_if(el, f.s.bars + 8 * (B_GU0 + i));
      }
    }
    tc_commit_if(el, f.s.bars + 8 * B_ACC1);
    f.s.wait(B_ACC1, 0, TIMEOUT_ACC);
  } else {
    const RowMap m = row_map();
    const uint32_t lane_addr = f.tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int part = warp >> 2;
    {
      const Rows8 in = rows8();
      float4 v[8];
      rows_in8(v, a.o, in, first, a.rows);
#pragma unroll
      for (int i = 0; i < 4; ++i) put_pieces8(smem, in.row(i), in.col, v[2 * i], v[2 * i + 1]);
    }
    post(f.s, B_OP0);
    {
      // residual and norm with a thread per row and 32 columns, as the accumulator comes: x in that layout
      // touches 32 lines a request, but while the product runs
      const int r = tid & (TILE - 1), row = first + r;
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = row < a.rows ? load4(a.x + (size_t)row * D + part * 32 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
      f.s.wait(B_ACC0, 0, TIMEOUT_ACC);
      tc_fence_after();
      uint32_t t[32];
      tmem_ld32(lane_addr + 128 + part * 32, t);
      float ss = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        x[q] = add4(x[q], make_float4(__uint_as_float(t[4 * q]), __uint_as_float(t[4 * q + 1]), __uint_as_float(t[4 * q + 2]), __uint_as_float(t[4 * q + 3])));
        ss += square4(x[q]);
      }
      float* sums = reinterpret_cast<float*>(smem + S_SUMS) + r;
      sums[part * TILE] = ss;
      asm volatile("bar.sync %0, 128;" ::"r"(3 + (warp & 3)) : "memory");
      const float inv = rsqrtf(((sums[0] + sums[TILE]) + (sums[2 * TILE] + sums[3 * TILE])) / (float)D + kRmsEps);
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        const float* g = a.gain + part * 32 + 4 * q;
        put_pieces8(smem, r, part * 32 + 4 * q, norm4(x[q], inv, load4(g)), norm4(x[q + 1], inv, load4(g + 4)));
      }
    }
    post(f.s, B_OP1);
#pragma unroll 1
    for (int i = 0; i < chunks; ++i) {
      f.s.wait(B_GU0 + i, 0, TIMEOUT_ACC);
      tc_fence_after();
      const uint32_t acc = lane_addr + 256 + 128 * (i & 1) + 16 * part;
      uint32_t g[16], u[16], hh[8], hm[8], hl[8];
      tmem_ld16_nowait(acc, g);
      tmem_ld16_nowait(acc + 64, u);
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 8; ++j)
        split3(gelu_erf(__uint_as_float(g[2 * j])) * __uint_as_float(u[2 * j]),
               gelu_erf(__uint_as_float(g[2 * j + 1])) * __uint_as_float(u[2 * j + 1]), hh[j], hm[j], hl[j]);
      tmem_st8_nowait(acc, hh);
      tmem_st8_nowait(acc + 8, hm);
      tmem_st8_nowait(acc + 64, hl);
      tmem_wait_st();
      post(f.s, B_H0 + i);
    }
    f.s.wait(B_ACC1, 0, TIMEOUT_ACC);
    tc_fence_after();
    // this CTA's part of the down projection, on rank 0 with the output projection: into the operand's memory,
    // 4 KB per 32 x 32 block in the row layout's order
    uint32_t t[32];
    tmem_ld32(lane_addr + part * 32, t);
    if (rank == 0) {
      uint32_t p[32];
      tmem_ld32(lane_addr + 128 + part * 32, p);
#pragma unroll
      for (int j = 0; j < 32; ++j) t[j] = __float_as_uint(__uint_as_float(t[j]) + __uint_as_float(p[j]));
    }
    uint8_t* at = smem + warp * 4096 + m.lane * 128;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      *reinterpret_cast<uint4*>(at + ((q ^ (m.lane & 7)) << 4)) = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
    if (a.cluster == 1) epi_sync();
  }
  if (a.cluster > 1) cluster_sync();
  if (warp < EPI_WARPS) {
    // this CTA's rows: the ranks' parts in order, then the residual
    const int rows = TILE / a.cluster;
#pragma unroll 1
    for (int i = tid; i < rows * 32; i += EPI_THREADS) {
      const int r = rank * rows + (i >> 5), c = i & 31, row = first + r;
      if (row >= a.rows) continue;
      const uint32_t at = base + ((r >> 5) + 4 * (c >> 3)) * 4096 + (r & 31) * 128 + (((c & 7) ^ (r & 7)) << 4);
      const float4 res = load4(a.x + (size_t)row * D + 4 * c);
      float4 sum;
      if (a.cluster == 1) {
        sum = *reinterpret_cast<const float4*>(smem + (at - base));
      } else {
        sum = peer_load4(at, 0);
#pragma unroll 1
        for (int k = 1; k < a.cluster; ++k) sum = add4(sum, peer_load4(at, k));
      }
      store4(a.y + (size_t)row * D + 4 * c, add4(res, sum));
    }
  }
  if (a.cluster > 1) cluster_sync();   // nobody leaves while its memory is read
  close_frame(f);
}

// ------------------------------------------------------------------ host side

bool configure() {
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!done[dev])
    done[dev] = cudaFuncSetAttribute(k_attend<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM) == cudaSuccess &&
                cudaFuncSetAttribute(k_attend<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM) == cudaSuccess &&
                cudaFuncSetAttribute(k_project, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) == cudaSuccess &&
                cudaFuncSetAttribute(k_front, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) == cudaSuccess &&
                cudaFuncSetAttribute(k_post, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) == cudaSuccess;
  return done[dev];
}

// Column splits: as many CTAs as the 148 SMs hold at once, since a CTA has an SM to itself and its time is mostly
// the fixed chain; a second wave costs more than narrower products save.
int splits_of(long long tiles, int most) {
  int s = 1;
  while (2 * s <= most && tiles * 2 * s <= 148) s *= 2;
  return s;
}

struct Call {
  cudaStream_t st;
  int* status;
  int* host_status;
  int launches = 0;        // after the images
  Waits waits() const { return {status, host_status, launches >= 1}; }
  template <class Args>
  int launch(void (*kernel)(Args), const Args& args, dim3 grid, int threads, size_t smem, int cluster) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    ++launches;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, args) == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH;
  }
};

int pack(const BnbSpatialWeights* s, int ns, const BnbTemporalWeights* t, int nt, bool bullets, bool fields, const Call& c) {
  PackJobs jobs{};
  int n = 0;
  jobs.status = c.status;
  auto flush = [&]() {
    if (n == 0) return;
    count_launch();
    k_pack<<<dim3(8, n), 256, 0, c.st>>>(jobs);
    n = 0;
    jobs.status = nullptr;
  };
  auto add = [&](const float* src, const void* image, size_t at, int rows, int k) {
    if (n == MAX_PACK) flush();
    jobs.src[n] = src;
    jobs.dst[n] = static_cast<uint8_t*>(const_cast<void*>(image)) + at;
    jobs.rows[n] = (short)rows;
    jobs.k[n++] = (short)k;
  };
  for (int i = 0; i < ns; ++i) {
    const BnbSpatialWeights& w = s[i];
    add(w.qkv_w, w.packed, spatial_at(IM_QKV), 384, D);
    add(w.out_w, w.packed, spatial_at(IM_OUT), D, D);
    add(w.gate_w, w.packed, spatial_at(IM_GATE), F, D);
    add(w.up_w, w.packed, spatial_at(IM_UP), F, D);
    add(w.down_w, w.packed, spatial_at(IM_DOWN), D, F);
    if (bullets && w.kv_bullet_w) add(w.kv_bullet_w, w.packed, spatial_at(IM_KVB), 256, D);
  }
  for (int i = 0; i < nt; ++i) {
    const BnbTemporalWeights& w = t[i];
    const float* square[5] = {w.linear1_w, w.linear2_w, w.a_w, w.x_w, w.out_w};
    for (int k = 0; k < 5; ++k) add(square[k], w.packed, temporal_at(k), D, D);
    add(w.gate_w, w.packed, temporal_at(IM_GATE_T), F, D);
    add(w.up_w, w.packed, temporal_at(IM_UP_T), F, D);
    add(w.down_w, w.packed, temporal_at(IM_DOWN_T), D, F);
    if (fields) add(w.field_sub_w, w.packed, temporal_at(IM_FIELD), D, D);
    add(w.log_lambda, w.packed, temporal_at(IM_DECAY), D, 0);
  }
  flush();
  return cudaGetLastError() == cudaSuccess ? BNB_OK : BNB_ERR_LAUNCH;
}

int tiles_of(long long rows) { return (int)((rows + TILE - 1) / TILE); }
Image image(const void* packed, size_t at, int rows) { return {static_cast<const uint8_t*>(packed) + at, rows}; }

int project(Call& c, const float* x, const float* gain, const Image& w, float* out, long long rows) {
  const int tiles = tiles_of(rows), units = w.rows / 128, per = splits_of((long long)tiles * units, 4);
  const ProjectArgs a{x, gain, w, out, (int)rows, 128 / per, units * per, c.waits()};
  return c.launch(k_project, a, dim3((unsigned)(tiles * a.splits)), THREADS, SMEM, 1);
}
int post_half(Call& c, const float* o, const float* x, float* y, const float* gain, const Image& out, const Image& gate, const Image& up,
              const Image& down, int rows) {
  const int tiles = tiles_of(rows), cluster = splits_of(tiles, 8);
  const PostArgs a{o, x, y, gain, out, gate, up, down, rows, cluster, c.waits()};
  return c.launch(k_post, a, dim3((unsigned)(tiles * cluster)), THREADS, SMEM, cluster);
}

}  // namespace

size_t spatial_image_bytes() { return spatial_at(IM_KVB) + image_bytes(256, 128); }
size_t temporal_image_bytes() { return temporal_at(IM_DECAY) + 2 * D * sizeof(float); }

int step(const BnbSpatialWeights* spatial, const BnbTemporalWeights* temporal, int n_blocks, int n_spatial, int n_temporal,
         const float* x, const uint8_t* alive, const BnbBullets* bullets, float* y, const float* hidden_in, float* hidden_out,
         const uint8_t* reset_env, const BnbBatch& b, const Scratch& scratch, cudaStream_t st) {
  if (!configure()) return BNB_ERR_LAUNCH;
  Call c{st, scratch.status, tensor::host_status_word(st)};
  const EnvMap map = make_env_map(b);
  const int rows = b.total_tokens, fields = b.total_tokens - b.total_ships;
  int rc = pack(spatial, n_blocks * n_spatial, temporal, n_blocks * n_temporal, bullets != nullptr, fields > 0, c);
  const float* cur = x;
  for (int i = 0; i < n_blocks; ++i) {
    for (int j = 0; j < n_spatial; ++j) {
      const BnbSpatialWeights& w = spatial[i * n_spatial + j];
      const void* im = w.packed;
      if (!rc) rc = project(c, cur, w.norm1_w, image(im, spatial_at(IM_QKV), 384), scratch.qkv, rows);
      const bool cross = bullets && w.kv_bullet_w;
      const int slice = cross ? scratch.kvb_envs : b.n_envs;
      for (int e0 = 0; e0 < b.n_envs && !rc; e0 += slice) {
        const int ne = b.n_envs - e0 < slice ? b.n_envs - e0 : slice;
        AttendArgs a{scratch.qkv, alive, scratch.o, map, e0, nullptr, nullptr, 0};
        if (cross) {
          a.kvb = scratch.kvb;
          a.active = bullets->active;
          a.nb = bullets->per_env;
          rc = project(c, static_cast<const float*>(bullets->tokens) + (size_t)e0 * a.nb * D, w.norm_bullet_w,
                       image(im, spatial_at(IM_KVB), 256), scratch.kvb, (long long)ne * a.nb);
        }
        if (!rc) rc = c.launch(cross ? k_attend<true> : k_attend<false>, a, dim3((unsigned)ne, (unsigned)((HEADS * b.max_tokens_per_env + ATT_PAIRS - 1) / ATT_PAIRS)), ATT_THREADS, ATT_SMEM, 1);
      }
      if (!rc)
        rc = post_half(c, scratch.o, cur, y, w.norm2_w, image(im, spatial_at(IM_OUT), D), image(im, spatial_at(IM_GATE), F),
                       image(im, spatial_at(IM_UP), F), image(im, spatial_at(IM_DOWN), D), rows);
      if (rc) return rc;
      cur = y;
    }
    for (int j = 0; j < n_temporal; ++j) {
      const int slot = i * n_temporal + j;
      const size_t at = (size_t)slot * b.total_ships * 4 * D;
      const BnbTemporalWeights& w = temporal[slot];
      const void* im = w.packed;
      const int ship_tiles = tiles_of(b.total_ships), tiles = ship_tiles + tiles_of(fields), splits = splits_of(tiles, 4);
      if (!rc) {
        const FrontArgs a{cur, scratch.o, hidden_in + at, hidden_out + at, reset_env, map, ship_tiles, 128 / splits, splits, w,
                          image(im, temporal_at(IM_LIN1), D), image(im, temporal_at(IM_LIN2), D), image(im, temporal_at(IM_A), D),
                          image(im, temporal_at(IM_X), D), image(im, temporal_at(IM_FIELD), D),
                          reinterpret_cast<const float*>(static_cast<const uint8_t*>(im) + temporal_at(IM_DECAY)), c.waits()};
        rc = c.launch(k_front, a, dim3((unsigned)(tiles * splits)), THREADS, SMEM, 1);
      }
      if (!rc)
        rc = post_half(c, scratch.o, cur, y, w.norm2_w, image(im, temporal_at(IM_OUT_T), D), image(im, temporal_at(IM_GATE_T), F),
                       image(im, temporal_at(IM_UP_T), F), image(im, temporal_at(IM_DOWN_T), D), rows);
      if (rc) return rc;
      cur = y;
    }
  }
  return rc;
}

}  // namespace split
}  // namespace bnb
