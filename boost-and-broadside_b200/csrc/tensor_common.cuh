// Shared pieces of the tensor-core trunk kernels (sm_100a): the sublayer program a launch
// runs, the layout constants of the packed weight image, and the inline-PTX wrappers
// (tcgen05 / mbarrier / bulk copy / ldmatrix / mma.sync) both tile kernels are written with.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "common.cuh"

namespace bnb {
namespace tensor {

constexpr int D = 128;
constexpr int HEADS = 4;
constexpr int DH = 32;
constexpr int TILE = 128;
constexpr int CHUNK_BYTES = 16384;       // one weight chunk: up to 128 rows x 64 bf16
constexpr int N_SPATIAL_CHUNKS = 32;       // chunks of a spatial sublayer proper
constexpr int N_BULLET_CHUNKS = 4;         // kv_bullet: keys (2 K atoms), values (2 K atoms); zero when absent
constexpr int N_SPATIAL_IMAGE = N_SPATIAL_CHUNKS + N_BULLET_CHUNKS;
constexpr int N_TEMPORAL_CHUNKS = 36;
constexpr int MAX_SUBLAYERS = 8;

// SUB_SPATIAL_PRE / _POST split a spatial sublayer around a separate attention kernel
// (environments larger than one tile): PRE = norm1 + QKV to global scratch, POST = attention
// output from scratch + out_proj + norm2 + GatedMLP.
enum : int { SUB_SPATIAL = 0, SUB_TEMPORAL = 1, SUB_SPATIAL_PRE = 2, SUB_SPATIAL_POST = 3 };
enum : int { ST_TIMEOUT_FULL = 101, ST_TIMEOUT_EMPTY = 102, ST_TIMEOUT_ACC = 103 };

struct SubLayer {
  int type;
  const uint8_t* packed;
  const float* conv_w;
  const float* conv_b;
  const float* decay_log2;   // 8 * log2(sigmoid(log_lambda)), then half of a_b, half of x_b (D floats each), written by the pack kernel
  const float* hid_in;
  float* hid_out;
  __nv_bfloat16* qkv_out;        // PRE: (rows, 384) q|k|v, head-major inside each third
  const __nv_bfloat16* o_in;     // POST: (rows, 128) attention output
};

struct TrunkArgs {
  const float* x;
  float* y;
  const uint8_t* alive;
  const uint8_t* done;
  const uint8_t* reset_env;
  EnvMap map;
  int n_groups;       // replication of the batch for the spatial fold (T for a sequence)
  int t_loop;         // passes over a tile: timesteps walked inside the kernel (temporal programs of a sequence), or chunks of them
  int chunk;          // timesteps of a token in one tile (4, 8, 16 or 32), 0: tiles of one timestep
  int steps;          // timesteps of the sequence (with chunks)
  int n_sub;
  int n_tiles;
  int envs_per_tile;
  int env_tiles;      // tiles per group
  int has_fields;
  int flat_rows;      // 1: tiles are plain 128-row slices of the token rows (no attention inside)
  const int* tile_env_begin;  // ragged batches: range of each tile in tile_env_ids (+ end), else null
  const int* tile_env_ids;    // ragged batches: environments in tile order
  int* status;
  int* host_status;   // pinned host word that a wait which runs out writes its code to, or null
  // Test hooks of the bounded waits (0 / -1 in normal use): the poll limit of this launch, and the
  // ring operation of CTA 0 whose weight copy the fetching lane leaves out, so that the issuing
  // lane's wait for it runs out and the kernel has to drain and return with a status code.
  int poll_limit;
  int skip_op;
  int wide;      // x, y, every hidden state and the split path's buffers are 32-byte aligned
  int io_bf16;   // x and y hold bfloat16 (BNB_BF16_IO) instead of float32
  SubLayer sub[MAX_SUBLAYERS];
};
// Process-wide values of the two hooks, set by bnb_debug_wait_test and copied into every launch.
extern int g_debug_poll_limit;
extern int g_debug_skip_op;

// ------------------------------------------------------------------ PTX wrappers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: gives up after a number of polls, records `code` in the status word and lets the
// caller go on.  `aborted` points at four shared ints: [0] is set once any wait of the CTA has run
// out (later waits then give up after four polls, so the kernel drains quickly), [1] is the poll
// limit of this launch, [2..3] hold the address of the host's status word (or null).
constexpr int DEFAULT_POLL_LIMIT = 1 << 20;
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, int* status, volatile int* aborted, int code) {
  if (mbar_try_wait(bar, parity)) return;   // the common case costs one instruction
  // a missing weight copy stalls the other waits too: they poll twice as long, so that its code is first
  const int limit = aborted[0] ? 4 : code == ST_TIMEOUT_FULL ? aborted[1] : 2 * aborted[1];
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return;
  *aborted = 1;
  if (atomicCAS(status, 0, code) == 0) {   // the first code of the call is the one reported
    if (int* host = *reinterpret_cast<int* volatile*>(const_cast<int*>(&aborted[2]))) *static_cast<volatile int*>(host) = code;
  }
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// Instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr) : "memory");
}
// N consecutive columns of this thread's lane (N a multiple of 8, at most 64); no wait.
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&v)[N]) {
  static_assert(N % 8 == 0 && N <= 64, "column count");
  int done = 0;
  if constexpr (N >= 32) {
    tmem_ld32_nowait(taddr, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
    done = 32;
    if constexpr (N >= 64) {
      tmem_ld32_nowait(taddr + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
      done = 64;
    }
  }
  if constexpr ((N % 32) >= 16) {
    tmem_ld16_nowait(taddr + done, *reinterpret_cast<uint32_t(*)[16]>(&v[N - (N % 32)]));
    done += 16;
  }
  if constexpr ((N % 16) == 8) tmem_ld8_nowait(taddr + done, &v[N - 8]);
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  tmem_ld32_nowait(taddr, v);
  tmem_wait_ld();
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st8_nowait(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The first product of a sum.
__device__ __forceinline__ void mma_bf16_fresh(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Two floats in one 64-bit register pair: one instruction for two multiply-adds.
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float lo, float hi) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ F2 f2(float both) { return f2(both, both); }
__device__ __forceinline__ float2 halves(F2 a) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v)); return r; }
__device__ __forceinline__ F2 mul(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 add(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
// MUFU-based elementwise functions for the bf16 path.  Their results are rounded to bf16 (or
// feed products that are), so approximations a few 1e-4 relative are below the rounding.
__device__ __forceinline__ float tanh_fast(float v) {
  float r;
  asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float ex2_fast(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rcp_fast(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// 1 / v for the sum of softmax weights: the instruction and one Newton-Raphson step r + r (1 - v r), which squares its relative
// error.  Largest error over every float of [1, 256): 1.65 x 2^-24 without the step, 1.00 with it and by division.  NaN stays NaN.
__device__ __forceinline__ float reciprocal(float v) {
  const float r = rcp_fast(v);
  return fmaf(r, fmaf(-v, r, 1.0f), r);
}
__device__ __forceinline__ float sqrt_fast(float v) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// erf GELU as 0.5 x (1 + tanh(x (c1 + c3 x^2 + c5 x^4))): the inner polynomial is a minimax fit to x * Phi(x) (max abs error 2.5e-5, max
// relative error 1.2e-3 where |gelu| > 1e-2); beyond |x| = 10 its x^2 is held at 100, where it is positive and tanh saturates.
// gelu(2 h) * u for two elements, packed as two bf16: that polynomial in h = gate / 2 (an exact halving), GELU in
// half precision (11 mantissa bits against the 8 of the bf16 result; h * h saturates at 25 as there, an overflow to inf lands
// there too), one tanh.approx.f16x2; the product with u in float32.  Halving in the weights saves the
// multiplication by 0.5 and leaving u in float32 two conversions: 12 instructions instead of 14 for what the GatedMLP spends most of its issue slots on.
__device__ __forceinline__ uint32_t gelu_half_mul(uint32_t h0, uint32_t h1, uint32_t u0, uint32_t u1) {
  const __half2 h = __floats2half2_rn(__uint_as_float(h0), __uint_as_float(h1));
  const __half2 y = __hmin2(__hmul2(h, h), __float2half2_rn(25.0f));
  __half2 p = __hfma2(y, __float2half2_rn(-32 * 3.51516841e-4f), __float2half2_rn(8 * 3.70056464e-2f));
  p = __hfma2(y, p, __float2half2_rn(2 * 7.97507884e-1f));
  const __half2 a = __hmul2(h, p);
  uint32_t ti, to;
  ti = *reinterpret_cast<const uint32_t*>(&a);
  asm("tanh.approx.f16x2 %0, %1;" : "=r"(to) : "r"(ti));
  const __half2 t = *reinterpret_cast<const __half2*>(&to);
  float2 f = __half22float2(__hfma2(h, t, h));
  asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(f.x), "+f"(f.y) : "f"(__uint_as_float(u0)), "f"(__uint_as_float(u1)));
  return pack_bf16(f.x, f.y);
}
// gelu(2 h) of two elements in float32.
__device__ __forceinline__ F2 gelu_half(F2 h) {
  const float2 y = halves(mul(h, h));
  const F2 y2 = f2(fminf(y.x, 25.0f), fminf(y.y, 25.0f));
  const float2 a = halves(mul(h, fma(y2, fma(y2, f2(-32 * 3.51516841e-4f), f2(8 * 3.70056464e-2f)), f2(2 * 7.97507884e-1f))));
  return fma(h, f2(tanh_fast(a.x), tanh_fast(a.y)), h);
}
// sigmoid(2 v) of two elements, each rounded to bfloat16.
__device__ __forceinline__ F2 sigmoid_twice_bf16(F2 v) {
  const float2 h = halves(v);
  const float2 g = halves(fma(f2(tanh_fast(h.x), tanh_fast(h.y)), f2(0.5f), f2(0.5f)));
  return f2(round_bf16(g.x), round_bf16(g.y));
}

__device__ __forceinline__ F2 unpack_bf16(uint32_t v) { return f2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u)); }
__device__ __forceinline__ uint32_t pack_bf16(F2 a) { const float2 v = halves(a); return pack_bf16(v.x, v.y); }
// GELU(norm) of two values: rounded to bfloat16 behind the norm (h inv gain) and behind the GELU, the fit above.  half_gain: half
// the gain, since gelu_half takes half its argument and a halving commutes with the rounding.
__device__ __forceinline__ uint32_t activation(uint32_t h, F2 inv, F2 half_gain) {
  return pack_bf16(gelu_half(unpack_bf16(pack_bf16(mul(mul(unpack_bf16(h), inv), half_gain)))));
}
// Product of two pairs of bfloat16, rounded once.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(c) : "r"(a), "r"(b));
  return c;
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

// Byte offset of the 16-byte group holding columns [8*c8, 8*c8+8) of row r inside a
// 128-row x 64-column bf16 atom with the 128-byte swizzle.
__device__ __forceinline__ uint32_t swz(int r, int c8) { return (uint32_t)(r * 128 + ((c8 ^ (r & 7)) << 4)); }

// ------------------------------------------------------------------ programmatic dependence (launch_after.h)
//
// let_next_start comes after the CTA's tensor memory is allocated (a successor on the same SM that allocated it first would
// wait for this kernel, and this kernel for it).  In the kernels of launch_after.h it comes before wait_for_previous, and nothing
// in global memory is read or written before that; the float32 step's chain (split_kernels.cu) has the other order, and reads early.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ------------------------------------------------------------------ issuing from a whole warp
//
// A warp that issues tensor-core work runs with the same values in every lane and lets one elected lane
// execute the instruction: its operands then stay in uniform registers.

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p;
}
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
// tcgen05.mma with the shared-memory descriptors built from 32-bit halves inside the asm block
// (K-major, 128-byte swizzle, 8-row groups 1024 B apart: the high word is a constant); A in shared
// memory, or (TMEM_A) in tensor memory: lane = row, a 32-bit column = two consecutive k as bfloat16.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
template <bool TMEM_A>
__device__ __forceinline__ void mma_one(uint32_t elected, uint32_t d_tmem, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  if constexpr (TMEM_A)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(0x40004040u), "r"(elected) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(0x40004040u), "r"(elected) : "memory");
}
__device__ __forceinline__ void tc_commit_if(uint32_t elected, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"(elected) : "memory");
}

// The fused one-CTA-per-SM kernel (pipelined_tile_kernel.cu): programs of whole-environment tiles
// made of SUB_SPATIAL and SUB_TEMPORAL sublayers only.
int launch_pipelined(const TrunkArgs& a, cudaStream_t st);

}  // namespace tensor
}  // namespace bnb
