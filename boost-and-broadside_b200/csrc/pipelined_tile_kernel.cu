// The fused trunk kernel for sm_100a: one CTA per SM walks a tile of 128 token rows (whole
// environments, or several timesteps of a token) through a program of spatial and temporal sublayers, with the residual
// stream resident in tensor memory and four warp roles that only meet at mbarriers:
//
//   16 epilogue warps   four threads per tile row (thread (row, part): TMEM lane = row, a quarter
//                       of whatever columns are being read).  RMSNorm, q|k|v staging, attention
//                       (mma.sync), gelu(gate) * up, causal conv, RG-LRU gates and state update.
//   1 issuing warp      issues every tcgen05.mma but the down projections.  It waits for "operand ready" (the
//                       epilogue warps arrive on an mbarrier after fence.proxy.async) and for
//                       "chunk landed" (the bulk copy's complete_tx), and signals "accumulator
//                       ready" / "slot free" with tcgen05.commit.
//   1 down warp         issues the down projections, and prepares the next pass: its row table, its tokens and the
//                       recurrent state on their way to the SM.
//   1 fetching warp     streams the pre-tiled weight image through a ring of nine 16 KB
//                       slots with cp.async.bulk, following a static schedule.
//
//   TMEM  [0,128)    residual stream, fp32, lane = tile row (out_proj, linear_out and down_proj
//                    accumulate straight into it)
//         [128,512)  three 128-column accumulators.  q, k and v fill them in one round; the GatedMLP uses two, one for
//                    each half of the epilogue warps (even and odd chunks of 64 hidden columns), and the third for four
//                    buffers of gated products, the A operands of the down projections.
//
//   SMEM  A (32 KB)  normed activations (K-major, 128-byte swizzle); rows of the result on their way out.
//         P (2 x 16 KB)  q of all heads, then the attention output; RG-LRU branch; the next pass's tokens.
//         KV (64 KB)  keys and values of all heads during attention, four more ring slots otherwise.
//         Ring (5 x 16 KB).  Row tables of two passes.
//
// Every mbarrier wait is bounded: a wait that runs out records a code in the status word, later
// waits give up at once, and the kernel drains and returns.
//
// Reference arithmetic: models/yemong/attention.py:76-169, models/yemong/griffin.py:67-317.
#include "launch_after.h"
#include "tensor_common.cuh"
#include "tensor_kernels.h"

namespace bnb {
namespace tensor {
namespace pipe {

constexpr int EPI_WARPS = 16;
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int MMA_WARP = EPI_WARPS;        // every product but the down projections
constexpr int DOWN_WARP = EPI_WARPS + 1;   // the down projections
constexpr int LOAD_WARP = EPI_WARPS + 2;
constexpr int THREADS = EPI_THREADS + 96;
// Weight ring: three pair slots (32 KB: both K atoms of one 128-row weight block, consumed by
// eight MMAs) and three single slots (16 KB: one down-projection chunk).  Slots 0, 1 (pairs) and
// 3 (single) are dedicated; 2, 4 and 5 live in the key/value staging area and carry weights only
// while no attention runs.
constexpr int N_SLOTS = 6;
constexpr int RING_BYTES = 5 * CHUNK_BYTES;

constexpr int OFF_A = 0;
constexpr int OFF_P = 32768;
constexpr int OFF_KV = 65536;
constexpr int OFF_RING = 131072;
constexpr int OFF_SS = OFF_RING + RING_BYTES;                   // partial sums of squares [4][128]
// What the rows of a pass are, twice (the pass at work and the next one): Place[128], then the blocks of 16 queries (first
// row | first row of the environment << 8 | its tokens less one << 16 | its tokens << 24; environments of up to 8 tokens
// share a block, and the second number is the block's rows less one), then the attention bias of each row as a key
// (float, 16 of slack), then the number of blocks.
constexpr int OFF_TAB = OFF_SS + 2048;
constexpr int TAB_BLOCKS = 2048, TAB_BIAS = TAB_BLOCKS + 512, TAB_COUNT = TAB_BIAS + 576, TAB_BYTES = TAB_COUNT + 16;
static_assert(TAB_BYTES % 16 == 0, "16-byte accesses");
constexpr int OFF_BAR = OFF_TAB + 2 * TAB_BYTES;
constexpr int SMEM_BYTES = OFF_BAR + 256 + 1024;

// mbarrier indices
// OP0: operand ready (epilogue warps -> issuing warp).  REL[g]: gate|up of a chunk have been read from the accumulator of group
// g (its eight warps -> issuing warp).  FFN[b]: a chunk's product stands in product buffer b (the eight warps that own the
// chunk -> down-projection warp); PFREE[b]: its down projection is complete, twice in a GatedMLP.  KVREL: the key/value area
// may take weights again (epilogue warps -> fetching warp).  FULL[s]: the weights of slot s have landed.
// DONE[s]: the MMAs that read slot s are complete (tcgen05.commit) -- the fetching warp takes it as
// "slot free", the epilogue warps as "accumulator ready" for gate|up of one chunk, whose slot is not
// used again before they have seen it.
// ACC: every MMA of a round is complete (one more commit per round).
// EARLY: the first half of a temporal sublayer's gates is.  PARK: linear2's accumulator has been read (epilogue warps ->
// issuing warp); FIELD: field_sub, multiplied into it then, is complete.  XFULL: the row table of the next pass is
// written and its tokens have landed in the P area (down-projection warp -> epilogue warps); XFREE: the tokens have been read, and
// nobody works on the pass before any more.  DRAIN: every MMA of the
// CTA is complete (once per issuing warp, at the end).
enum : int { B_OP0 = 0, B_FFN0, B_FFN3 = B_FFN0 + 3, B_REL0, B_REL1, B_KVREL, B_PARK, B_XFREE, B_XFULL, B_DRAIN, B_ACC, B_EARLY, B_FIELD, B_PFREE0, B_FULL0 = B_PFREE0 + 4, B_DONE0 = B_FULL0 + N_SLOTS, B_COUNT = B_DONE0 + N_SLOTS };
static_assert(B_COUNT * 8 + 8 <= 256, "barrier area");

constexpr uint32_t COL_RESID = 0;
constexpr uint32_t COL_ACC0 = 128, COL_ACC1 = 256, COL_ACC2 = 384;
constexpr uint32_t TMEM_COLS = 512;

enum : int { ST_TIMEOUT_FULL = 101, ST_TIMEOUT_FREE = 102, ST_TIMEOUT_ACC = 103, ST_TIMEOUT_OPERAND = 104 };

// Optional cycle accounting (compile with -DBNB_TIMING): thread 0 (an epilogue thread), the
// issuing lane and the fetching lane of every CTA add up the cycles they spend in each phase and
// store them behind the status word: 32 counters per CTA from byte 256 on.
// Of a temporal sublayer: TE_TAPS the first taps asked for, TE_B1 linear1's result into the A operand, TE_SYNC the barrier
// behind it, TE_CONV the conv with its waits for taps, TE_PARK the state asked for and linear2's GELU, TE_GATES
// gates, state update and the state's rows, TE_FIELDS field rows.  TE_POST: everywhere an operand is posted.
enum : int { TE_ACC_WAIT = 0, TE_FFN_ACC_WAIT, TE_FFN_MATH, TE_NORM, TE_STAGE, TE_ATTN, TE_TAPS, TE_B1, TE_SYNC, TE_CONV, TE_PARK,
             TE_GATES, TE_FIELDS, TE_POST, TE_IO, TE_TOTAL, TM_FULL_WAIT, TM_OP_WAIT, TM_ISSUE, TM_TOTAL, TL_FREE_WAIT, TL_KV_WAIT, TL_TOTAL, T_COUNT };
#ifdef BNB_TIMING
static_assert(T_COUNT <= 32, "counters of a CTA");
// In shared memory, 32 bits each: as arrays of every thread they lay in local memory, and the kernel took half as long again.
__device__ __forceinline__ uint32_t* time_counters() { __shared__ uint32_t counters[32]; return counters; }
__device__ __forceinline__ void count_time(int slot, uint32_t cycles) {
  if (threadIdx.x == 0 || threadIdx.x == 32 * MMA_WARP || threadIdx.x == 32 * LOAD_WARP) time_counters()[slot] += cycles;
}
__device__ __forceinline__ uint32_t cycles_now() { return (uint32_t)clock64(); }
#define T_BEGIN() const uint32_t _t0 = cycles_now()
#define T_END(slot) count_time(slot, cycles_now() - _t0)
#define T_MARK(name) uint32_t name = cycles_now()
#define T_RESET(name) name = cycles_now()
#define T_SINCE(slot, name) do { const uint32_t _n = cycles_now(); count_time(slot, _n - name); name = _n; } while (0)
#else
#define T_BEGIN()
#define T_END(slot)
#define T_MARK(name)
#define T_RESET(name)
#define T_SINCE(slot, name)
#endif

// Optional event trace (compile with -DBNB_TRACE): CTA 0 records (event id, clock) pairs of one
// epilogue thread, the issuing lane and the fetching lane from byte 16384 of the status area on,
// 1500 events per role.
#ifdef BNB_TRACE
struct Trace { unsigned long long* buf; int n; };
__device__ __forceinline__ void trace_init(Trace& t, int* status, int role) {
  t.buf = reinterpret_cast<unsigned long long*>(status) + 2048 + role * 1500;
  t.n = blockIdx.x == 0 ? 0 : 1500;
}
__device__ __forceinline__ void trace(Trace& t, int id) {
  if (t.n < 1500) t.buf[t.n++] = ((unsigned long long)id << 48) | ((unsigned long long)clock64() & 0xFFFFFFFFFFFFull);
}
#define TRACE(t, id) trace(t, id)
#else
#define TRACE(t, id)
#endif

// One ring operation as the fetching warp needs it: source (64 bits), place in shared memory (relative to its start, a multiple
// of 1 KB) | slot (bits 0-2) | wait for the key/value area first (8), bytes.  Resolved once at kernel start, a thread per
// operation: the warp's time per operation bounds the GatedMLP (see the fetching loop).
constexpr int MAX_SCHED = MAX_SUBLAYERS * 22;
static_assert(MAX_SCHED <= THREADS, "one thread writes one entry");

// Ring operations of a sublayer.  Every sublayer starts at pair slot 0 and single slot 3 and takes them in turn, so that
// all roles know the slot of an operation from its place in the sublayer.
//   spatial    q, k, v -> pairs 0 1 2; out_proj -> 0 (dedicated: fetched while the attention runs); GatedMLP from pair 1 on,
//              whose second gate|up is the first operation that goes to the key/value area and waits for it
//   PRE        q, k, v;  POST  out_proj and the GatedMLP
//   temporal   linear2, linear1 -> 0 1; gates -> 2 0; field_sub -> 1 (left out without fields); linear_out -> 2; GatedMLP from 0 on
// GatedMLP with image base b: gate|up of chunk c are chunks b + 3c, b + 3c + 1 (a pair), its down projection is
// b + 3c + 2 (a single); fetched in the order GU0 GU1 GU2 D0 GU3 D1 GU4 D2 ... GU7 D5 D6 D7.
constexpr uint32_t SPATIAL_FFN_PAIR = 1, TEMPORAL_FFN_PAIR = 0;   // pair slot of gate|up of chunk 0
constexpr int FFN_OPS = 16;
__device__ __forceinline__ uint32_t pair_offset(uint32_t slot) { return slot == 2 ? OFF_KV : OFF_RING + slot * 2 * CHUNK_BYTES; }
__device__ __forceinline__ uint32_t single_offset(uint32_t i) { return i == 0 ? OFF_RING + 4 * CHUNK_BYTES : OFF_KV + (1 + i) * CHUNK_BYTES; }
__device__ __forceinline__ uint32_t slot_offset(uint32_t slot) { return slot < 3 ? pair_offset(slot) : single_offset(slot - 3); }
__device__ __forceinline__ int sublayer_ops(int type, bool has_fields) {
  return type == SUB_SPATIAL ? 4 + FFN_OPS : type == SUB_SPATIAL_PRE ? 3 : type == SUB_SPATIAL_POST ? 1 + FFN_OPS : (has_fields ? 6 : 5) + FFN_OPS;
}
__device__ __forceinline__ uint4 sched_entry(const SubLayer& s, int op, bool has_fields) {
  int slot, chunk, base;
  bool pair = true, kvwait = false;
  int f;   // place inside the GatedMLP, negative before it
  uint32_t first;
  if (s.type == SUB_TEMPORAL) {
    f = op - (has_fields ? 6 : 5);
    const int k = has_fields || op < 4 ? op : op + 1;   // 0 linear2, 1 linear1, 2 and 3 gates, 4 field_sub, 5 linear_out
    slot = k % 3;
    chunk = 2 * k;
    base = 12;
    first = TEMPORAL_FFN_PAIR;
  } else {
    const int k = s.type == SUB_SPATIAL_POST ? op + 3 : op;   // 0 q, 1 k, 2 v, 3 out_proj
    f = k - 4;
    slot = k % 3;
    chunk = 2 * k;
    base = 8;
    first = SPATIAL_FFN_PAIR;
  }
  if (f >= 0) {
    const int k = f - 3;
    const int c = f < 3 ? f : k < 10 ? ((k & 1) ? 3 + (k >> 1) : k >> 1) : k - 5;
    pair = f < 3 || (k < 10 && (k & 1));
    slot = pair ? (int)(first + c) % 3 : 3 + c % 3;
    chunk = base + 3 * c + (pair ? 0 : 2);
    kvwait = s.type == SUB_SPATIAL && f == 1;
  }
  const unsigned long long src = reinterpret_cast<unsigned long long>(s.packed + (size_t)chunk * CHUNK_BYTES);
  return make_uint4((uint32_t)src, (uint32_t)(src >> 32), slot_offset((uint32_t)slot) | (uint32_t)slot | (kvwait ? 8u : 0u), pair ? 2u * CHUNK_BYTES : (uint32_t)CHUNK_BYTES);
}

// Bounded wait of this kernel: as mbar_wait, but a wait that runs out only leaves its code in the CTA's abort word, which the
// last thread out reports; two dozen waits are inlined here, and the kernel's code is what its warps stall on
// in every phase they meet for the first time.  aborted[0]: 0, or the first code (-1: the call had failed before).
__device__ __forceinline__ void wait_bar(uint32_t bar, uint32_t parity, volatile int* aborted, int code) {
  if (mbar_try_wait(bar, parity)) return;
  const int limit = aborted[0] ? 4 : code == ST_TIMEOUT_FULL ? aborted[1] : 2 * aborted[1];
#pragma unroll 1
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return;
  if (aborted[0] == 0) aborted[0] = code;
}

// What one tile row is in a pass (16 bytes of the row table).
struct Place {
  int hrow;        // row of the packed hidden state, -1 for field / invalid rows
  uint32_t flags;  // P_*, and from bit 8 on the stored conv lags still inside the current episode (0..3)
  int trow;        // token row of the call, -1 for rows outside every environment
  int unused;
};
enum : uint32_t { P_VALID = 1, P_ZERO_IN = 2 /* incoming state taken as zero (reset_env) */, P_BOUNDARY = 4, P_LAST = 8 /* its step's state is stored */ };

// What a launch's program may hold; the code it does not need costs registers and instruction fetches.
//   ANY    every kind of sublayer
//   WHOLE  whole sublayers on tiles of whole environments, most calls by far
//   STEPS  one temporal sublayer of a sequence on tiles of 128 / C tokens x C consecutive timesteps (TrunkArgs::chunk); a CTA
//          walks the chunks of its tokens in order
enum : int { ANY = 0, WHOLE = 1, STEPS = 2 };

// ------------------------------------------------------------------ epilogue side

struct Epi {
#ifdef BNB_TRACE
  Trace tr;
#endif
  uint8_t* smem;
  uint32_t sbase;       // shared address of smem
  uint32_t bars;        // shared address of the barrier array
  uint32_t lane_addr;   // tensor-memory address of this thread's lane, column 0
  uint32_t par;         // phase bits of the pair slots' DONE barriers (0..2), of ACC (8), EARLY (10), FIELD (11)
                        // and XFULL (12)
  int row, part;
  bool wide;            // 32-byte accesses: every row pointer is aligned for them
  volatile int* aborted;
  const uint8_t* tab;   // the row table of this pass
  float* ss_part;
};

// "My share of the operand is written and my reads of the accumulator are done."
__device__ __forceinline__ void post(Epi& e, int bar) {
  TRACE(e.tr, 200 + bar);
  T_BEGIN();
  fence_proxy_async();
  tc_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(e.bars + 8 * bar);
  T_END(TE_POST);
  TRACE(e.tr, 210 + bar);
}
// The epilogue threads keep one phase bit per pair slot and flip it for every pair operation of the
// schedule, whether they wait for it or not.
//
// wait_acc: every MMA issued so far is complete (a commit on ACC ends every round).
__device__ __forceinline__ void wait_acc(Epi& e) {
  T_BEGIN();
  wait_bar(e.bars + 8 * B_ACC, (e.par >> 8) & 1u, e.aborted, ST_TIMEOUT_ACC);
  e.par ^= 1u << 8;
  tc_fence_after();
  T_END(TE_ACC_WAIT);
  TRACE(e.tr, 110);
}
// The first half of a temporal sublayer's gates, read while the others are multiplied; field_sub.
// Every thread waits for each of its phases before it posts what the next one is issued after.
__device__ __forceinline__ void wait_other(Epi& e, int bar, uint32_t bit) {
  T_BEGIN();
  wait_bar(e.bars + 8 * bar, (e.par >> bit) & 1u, e.aborted, ST_TIMEOUT_ACC);
  e.par ^= 1u << bit;
  tc_fence_after();
  T_END(TE_ACC_WAIT);
}
__device__ __forceinline__ void wait_early(Epi& e) { wait_other(e, B_EARLY, 10); }
__device__ __forceinline__ void wait_field(Epi& e) { wait_other(e, B_FIELD, 11); }
// wait_round: a round whose pair operations took an odd number of turns on the slots of `flips`, then a commit on ACC.
__device__ __forceinline__ void wait_round(Epi& e, uint32_t flips) {
  wait_acc(e);
  e.par ^= flips;
}
// wait_op: gate|up of one chunk.  A thread that skips operations of a slot must not find the slot a phase
// behind or two ahead: it waits only when an operation issued after the skipped one is known to be
// complete (MMAs complete in order), and the slot's next one is issued only after its post.
__device__ __forceinline__ void wait_op(Epi& e, uint32_t slot) {
  T_BEGIN();
  wait_bar(e.bars + 8 * (B_DONE0 + slot), (e.par >> slot) & 1u, e.aborted, ST_TIMEOUT_ACC);
  tc_fence_after();
  T_END(TE_FFN_ACC_WAIT);
  TRACE(e.tr, 100);
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }

// Eight floats of one row per thread.  Threads own rows here, so every request of a warp touches 32 lines
// whatever its width: 32-byte accesses (where the pointers allow them) make it half as many requests as
// 16-byte ones.  In a sequence of 32 steps, whose state is read and written at every step, that is 4 % of
// the time (7442 -> 7153 us at 4096 x 8 tokens).
__device__ __forceinline__ void load8(float (&v)[8], const float* p, bool wide) {
  if (wide) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p) : "memory");
  } else {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(p) : "memory");
  } else {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

__device__ __forceinline__ void load4(float4& v, const float* p) {
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
}
__device__ __forceinline__ void store4(float* p, const float4& v) {
  asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
}

// residual (TMEM) -> x * rsqrt(mean x^2 + eps) -> bf16 A operand (the RMSNorm gain is in the weights)
__device__ __forceinline__ void norm_to_A(Epi& e) {
  TRACE(e.tr, 300);
  T_BEGIN();
  uint32_t v[32];
  tmem_ld32(e.lane_addr + COL_RESID + e.part * 32, v);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float a = __uint_as_float(v[i]);
    ss = fmaf(a, a, ss);
  }
  e.ss_part[e.part * TILE + e.row] = ss;
  // the four warps that share these 32 rows exchange partial sums (named barriers 3..6)
  asm volatile("bar.sync %0, 128;" ::"r"(3 + ((threadIdx.x >> 5) & 3)) : "memory");
  ss = (e.ss_part[e.row] + e.ss_part[TILE + e.row]) + (e.ss_part[2 * TILE + e.row] + e.ss_part[3 * TILE + e.row]);
  const float inv = rsqrtf(ss * (1.0f / D) + kRmsEps);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int col = e.part * 32 + q * 8;
    const uint32_t* s = &v[q * 8];
    uint4 o;
    o.x = pack_bf16(__uint_as_float(s[0]) * inv, __uint_as_float(s[1]) * inv);
    o.y = pack_bf16(__uint_as_float(s[2]) * inv, __uint_as_float(s[3]) * inv);
    o.z = pack_bf16(__uint_as_float(s[4]) * inv, __uint_as_float(s[5]) * inv);
    o.w = pack_bf16(__uint_as_float(s[6]) * inv, __uint_as_float(s[7]) * inv);
    *reinterpret_cast<uint4*>(e.smem + OFF_A + (col >> 6) * CHUNK_BYTES + swz(e.row, (col & 63) >> 3)) = o;
  }
  // the partial sums are read again by the next norm only after at least one full barrier
  T_END(TE_NORM);
}

__device__ __forceinline__ F2 acc_pair(const uint32_t* v) { return f2(__uint_as_float(v[0]), __uint_as_float(v[1])); }
__device__ __forceinline__ uint4 pack8(const uint32_t* s) {
  return make_uint4(pack_bf16(__uint_as_float(s[0]), __uint_as_float(s[1])), pack_bf16(__uint_as_float(s[2]), __uint_as_float(s[3])),
                    pack_bf16(__uint_as_float(s[4]), __uint_as_float(s[5])), pack_bf16(__uint_as_float(s[6]), __uint_as_float(s[7])));
}

// GatedMLP on the A operand (already normed and posted on OP0): residual += down(gelu(gate) * up).
// Two groups of eight warps take turns (parts 0, 1 the even chunks, parts 2, 3 the odd ones), so that one group's waits and
// tensor-memory latencies hide behind the other's arithmetic.  A group has an accumulator of its own: gate / 2 (the image
// holds half the gate weights) in columns [0,64), up in [64,128); a thread owns 32 of the 64 hidden columns of its row,
// columns [32 (part & 1), +32).  As soon as both are in registers the accumulator takes the group's next chunk.
//
// The gated product becomes the A operand of the down projection in tensor memory, in one of four buffers of 32 columns
// (column = two k as bfloat16), so that gate|up of a later chunk needn't wait for it: with the product over the gate columns it
// had been read from, three accumulators in turn, a chunk was the third of a chain of 2 700 cycles (product, commit, arithmetic,
// post, down projection, commit).
__device__ __forceinline__ void gated_product(const uint32_t (&gv)[16], const uint32_t (&uv)[16], uint32_t dst) {
  uint32_t w8[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w8[j] = gelu_half_mul(gv[2 * j], gv[2 * j + 1], uv[2 * j], uv[2 * j + 1]);
  tmem_st8_nowait(dst, w8);
}
__device__ __forceinline__ void ffn(Epi& e, uint32_t slot) {   // slot: pair slot of chunk 0
  const uint32_t group = e.part >> 1;
  const uint32_t acc = e.lane_addr + COL_ACC0 + group * 128 + (e.part & 1) * 32;
  if (group) {   // past chunk 0
    e.par ^= 1u << slot;
    slot = slot == 2 ? 0 : slot + 1;
  }
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    // gate|up of chunk 2 i + group; the slot's previous operation came before those of the two chunks in between
    wait_op(e, slot);
    T_BEGIN();
    const uint32_t buffer = 2 * (i & 1) + group;
    uint32_t gv[16], uv[16], gw[16], uw[16];
    tmem_ld16_nowait(acc, gv);
    tmem_ld16_nowait(acc + 64, uv);
    tmem_ld16_nowait(acc + 16, gw);
    tmem_ld16_nowait(acc + 80, uw);
    tmem_wait_ld();
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(e.bars + 8 * (B_REL0 + group));
    // the buffer's previous product has been multiplied (its next one is this, so no phase is missed)
    if (i >= 2) wait_bar(e.bars + 8 * (B_PFREE0 + buffer), 0, e.aborted, ST_TIMEOUT_ACC);
    const uint32_t dst = e.lane_addr + COL_ACC2 + 32 * buffer + 16 * (e.part & 1);
    gated_product(gv, uv, dst);
    gated_product(gw, uw, dst + 8);
    tmem_wait_st();
    T_END(TE_FFN_MATH);
    // nothing of this operand is in shared memory: no proxy fence
    TRACE(e.tr, 201);
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(e.bars + 8 * (B_FFN0 + buffer));
    // two operations further: chunks c + 1 and c + 2, whose slots are this one's successors
    e.par ^= 1u << slot;
    slot = slot == 2 ? 0 : slot + 1;
    e.par ^= 1u << slot;
    slot = slot == 2 ? 0 : slot + 1;
  }
  if (group) e.par ^= 1u << (slot == 0 ? 2 : slot - 1);   // there is no chunk 8
  wait_acc(e);   // residual complete: every down projection
}

// Attention of every head and environment of the tile from the staged q (P area), k and v (KV
// area), all in the swizzled operand layout (128 rows x 64 bf16 atoms; head h sits in atom h / 2,
// columns 32 (h % 2) ..).  The four warps of part h serve head h, which they have staged themselves,
// and take turns at the blocks of up to 16 query rows (each head from another warp on: warp & 3 is the scheduler).
// Output: bf16 into the P area as the A operand of out_proj, each block over its own q.
//
// Environments of up to 16 tokens need no running maximum, and those of up to 8 share a block (keys of another environment score
// -inf): 32 steps of 4096 x 8
// tokens 5 730 -> 5 400 us.  The division's code took 1.5 % of a step, `reciprocal` is as exact.

// A block of queries whose environments' keys are the block's own rows: block = first row | .. | rows less one << 16 | tokens of
// an environment << 24.  False, and nothing written: it holds several environments and a value that is not finite.  Keys of
// another environment have weight 0, but 0 times such a value is NaN, so the caller takes its environments one by one.
__device__ __forceinline__ bool attend_block(const Epi& e, uint32_t block) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t atom = (uint32_t)(e.part >> 1) * CHUNK_BYTES;
  const int c8h = (e.part & 1) * 4;
  const uint32_t sQ = e.sbase + OFF_P + atom, sK = e.sbase + OFF_KV + atom, sV = sK + 2 * CHUNK_BYTES;
  const float* key_bias = reinterpret_cast<const float*>(e.tab + TAB_BIAS);
  const float c2 = 0.17677669529663687f * 1.4426950408889634f;  // log2(e) / sqrt(32): scores in the log2 domain
  const int r0 = block & 255, n = (int)(block >> 16 & 255) + 1, size = (int)(block >> 24), last = r0 + n - 1;
  uint32_t qa[2][4], kf[2][4], vf[2][4];
  {
    const int row = min(r0 + (lane & 7) + ((lane >> 3) & 1) * 8, last), krow = min(r0 + (lane >> 4) * 8 + (lane & 7), last);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      ldsm_x4(sQ + swz(row, c8h + ks * 2 + (lane >> 4)), qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
      ldsm_x4(sK + swz(krow, c8h + ks * 2 + ((lane >> 3) & 1)), kf[ks][0], kf[ks][1], kf[ks][2], kf[ks][3]);
    }
#pragma unroll
    for (int np = 0; np < 2; ++np) ldsm_x4_t(sV + swz(row, c8h + np * 2 + (lane >> 4)), vf[np][0], vf[np][1], vf[np][2], vf[np][3]);
  }
  float sc[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) sc[nt][i] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    mma_bf16(sc[0], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kf[ks][0], kf[ks][1]);
    mma_bf16(sc[1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kf[ks][2], kf[ks][3]);
  }
  // first key of the environment of query g, g + 8
  const float per = rcp_fast((float)size);
  const int lo0 = (int)(((float)min(g, n - 1) + 0.5f) * per) * size, lo1 = (int)(((float)min(g + 8, n - 1) + 0.5f) * per) * size;
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j = nt * 8 + 2 * t + i;
      // a dead key's bias (kMaskedScore) swallows its score: weight exactly 0 unless every key is dead, then uniform
      const float bj = key_bias[r0 + j];
      sc[nt][i] = (unsigned)(j - lo0) < (unsigned)size ? fmaf(sc[nt][i], c2, bj) : -INFINITY;
      sc[nt][2 + i] = (unsigned)(j - lo1) < (unsigned)size ? fmaf(sc[nt][2 + i], c2, bj) : -INFINITY;
      m0 = fmaxf(m0, sc[nt][i]);
      m1 = fmaxf(m1, sc[nt][2 + i]);
    }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
  }
  float l0 = 0.f, l1 = 0.f;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      sc[nt][i] = ex2_fast(sc[nt][i] - m0);
      sc[nt][2 + i] = ex2_fast(sc[nt][2 + i] - m1);
      l0 += sc[nt][i];
      l1 += sc[nt][2 + i];
    }
  const uint32_t a0 = pack_bf16(sc[0][0], sc[0][1]), a1 = pack_bf16(sc[0][2], sc[0][3]);
  const uint32_t a2 = pack_bf16(sc[1][0], sc[1][1]), a3 = pack_bf16(sc[1][2], sc[1][3]);
  float acc[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
    mma_bf16(acc[nt], a0, a1, a2, a3, vf[nt >> 1][2 * (nt & 1)], vf[nt >> 1][2 * (nt & 1) + 1]);
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, o);
    l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  }
  // The look costs nothing here, behind the sums (8192 x 12 tokens 549 us; before the scores it held them up, 560).
  if (size < n) {
    uint32_t zero = 0u;   // 0 v + 0 v + ..: not 0 once a value is not finite
#pragma unroll
    for (int i = 0; i < 8; ++i) zero = fma_bf16x2(vf[i >> 2][i & 3], 0u, zero);
    if (__builtin_expect(__any_sync(0xffffffffu, zero != 0u), 0)) return false;
  }
  const float i0 = reciprocal(l0), i1 = reciprocal(l1);
  uint8_t* po = e.smem + OFF_P + atom;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    if (g < n) *reinterpret_cast<uint32_t*>(po + swz(r0 + g, c8h + nt) + t * 4) = pack_bf16(acc[nt][0] * i0, acc[nt][1] * i0);
    if (g + 8 < n) *reinterpret_cast<uint32_t*>(po + swz(r0 + g + 8, c8h + nt) + t * 4) = pack_bf16(acc[nt][2] * i1, acc[nt][3] * i1);
  }
  return true;
}

__device__ __forceinline__ void attention(Epi& e, int n_items) {
  TRACE(e.tr, 310);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int h = e.part;
  const uint32_t atom = (uint32_t)(h >> 1) * CHUNK_BYTES;
  const int c8h = (h & 1) * 4;
  const uint32_t sQ = e.sbase + OFF_P + atom, sK = e.sbase + OFF_KV + atom, sV = sK + 2 * CHUNK_BYTES;
  const float* key_bias = reinterpret_cast<const float*>(e.tab + TAB_BIAS);
  const uint32_t* blocks = reinterpret_cast<const uint32_t*>(e.tab + TAB_BLOCKS);
  const float c2 = 0.17677669529663687f * 1.4426950408889634f;  // log2(e) / sqrt(32): scores in the log2 domain
  for (int it = (warp + h) & 3; it < n_items; it += EPI_WARPS / 4) {
    const uint32_t block = blocks[it];
    if ((block >> 16 & 255) < 16 && attend_block(e, block)) continue;
    // larger environments, and those of a block that is taken apart, one after the other: keys are walked in blocks of 16 with a
    // running maximum
    const int n = max((int)(block >> 24), 1);   // tokens of the environment (0 may stand there after a wait has run out)
    const int end = (int)(block & 255) + (int)(block >> 16 & 255);
    int r0 = block & 255, e0 = block >> 8 & 255;   // first row; first tile row of the environment
#pragma unroll 1
    do {
      const int last = e0 + n - 1;
      uint32_t qa[2][4];
      {
        const int row = min(r0 + (lane & 7) + ((lane >> 3) & 1) * 8, last);
  #pragma unroll
        for (int ks = 0; ks < 2; ++ks)
          ldsm_x4(sQ + swz(row, c8h + ks * 2 + (lane >> 4)), qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);
      }
      const int nkb = (n + 15) >> 4;
      float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
      float acc[4][4];
  #pragma unroll
      for (int nt = 0; nt < 4; ++nt)
  #pragma unroll
        for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
  #pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb) {
        float sc[2][4];
  #pragma unroll
        for (int nt = 0; nt < 2; ++nt)
  #pragma unroll
          for (int i = 0; i < 4; ++i) sc[nt][i] = 0.f;
        const int krow = min(e0 + kb * 16 + (lane >> 4) * 8 + (lane & 7), last);
  #pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4(sK + swz(krow, c8h + ks * 2 + ((lane >> 3) & 1)), b0, b1, b2, b3);
          mma_bf16(sc[0], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
          mma_bf16(sc[1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
        }
        float bm0 = -INFINITY, bm1 = -INFINITY;
  #pragma unroll
        for (int nt = 0; nt < 2; ++nt)
  #pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int j = kb * 16 + nt * 8 + 2 * t + i;
            const bool valid = j < n;
            // a dead key's bias (kMaskedScore) swallows its score: weight exactly 0 unless every key is
            // dead, then uniform; rows past the environment's last are no keys at all
            const float bj = key_bias[e0 + j];
            const float a = valid ? fmaf(sc[nt][i], c2, bj) : -INFINITY;
            const float b = valid ? fmaf(sc[nt][2 + i], c2, bj) : -INFINITY;
            sc[nt][i] = a;
            sc[nt][2 + i] = b;
            bm0 = fmaxf(bm0, a);
            bm1 = fmaxf(bm1, b);
          }
        bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 1));
        bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, 2));
        bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 1));
        bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, 2));
        const float n0 = fmaxf(m0, bm0), n1 = fmaxf(m1, bm1);   // finite: every block holds a valid key
        const float c0 = ex2_fast(m0 - n0), c1 = ex2_fast(m1 - n1); // 2^(-inf) = 0 on the first block
        m0 = n0;
        m1 = n1;
        l0 *= c0;
        l1 *= c1;
  #pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          acc[nt][0] *= c0; acc[nt][1] *= c0;
          acc[nt][2] *= c1; acc[nt][3] *= c1;
        }
  #pragma unroll
        for (int nt = 0; nt < 2; ++nt)
  #pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float a = ex2_fast(sc[nt][i] - m0), b = ex2_fast(sc[nt][2 + i] - m1);
            sc[nt][i] = a;
            sc[nt][2 + i] = b;
            l0 += a;
            l1 += b;
          }
        const uint32_t a0 = pack_bf16(sc[0][0], sc[0][1]), a1 = pack_bf16(sc[0][2], sc[0][3]);
        const uint32_t a2 = pack_bf16(sc[1][0], sc[1][1]), a3 = pack_bf16(sc[1][2], sc[1][3]);
        const int vrow = min(e0 + kb * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), last);
  #pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t b0, b1, b2, b3;
          ldsm_x4_t(sV + swz(vrow, c8h + np * 2 + (lane >> 4)), b0, b1, b2, b3);
          mma_bf16(acc[np * 2], a0, a1, a2, a3, b0, b1);
          mma_bf16(acc[np * 2 + 1], a0, a1, a2, a3, b2, b3);
        }
      }
      l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
      l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
      l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
      l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
      const float i0 = reciprocal(l0), i1 = reciprocal(l1);
      const int q0 = r0 + g, q1 = r0 + g + 8;
      uint8_t* po = e.smem + OFF_P + atom;
  #pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        if (q0 <= last) *reinterpret_cast<uint32_t*>(po + swz(q0, c8h + nt) + t * 4) = pack_bf16(acc[nt][0] * i0, acc[nt][1] * i0);
        if (q1 <= last) *reinterpret_cast<uint32_t*>(po + swz(q1, c8h + nt) + t * 4) = pack_bf16(acc[nt][2] * i1, acc[nt][3] * i1);
      }
      r0 += n;
      e0 += n;
    } while (n < 16 && r0 <= end);
  }
}

// q | k | v of all heads in the three accumulators.
constexpr uint32_t QKV_FLIPS = 7, OUT_FLIPS = 1, LINEAR_OUT_FLIPS = 4;

// The sublayers from "normed operand posted" to "last operand of the round that ends in the residual posted"; the norms, the
// wait for that round and the GatedMLP are the same code for all of them (the kernel's loop).
__device__ __forceinline__ void run_spatial(Epi& e, int n_items, bool row_valid) {
  wait_round(e, QKV_FLIPS);
  {
    T_BEGIN();
    // this thread stages head `part` of its row: q into the P area, k and v into the KV area (whose ring slot
    // served v), all in the swizzled atom layout.  Rows outside every environment are zero rows from the input on.
    const int h = e.part;
    const uint32_t atom = (uint32_t)(h >> 1) * CHUNK_BYTES;
    const int c8h = (h & 1) * 4;
    const uint32_t dst[3] = {OFF_P + atom, OFF_KV + atom, OFF_KV + 2 * CHUNK_BYTES + atom};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      uint32_t v[32];
      tmem_ld32(e.lane_addr + COL_ACC0 + p * D + h * DH, v);
#pragma unroll
      for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(e.smem + dst[p] + swz(e.row, c8h + q)) = row_valid ? pack8(&v[q * 8]) : make_uint4(0u, 0u, 0u, 0u);
    }
    T_END(TE_STAGE);
  }
  tc_fence_before();
  asm volatile("bar.sync %0, 128;" ::"r"(7 + e.part) : "memory");   // the four warps of this head
  {
    T_BEGIN();
    attention(e, n_items);
    T_END(TE_ATTN);
  }
  // keys and values are dead: the area may take weight chunks again
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(e.bars + 8 * B_KVREL);
  post(e, B_OP0);   // attention output in P
}

// A spatial sublayer around a separate attention kernel (environments larger than a tile, or a
// sublayer that reads bullets).  First part: norm1 and q|k|v of every head, written as bf16 to
// global scratch, (rows, 384) = q | k | v with the heads side by side inside each third.
__device__ __forceinline__ void run_spatial_pre(Epi& e, const SubLayer& s, size_t grow, bool row_valid) {
  wait_round(e, QKV_FLIPS);
  const int h = e.part;
  __nv_bfloat16* dst = s.qkv_out + grow * (3 * D) + h * DH;
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    uint32_t v[32];
    tmem_ld32(e.lane_addr + COL_ACC0 + p * D + h * DH, v);
    if (row_valid) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = __uint_as_float(pack_bf16(__uint_as_float(v[q * 16 + 2 * j]), __uint_as_float(v[q * 16 + 2 * j + 1])));
        store8(reinterpret_cast<float*>(dst + p * D + q * 16), w, e.wide);
      }
    }
  }
  tc_fence_before();
}
// Second part: the attention output (bf16, (rows, 128)) becomes the A operand of out_proj, which
// accumulates into the residual; then norm2 and the GatedMLP.
__device__ __forceinline__ void run_spatial_post(Epi& e, const SubLayer& s, size_t grow, bool row_valid) {
  const float* src = reinterpret_cast<const float*>(s.o_in + grow * D + e.part * 32);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (row_valid) load8(o, src + 8 * q, e.wide);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int col = e.part * 32 + q * 16 + j * 8;
      *reinterpret_cast<float4*>(e.smem + OFF_A + (col >> 6) * CHUNK_BYTES + swz(e.row, (col & 63) >> 3)) = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
    }
  }
  post(e, B_OP0);
}

// u = bias + w0 tap0 + w1 tap1 + w2 tap2 + w3 b1 of four columns, summed in the reference's order; lag: taps that belong to the
// episode.  Returned as packed bf16.
struct ConvWeights { float w[4][4], b[4]; };
__device__ __forceinline__ ConvWeights conv_weights(const SubLayer& s, int col) {
  ConvWeights c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 w4 = __ldg(reinterpret_cast<const float4*>(s.conv_w + (col + i) * 4));
    c.w[i][0] = w4.x; c.w[i][1] = w4.y; c.w[i][2] = w4.z; c.w[i][3] = w4.w;
    c.b[i] = __ldg(s.conv_b + col + i);
  }
  return c;
}
__device__ __forceinline__ uint2 conv4(const ConvWeights& c, const float4& t0, const float4& t1, const float4& t2, const float4& b1, int lag) {
  const float a0[4] = {t0.x, t0.y, t0.z, t0.w}, a1[4] = {t1.x, t1.y, t1.z, t1.w}, a2[4] = {t2.x, t2.y, t2.z, t2.w}, a3[4] = {b1.x, b1.y, b1.z, b1.w};
  float u[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float p0 = lag >= 3 ? __fmul_rn(a0[i], c.w[i][0]) : 0.f;
    const float p1 = lag >= 2 ? __fmul_rn(a1[i], c.w[i][1]) : 0.f;
    const float p2 = lag >= 1 ? __fmul_rn(a2[i], c.w[i][2]) : 0.f;
    const float p3 = __fmul_rn(a3[i], c.w[i][3]);
    u[i] = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(p0, p1), p2), p3), c.b[i]);
  }
  return make_uint2(pack_bf16(u[0], u[1]), pack_bf16(u[2], u[3]));
}
__device__ __forceinline__ float4 unpack4(const uint2& v) { return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y)); }

// One temporal sublayer on the tile: at one timestep, or (STEPS) on chunks of `chunk` consecutive timesteps of its
// tokens.  In the gate epilogue thread (row, part) works on hidden columns [64 rnd + 16 part, +16), and parks b2 for exactly
// those.
//
// Chunks: a time walk of whole batches moves a state of 2 KB a row in and out of L2 at every step (512 KB a tile, all SMs at
// once) and has as few tiles as the batch has rows.  With 128 / C tokens x C steps the state is read and written once a chunk,
// taps come from the rows above, and the recurrence is a scan over the lanes of a warp (C rows of a
// token are neighbouring lanes): 32 steps of 4096 x 8 tokens 6075 -> 5723, 5 of 67 x 11 306 -> 197 us.
template <bool STEPS>
__device__ __forceinline__ void run_temporal(Epi& e, const SubLayer& s, const Place& rs, bool has_fields, const float* hid_in, int chunk) {
  const bool is_ship = rs.hrow >= 0;
  const float* hin = is_ship ? hid_in + (size_t)rs.hrow * 4 * D : nullptr;
  float* hout = is_ship ? s.hid_out + (size_t)rs.hrow * 4 * D : nullptr;
  // Causal conv, one warp per ship row and four columns per lane, so that the stored taps are
  // read and written as whole 512-byte rows; new taps = (tap1, tap2, b1); bf16(u) replaces b1 in A.
  T_MARK(tt);
  {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = lane * 4;
    const auto in_A = [&](int r) { return reinterpret_cast<uint2*>(e.smem + OFF_A + (lane >> 4) * CHUNK_BYTES + swz(r, (lane & 15) >> 1) + (lane & 1) * 8); };
    // One timestep: a warp takes rows warp, warp + 16, ...: four rows' taps are on their way at any time, the first four
    // before the products are waited for, and each row's registers ask for the row four further on as soon as it is done.
    // Rows are distinct, so no load needs to wait for another row's store; volatile accesses keep the compiler to that
    // order (the state may be updated in place).
    // Chunks: a warp takes rows 8 warp .. + 8, the stored taps of the tokens that begin there (two of them at most).
    constexpr int IN_FLIGHT = STEPS ? 2 : 4;
    float4 t0[IN_FLIGHT], t1[IN_FLIGHT], t2[IN_FLIGHT];
    int hr[IN_FLIGHT], fl[IN_FLIGHT];
    const auto request = [&](int k, int r) {
      const int2 at = *reinterpret_cast<const int2*>(e.tab + 16 * r);
      hr[k] = at.x;
      fl[k] = at.y;
      t0[k] = t1[k] = t2[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (hr[k] >= 0 && !(fl[k] & P_ZERO_IN)) {
        const float* hi = hid_in + (size_t)hr[k] * 4 * D + col;
        load4(t0[k], hi + D);
        load4(t1[k], hi + 2 * D);
        load4(t2[k], hi + 3 * D);
      }
    };
    ConvWeights cw;
    if constexpr (STEPS) {
      cw = conv_weights(s, col);
      if ((8 * warp & (chunk - 1)) == 0) request(0, 8 * warp);
      if (chunk == 4) request(1, 8 * warp + 4);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) request(k, warp + EPI_WARPS * k);
    }
    T_SINCE(TE_TAPS, tt);
    wait_round(e, 3);   // acc0 = linear1 n, acc1 = linear2 n / 2; slots 0 and 1
    T_RESET(tt);
    // b1 = bf16(linear1 n) into the A operand
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      uint32_t v[16];
      tmem_ld16_nowait(e.lane_addr + COL_ACC0 + e.part * 32 + p * 16, v);
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c8 = e.part * 32 + p * 16 + q * 8;
        *reinterpret_cast<uint4*>(e.smem + OFF_A + (c8 >> 6) * CHUNK_BYTES + swz(e.row, (c8 & 63) >> 3)) = pack8(&v[q * 8]);
      }
    }
    if constexpr (!STEPS) cw = conv_weights(s, col);
    tc_fence_before();
    T_SINCE(TE_B1, tt);
    epi_sync();
    T_SINCE(TE_SYNC, tt);
    if constexpr (STEPS) {
      uint2 bw[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) bw[i] = *in_A(8 * warp + i);
      if (chunk > 8) {
        if (8 * warp & (chunk - 1)) {   // the taps are the rows above, which their own warp is about to replace by u
          t0[0] = unpack4(*in_A(8 * warp - 3));
          t1[0] = unpack4(*in_A(8 * warp - 2));
          t2[0] = unpack4(*in_A(8 * warp - 1));
        }
        asm volatile("bar.sync %0, 128;" ::"r"(11 + (warp >> 2)) : "memory");   // the four warps of 32 rows
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 8 * warp + i;
        if (i == 4 && chunk == 4) {
          t0[0] = t0[1];
          t1[0] = t1[1];
          t2[0] = t2[1];
        }
        const int2 at = *reinterpret_cast<const int2*>(e.tab + 16 * r);
        if (at.x >= 0) {
          const float4 b1 = unpack4(bw[i]);
          *in_A(r) = conv4(cw, t0[0], t1[0], t2[0], b1, at.y >> 8);
          t0[0] = t1[0];
          t1[0] = t2[0];
          t2[0] = b1;
          if (at.y & P_LAST) {
            float* ho = s.hid_out + (size_t)at.x * 4 * D + col;
            store4(ho + D, t0[0]);
            store4(ho + 2 * D, t1[0]);
            store4(ho + 3 * D, t2[0]);
          }
        }
      }
    } else {
#pragma unroll 1
      for (int r0 = warp; r0 < TILE; r0 += 4 * EPI_WARPS) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = r0 + EPI_WARPS * k;
          if (hr[k] >= 0) {
            const float4 b1 = unpack4(*in_A(r));
            float* ho = s.hid_out + (size_t)hr[k] * 4 * D + col;
            store4(ho + D, t1[k]);
            store4(ho + 2 * D, t2[k]);
            store4(ho + 3 * D, b1);
            *in_A(r) = conv4(cw, t0[k], t1[k], t2[k], b1, fl[k] >> 8);
          }
          if (r + 4 * EPI_WARPS < TILE) request(k, r + 4 * EPI_WARPS);
        }
      }
    }
  }
  T_SINCE(TE_CONV, tt);
  post(e, B_OP0);   // A = u (ship rows) / b1 (field rows)
  T_RESET(tt);
  // While the gates are multiplied: the previous state of this thread's columns is asked for ...
  float hprev[2][2][8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) hprev[i >> 1][i & 1][j] = 0.f;
    if (is_ship && !(rs.flags & P_ZERO_IN) && (!STEPS || (e.row & (chunk - 1)) == 0)) load8(hprev[i >> 1][i & 1], hin + (i >> 1) * 64 + e.part * 16 + (i & 1) * 8, e.wide);
  }
  // ... and b2 = bf16(gelu(linear2 n)) parked as packed bf16 pairs
  uint32_t b2p[2][8];
#pragma unroll
  for (int rnd = 0; rnd < 2; ++rnd) {
    uint32_t v[16];
    tmem_ld16_nowait(e.lane_addr + COL_ACC1 + rnd * 64 + e.part * 16, v);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 8; ++j) b2p[rnd][j] = pack_bf16(gelu_half(acc_pair(&v[2 * j])));
  }
  if (has_fields) {   // acc1 may take field_sub
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(e.bars + 8 * B_PARK);
  }
  T_SINCE(TE_PARK, tt);
  wait_early(e);   // acc0 / acc2 = halves of [W_a u | W_x u] of hidden columns [0,64) / [64,128)
  // gates and state update
  const F2 keep = f2(rs.flags & P_BOUNDARY ? 0.f : 1.f), one = f2(1.f);
#pragma unroll
  for (int rnd = 0; rnd < 2; ++rnd) {
    if (rnd == 1) wait_round(e, has_fields ? 7 : 5);   // slots 2, 0 (and 1 for field_sub)
    T_RESET(tt);
    uint32_t rv[16], iv[16];
    const uint32_t acc = e.lane_addr + (rnd ? COL_ACC2 : COL_ACC0) + e.part * 16;
    tmem_ld16_nowait(acc, rv);        // executed by every lane of the warp
    tmem_ld16_nowait(acc + 64, iv);
    tmem_wait_ld();
    // per column: h = a h_prev + b; with chunks h_prev stands in a token's first row (0 in the others) and the rest follows
    // from the scan over its rows below, which lanes of field and empty rows run along with.
    F2 av[STEPS ? 8 : 1], bv[STEPS ? 8 : 1];
    // result of a pair of columns: new state, and the branch operand of linear_out
    const auto finish = [&](F2 h, int k, float* hn, uint32_t& ob) {
      const float2 n = halves(h);
      hn[0] = n.x;
      hn[1] = n.y;
      ob = pack_bf16(mul(h, unpack_bf16(b2p[rnd][k])));
    };
    const auto put = [&](int q, const float (&hn)[8], const uint32_t (&ob)[4]) {
      if (!STEPS || (rs.flags & P_LAST)) store8(hout + rnd * 64 + e.part * 16 + q * 8, hn, e.wide);
      // K atom 0 of the operand lives in P0, K atom 1 in place in A
      uint8_t* dst = rnd == 0 ? e.smem + OFF_P + swz(e.row, e.part * 2 + q) : e.smem + OFF_A + CHUNK_BYTES + swz(e.row, e.part * 2 + q);
      *reinterpret_cast<uint4*>(dst) = make_uint4(ob[0], ob[1], ob[2], ob[3]);
    };
    if (STEPS || is_ship) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int col = rnd * 64 + e.part * 16 + q * 8;
        // u (bf16) back from the A operand (K atom rnd)
        const uint4 ub = *reinterpret_cast<const uint4*>(e.smem + OFF_A + rnd * CHUNK_BYTES + swz(e.row, e.part * 2 + q));
        const uint32_t uw[4] = {ub.x, ub.y, ub.z, ub.w};
        float hn[8];
        uint32_t ob[4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const float* table = s.decay_log2 + col + hf * 4;
          const float4 dl = __ldg(reinterpret_cast<const float4*>(table)), ab = __ldg(reinterpret_cast<const float4*>(table + D)),
                       xb = __ldg(reinterpret_cast<const float4*>(table + 2 * D));
          const F2 dlv[2] = {f2(dl.x, dl.y), f2(dl.z, dl.w)}, abv[2] = {f2(ab.x, ab.y), f2(ab.z, ab.w)}, xbv[2] = {f2(xb.x, xb.y), f2(xb.z, xb.w)};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int k = q * 8 + hf * 4 + 2 * i, w = hf * 2 + i;
            const F2 rg = sigmoid_twice_bf16(add(acc_pair(&rv[k]), abv[i])), ig = sigmoid_twice_bf16(add(acc_pair(&iv[k]), xbv[i]));
            // sigmoid(Lambda)^(8 r) = 2^(r * 8 log2 sigmoid(Lambda)); the table is part of the weight image
            const float2 ad = halves(mul(rg, dlv[i]));
            const F2 a = f2(ex2_fast(ad.x), ex2_fast(ad.y));
            const float2 rest = halves(mul(fma(a, f2(-1.f), one), add(one, a)));
            const F2 gate = f2(sqrt_fast(fmaxf(rest.x, kGateFloor)), sqrt_fast(fmaxf(rest.y, kGateFloor)));
            const F2 ak = mul(a, keep);
            const F2 b = fma(ak, f2(hprev[rnd][q][k & 7], hprev[rnd][q][(k & 7) + 1]), mul(gate, mul(ig, unpack_bf16(uw[w]))));
            if constexpr (STEPS) {
              av[k >> 1] = ak;
              bv[k >> 1] = b;
            } else {
              finish(b, k >> 1, hn + 2 * w, ob[w]);
            }
          }
        }
        if constexpr (!STEPS) put(q, hn, ob);
      }
    }
    if constexpr (STEPS) {
      const int step = e.row & (chunk - 1);
      const auto level = [&](int d, bool last) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 b = halves(bv[k]);
          const F2 b_up = f2(__shfl_up_sync(0xffffffffu, b.x, d), __shfl_up_sync(0xffffffffu, b.y, d));
          F2 a_up = one;
          if (!last) {
            const float2 a = halves(av[k]);
            a_up = f2(__shfl_up_sync(0xffffffffu, a.x, d), __shfl_up_sync(0xffffffffu, a.y, d));
          }
          if (step >= d) {
            bv[k] = fma(av[k], b_up, bv[k]);
            av[k] = mul(av[k], a_up);
          }
        }
      };
#pragma unroll 1
      for (int d = 1; 2 * d < chunk; d <<= 1) level(d, false);
      level(chunk >> 1, true);   // nobody needs this level's products of a
      if (is_ship) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float hn[8];
          uint32_t ob[4];
#pragma unroll
          for (int w = 0; w < 4; ++w) finish(bv[q * 4 + w], q * 4 + w, hn + 2 * w, ob[w]);
          put(q, hn, ob);
        }
      }
    }
    T_SINCE(TE_GATES, tt);
  }
  if (has_fields) {
    // field rows: branch = bf16(bf16(field_sub b1) * b2); rows outside every environment are zeros throughout
    wait_field(e);
    T_RESET(tt);
#pragma unroll
    for (int rnd = 0; rnd < 2; ++rnd) {
      uint32_t v[16];
      tmem_ld16_nowait(e.lane_addr + COL_ACC1 + rnd * 64 + e.part * 16, v);        // executed by every lane of the warp
      tmem_wait_ld();
      if (!is_ship) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 f = pack8(&v[q * 8]);
          const uint32_t* b2 = &b2p[rnd][q * 4];
          uint8_t* dst = rnd == 0 ? e.smem + OFF_P + swz(e.row, e.part * 2 + q)
                                  : e.smem + OFF_A + CHUNK_BYTES + swz(e.row, e.part * 2 + q);
          *reinterpret_cast<uint4*>(dst) = make_uint4(mul_bf16x2(f.x, b2[0]), mul_bf16x2(f.y, b2[1]), mul_bf16x2(f.z, b2[2]), mul_bf16x2(f.w, b2[3]));
        }
      }
    }
  } else if (!is_ship) {
    // rows outside every environment: zero operand rows
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      *reinterpret_cast<uint4*>(e.smem + OFF_P + swz(e.row, e.part * 2 + q)) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(e.smem + OFF_A + CHUNK_BYTES + swz(e.row, e.part * 2 + q)) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  T_SINCE(TE_FIELDS, tt);
  post(e, B_OP0);   // branch operand
}

// ------------------------------------------------------------------ issuing side (two warps)
//
// A whole warp runs this code with the same values in every lane, and one elected lane issues: the
// operands of the MMAs then stay in uniform registers and an MMA costs three instructions.
//
// What bounds the GatedMLP is issue, not the tensor pipe: with one warp issuing everything, a chunk's two waits for
// weights, one for its operand and twelve MMAs were a serial chain of 1 400 cycles where the pipe needs 770 (64 cycles per
// 128 x 128 x 16).  So the down projections have a warp of their own, on another scheduler.

struct Issuer {
#ifdef BNB_TRACE
  Trace tr;
#endif
  uint32_t sbase, bars, tmem;
  uint32_t elected;    // 1 in the lane that issues
  uint32_t full_par;   // per-slot phase bits of the FULL barriers
  uint32_t op_par;     // phase bits of OP0, FFN and REL
  volatile int* aborted;
};

__device__ __forceinline__ void wait_operand(Issuer& m, int bar) {
  T_BEGIN();
  wait_bar(m.bars + 8 * bar, (m.op_par >> bar) & 1u, m.aborted, ST_TIMEOUT_OPERAND);
  m.op_par ^= 1u << bar;
  tc_fence_after();
  T_END(TM_OP_WAIT);
  TRACE(m.tr, 400 + bar);
}
__device__ __forceinline__ void commit_one(const Issuer& m, uint32_t bar) { tc_commit_if(m.elected, m.bars + 8 * bar); }
// Waits for the weights of a slot.
__device__ __forceinline__ void wait_weights(Issuer& m, uint32_t slot) {
  T_MARK(tw);
  wait_bar(m.bars + 8 * (B_FULL0 + slot), (m.full_par >> slot) & 1u, m.aborted, ST_TIMEOUT_FULL);
  m.full_par ^= 1u << slot;
  T_SINCE(TM_FULL_WAIT, tw);
  TRACE(m.tr, 410);
}
// A pair operation: D[128 x 128] (+)= A[128 x 128] * W[128 x 128]^T, K atom 0 of the operand at a_off0 and K
// atom 1 at a_off1; commits on the slot's DONE barrier.  (A step of 16 K columns = 32 bytes = 2 in
// descriptor units; a K atom = 16 KB = 1024 units.)
__device__ __forceinline__ void multiply_pair(Issuer& m, uint32_t slot, uint32_t a_off0, uint32_t a_off1, uint32_t d_col, uint32_t accumulate) {
  T_MARK(tw);
  constexpr uint32_t idesc = instr_desc(128);
  const uint32_t b_lo = uniform(desc_lo(m.sbase + pair_offset(slot)));
  const uint32_t a0 = desc_lo(m.sbase + a_off0), a1 = desc_lo(m.sbase + a_off1);
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) mma_one<false>(m.elected, m.tmem + d_col, a0 + 2 * k, b_lo + 2 * k, idesc, (accumulate | k) ? 1u : 0u);
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) mma_one<false>(m.elected, m.tmem + d_col, a1 + 2 * k, b_lo + 1024 + 2 * k, idesc, 1u);
  commit_one(m, B_DONE0 + slot);
  T_SINCE(TM_ISSUE, tw);
  TRACE(m.tr, 420);
}
__device__ __forceinline__ void issue_pair(Issuer& m, uint32_t slot, uint32_t a_off0, uint32_t a_off1, uint32_t d_col, uint32_t accumulate) {
  wait_weights(m, slot);
  multiply_pair(m, slot, a_off0, a_off1, d_col, accumulate);
}
__device__ __forceinline__ void issue_from_A(Issuer& m, uint32_t slot, uint32_t d_col) {
  issue_pair(m, slot, OFF_A, OFF_A + CHUNK_BYTES, d_col, 0);
}
__device__ __forceinline__ void commit_round(const Issuer& m) { commit_one(m, B_ACC); }

// gate|up of the eight chunks; slot: pair slot of chunk 0.
__device__ __forceinline__ void issue_gate_up(Issuer& m, uint32_t slot) {
  wait_operand(m, B_OP0);
#pragma unroll 1
  for (uint32_t c = 0; c < 8; ++c) {
    wait_weights(m, slot);
    if (c >= 2) wait_operand(m, B_REL0 + (c & 1));   // gate|up of chunk c - 2 have been read
    multiply_pair(m, slot, OFF_A, OFF_A + CHUNK_BYTES, COL_ACC0 + 128 * (c & 1), 0);
    slot = slot == 2 ? 0 : slot + 1;
  }
  m.op_par ^= 3u << B_REL0;   // those of chunks 6 and 7 are not waited for here: every operand posted from now on comes after them
}
// Rows that the tile owners need next are asked into L2 by the warp of the down projections, whose own work is a quarter of its
// time.  As prefetches of the epilogue threads the state alone held their load pipe for 1 400 cycles of every tile and
// temporal sublayer; as bulk prefetches they stand in the way of the weight copies (7 000 cycles).
__device__ __forceinline__ void prefetch_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// The recurrent state of 16 tile rows (2 KB each, two lanes a row).
__device__ __forceinline__ void prefetch_state(const float* hid, const uint8_t* tab, int row0) {
  const int lane = threadIdx.x & 31, hrow = *reinterpret_cast<const int*>(tab + 16 * (row0 + (lane >> 1)));
  if (hrow < 0) return;
  const float* p = hid + (size_t)hrow * 4 * D + (lane & 1) * 2 * D;
#pragma unroll
  for (int i = 0; i < 8; ++i) prefetch_line(p + 32 * i);
}
// The row table of a pass: tile `tile` at timestep t.
template <int MODE>
__device__ __forceinline__ void fill_table(const TrunkArgs& args, int tile, int t, uint8_t* tab) {
  const EnvMap& map = args.map;
  const int lane = threadIdx.x & 31;
  const int grp = tile / args.env_tiles, eb = tile - grp * args.env_tiles;
  uint32_t* blocks = reinterpret_cast<uint32_t*>(tab + TAB_BLOCKS);
  float* bias = reinterpret_cast<float*>(tab + TAB_BIAS);
  const auto invalid = [&](int row) {
    reinterpret_cast<int4*>(tab)[row] = make_int4(-1, 0, -1, 0);
    bias[row] = kMaskedScore;
  };
  // token `tok` of environment env, which has `ships` ships, at timestep t
  const auto put = [&](int row, int env, int tok, int ships, int step_row, int hrow, int t, uint32_t flags, bool live) {
    const int trow = (grp + t) * map.total_tokens + step_row;
    if (MODE != STEPS) bias[row] = live ? 0.f : kMaskedScore;
    if (tok < ships) {
      // steps since the last episode boundary, as far as the conv looks back; before the call there was none
      uint32_t lags = BNB_CONV_KERNEL - 1;
      if (args.done)
#pragma unroll
        for (int k = BNB_CONV_KERNEL - 1; k >= 1; --k)
          if (t >= k && args.done[(size_t)(t - k) * map.n_envs + env]) lags = k - 1;
      if (t >= 1 && lags == 0) flags |= P_BOUNDARY;
      flags |= lags << 8;
      if (t == 0 && args.reset_env && args.reset_env[env]) flags |= P_ZERO_IN;
    } else {
      hrow = -1;
    }
    reinterpret_cast<int4*>(tab)[row] = make_int4(hrow, (int)flags, trow, 0);
  };
  int n_blocks = 0;
  if constexpr (MODE == STEPS) {
#pragma unroll 1
    for (int row = lane; row < TILE; row += 32) {
      const int step = row & (args.chunk - 1), r = (eb * TILE + row) / args.chunk, time = t * args.chunk + step;
      if (r < map.total_tokens && time < args.steps) {
        const int env = map.env_of_token(r), tok = r - map.env_tok_begin(env);
        put(row, env, tok, map.env_ship_count(env), r, map.env_ship_begin(env) + tok, time,
            P_VALID | (step == args.chunk - 1 || time == args.steps - 1 ? P_LAST : 0u), true);
      } else {
        invalid(row);
      }
    }
  } else if (MODE == ANY && args.flat_rows) {
    // plain 128-row slices of the token rows (programs without attention inside: the
    // environments are larger than a tile); the environment of a row is looked up
#pragma unroll 1
    for (int row = lane; row < TILE; row += 32) {
      const int r = eb * TILE + row;
      if (r < map.total_tokens) {
        const int env = map.env_of_token(r), tok = r - map.env_tok_begin(env);
        put(row, env, tok, map.env_ship_count(env), r, map.env_ship_begin(env) + tok, t, P_VALID, true);   // no attention on such tiles
      } else {
        invalid(row);
      }
    }
  } else if (args.tile_env_begin) {
    // ragged: the tile holds the environments tile_env_ids[k_lo .. k_hi), rows in that order
    const int end = args.tile_env_begin[eb + 1];
    int first = 0;
    for (int k0 = args.tile_env_begin[eb]; k0 < end; k0 += 32) {
      int my_env = 0, my_tok = 0, my_n = 0, my_ship = 0, my_ships = 0;
      if (k0 + lane < end) {
        my_env = args.tile_env_ids[k0 + lane];
        my_tok = map.tok_off[my_env];
        my_n = map.tok_off[my_env + 1] - my_tok;
        my_ship = map.ship_off[my_env];
        my_ships = map.ship_off[my_env + 1] - my_ship;
      }
      for (int j = 0; j < min(32, end - k0); ++j) {
        const int env = __shfl_sync(0xffffffffu, my_env, j), tok0 = __shfl_sync(0xffffffffu, my_tok, j), n = __shfl_sync(0xffffffffu, my_n, j),
                  ship0 = __shfl_sync(0xffffffffu, my_ship, j), ships = __shfl_sync(0xffffffffu, my_ships, j);
        for (int i = lane; i < n; i += 32) {
          put(first + i, env, i, ships, tok0 + i, ship0 + i, t, P_VALID, !args.alive || args.alive[(size_t)(grp + t) * map.total_tokens + tok0 + i]);
          if ((i & 15) == 0) blocks[n_blocks + (i >> 4)] = (uint32_t)(first + i) | (uint32_t)first << 8 | (uint32_t)(n - 1) << 16 | (uint32_t)n << 24;
        }
        first += n;
        n_blocks += (n + 15) >> 4;
      }
    }
    for (int row = first + lane; row < TILE; row += 32) invalid(row);
  } else {
    const int NM = map.tokens_per_env, per_env = (NM + 15) >> 4;
    const int share = NM <= 8 ? 16 / NM : 1;   // environments whose queries share a block (attend_block)
    const int env0 = eb * args.envs_per_tile, envs = min(args.envs_per_tile, map.n_envs - env0);
    int el[4], tok[4];
    uint8_t live[4];   // the masks of this lane's rows, all on their way at once
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = lane + 32 * k;
      el[k] = row / NM;
      tok[k] = row - el[k] * NM;
      live[k] = 1;
      if (el[k] < envs && args.alive) live[k] = args.alive[(size_t)(grp + t) * map.total_tokens + env0 * NM + row];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = lane + 32 * k;
      if (el[k] < envs) {
        put(row, env0 + el[k], tok[k], map.ships_per_env, env0 * NM + row, (env0 + el[k]) * map.ships_per_env + tok[k], t, P_VALID, live[k] != 0);
        if ((tok[k] & 15) == 0 && el[k] % share == 0)
          blocks[el[k] / share * per_env + (tok[k] >> 4)] = (uint32_t)row | (uint32_t)(el[k] * NM) << 8 | (uint32_t)(min(share, envs - el[k]) * NM - 1) << 16 | (uint32_t)NM << 24;
      } else {
        invalid(row);
      }
    }
    n_blocks = (envs + share - 1) / share * per_env;
  }
  if (lane == 0) *reinterpret_cast<int*>(tab + TAB_COUNT) = n_blocks;
  __syncwarp();
}
// The tokens of a pass into L2, and bfloat16 ones into the P area (free from a sublayer's out_proj or linear_out on) as two
// swizzled atoms: rows as the pass's table has them.
__device__ __forceinline__ int row_of(const uint8_t* tab, int row) { return *reinterpret_cast<const int*>(tab + 16 * row + 8); }
__device__ __forceinline__ void prefetch_tokens(const TrunkArgs& args, const uint8_t* tab) {
  const int lane = threadIdx.x & 31;
  const uint8_t* x = reinterpret_cast<const uint8_t*>(args.x);
  const int lines = args.io_bf16 ? 2 : 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int at = row_of(tab, lane + 32 * k);
    if (at >= 0)
      for (int l = 0; l < lines; ++l) prefetch_line(x + ((size_t)at * lines + l) * 128);
  }
}
// (Eight rows' places are read before the first copy: one by one, each copy waited for its own, 7 000 cycles a tile.)
__device__ __forceinline__ void copy_tokens(const TrunkArgs& args, const uint8_t* tab, uint32_t p_area) {
  const int lane = threadIdx.x & 31, c8 = lane & 15;
  const uint8_t* x = reinterpret_cast<const uint8_t*>(args.x) + 16 * c8;
  p_area += (c8 >> 3) * CHUNK_BYTES;
#pragma unroll 1
  for (int row0 = lane >> 4; row0 < TILE; row0 += 16) {
    int at[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) at[k] = row_of(tab, row0 + 2 * k);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (at[k] >= 0) cp_async16(p_area + swz(row0 + 2 * k, c8 & 7), x + (size_t)at[k] * (2 * D));
  }
}
// What this lane has written and copied for the next pass: two arrivals on XFULL.
__device__ __forceinline__ void hand_over(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
  mbar_arrive(bar);
}

// The down projections of the eight chunks: A operand in tensor memory, K step k in the 8 columns at 8 k of the buffer.
// next_hid: the state that the following sublayer reads (null: none, or it is at hand), asked for on the way.
__device__ __forceinline__ void issue_downs(Issuer& m, const float* next_hid, const uint8_t* tab) {
  constexpr uint32_t idesc = instr_desc(128);
  uint32_t a = 0;
#pragma unroll 1
  for (uint32_t c = 0; c < 8; ++c) {
    wait_weights(m, 3 + a);
    wait_operand(m, B_FFN0 + (c & 3));   // product of chunk c written
    T_MARK(tw);
    const uint32_t b_lo = uniform(desc_lo(m.sbase + single_offset(a)));
    const uint32_t a_col = m.tmem + COL_ACC2 + 32 * (c & 3);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) mma_one<true>(m.elected, m.tmem + COL_RESID, a_col + 8 * k, b_lo + 2 * k, idesc, 1u);
    commit_one(m, B_DONE0 + 3 + a);
    commit_one(m, B_PFREE0 + (c & 3));
    T_SINCE(TM_ISSUE, tw);
    TRACE(m.tr, 430);
    if (next_hid) prefetch_state(next_hid, tab, 16 * (int)c);
    __syncwarp();
    a = a == 2 ? 0 : a + 1;
  }
  commit_round(m);
}
__device__ __forceinline__ void issue_qkv(Issuer& m) {
  wait_operand(m, B_OP0);
#pragma unroll 1
  for (uint32_t i = 0; i < 3; ++i) issue_from_A(m, i, COL_ACC0 + 128 * i);
  commit_round(m);
}
__device__ __forceinline__ void issue_out_proj(Issuer& m, uint32_t a_off) {
  wait_operand(m, B_OP0);   // attention output: K atom 0 = heads 0, 1; K atom 1 = heads 2, 3
  issue_pair(m, 0, a_off, a_off + CHUNK_BYTES, COL_RESID, 1);
  commit_round(m);
}
__device__ __forceinline__ void issue_temporal(Issuer& m, bool has_fields) {
  wait_operand(m, B_OP0);
  issue_from_A(m, 0, COL_ACC1);   // linear2
  issue_from_A(m, 1, COL_ACC0);   // linear1
  commit_round(m);
  wait_operand(m, B_OP0);
  issue_from_A(m, 2, COL_ACC0);   // gates of hidden columns [0,64)
  commit_one(m, B_EARLY);
  issue_from_A(m, 0, COL_ACC2);   // gates of hidden columns [64,128)
  commit_round(m);
  if (has_fields) {
    wait_operand(m, B_PARK);
    issue_from_A(m, 1, COL_ACC1);   // field_sub
    commit_one(m, B_FIELD);
  }
  wait_operand(m, B_OP0);
  issue_pair(m, 2, OFF_P, OFF_A + CHUNK_BYTES, COL_RESID, 1);   // linear_out: K atom 0 from P0, K atom 1 in place in A
  commit_round(m);
}

// ------------------------------------------------------------------ the kernel

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1) k_trunk_pipelined(const __grid_constant__ TrunkArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // an offset: the compiler still knows it as shared memory
  __shared__ int s_aborted[2];
  __shared__ SubLayer s_sub[MAX_SUBLAYERS];  // kernel parameters are slow to index dynamically
  __shared__ uint4 s_sched[MAX_SCHED];
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid < args.n_sub) s_sub[tid] = args.sub[tid];
  int sched_len = 0;
  for (int si = 0; si < args.n_sub; ++si) {
    const int ops = sublayer_ops(args.sub[si].type, args.has_fields != 0), op = tid - sched_len;
    if (op >= 0 && op < ops) s_sched[tid] = sched_entry(args.sub[si], op, args.has_fields != 0);
    sched_len += ops;
  }
  // Both row tables start without rows: after a wait has run out they may be read before they are written.
#ifdef BNB_TIMING
  if (tid < 32) time_counters()[tid] = 0;
#endif
  for (int i = tid; i < 2 * TAB_BYTES / 16; i += THREADS)
    reinterpret_cast<int4*>(smem + OFF_TAB)[i] = i % (TAB_BYTES / 16) < TILE ? make_int4(-1, 0, -1, 0) : make_int4(0, 0, 0, 0);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_BAR + 8 * B_COUNT);
  if (tid == 0) {
    s_aborted[0] = 0;
    s_aborted[1] = args.poll_limit > 0 ? args.poll_limit : DEFAULT_POLL_LIMIT;
    mbar_init(smem_u32(&bars[B_OP0]), EPI_WARPS);
    for (int i = B_FFN0; i <= B_REL1; ++i) mbar_init(smem_u32(&bars[i]), EPI_WARPS / 2);
    mbar_init(smem_u32(&bars[B_KVREL]), EPI_WARPS);
    mbar_init(smem_u32(&bars[B_PARK]), EPI_WARPS);
    mbar_init(smem_u32(&bars[B_XFREE]), EPI_WARPS);
    mbar_init(smem_u32(&bars[B_XFULL]), 64);   // every lane of the copying warp: its copies, its writes
    mbar_init(smem_u32(&bars[B_DRAIN]), 2);   // both issuing warps
    for (int i = B_ACC; i < B_COUNT; ++i) mbar_init(smem_u32(&bars[i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  wait_for_previous();
  if (tid == 0 && *args.status != 0) *static_cast<volatile int*>(s_aborted) = -1;
  const int my_tiles = blockIdx.x < args.n_tiles ? (args.n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const int passes = my_tiles * args.t_loop;

  if (warp == LOAD_WARP) {
    // ---------------------------------------------------------------- weight stream
    // The whole warp runs the same code and one elected lane copies, as on the issuing side.
    {
      const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(bars);
      const bool elected = elect_one() != 0;
      uint32_t free_par = (1u << N_SLOTS) - 1u;   // a fresh barrier passes a wait on parity 1: every slot starts free
      uint32_t kv_par = 0;
      const int len = sched_len;
      const int skip_op = blockIdx.x == 0 ? args.skip_op : -1;
      T_MARK(t_start);
#ifdef BNB_TRACE
      Trace ltr;
      trace_init(ltr, args.status, 2);
      if ((tid & 31) != 0) ltr.n = 1500;
#endif
      // A chunk of the GatedMLP takes two operations, so what one takes here, instruction after instruction of a lone warp, is
      // half of the least a chunk can take (770 cycles would keep the tensor pipe full).  One copy for a pair (its K halves are neighbours in the image and in the slot), the
      // next entry read ahead, addresses from the table: 8192 x 12 tokens 586 -> 566 us.
      int op = 0;
      uint4 en = s_sched[0];
      for (int pass = 0; pass < passes; ++pass)
        for (int i = 0; i < len; ++i, ++op) {
          const uint4 now = en;
          en = s_sched[i + 1 < len ? i + 1 : 0];
          const uint32_t slot = now.z & 7u;
          T_MARK(tw);
          if (now.z & 8u) {
            wait_bar(bar0 + 8 * B_KVREL, kv_par, s_aborted, ST_TIMEOUT_FREE);
            kv_par ^= 1u;
          }
          T_SINCE(TL_KV_WAIT, tw);
          wait_bar(bar0 + 8 * (B_DONE0 + slot), (free_par >> slot) & 1u, s_aborted, ST_TIMEOUT_FREE);
          free_par ^= 1u << slot;
          // Once a wait of this CTA has run out nothing is in step any more: stop fetching.  Arming a
          // FULL barrier again before its previous copy has landed would arrive on it twice in one
          // phase, which is undefined; the other roles' waits give up at once and the kernel drains.
          if (*static_cast<volatile int*>(s_aborted)) { pass = passes; break; }
          T_SINCE(TL_FREE_WAIT, tw);
          TRACE(ltr, 500 + slot);
          if (elected && op != skip_op) {   // skip_op: test hook, this operation's weights never arrive
            const uint32_t full = bar0 + 8 * (B_FULL0 + slot);
            mbar_expect_tx(full, now.w);
            bulk_g2s(sbase + (now.z & ~15u), reinterpret_cast<const void*>(((unsigned long long)now.y << 32) | now.x), now.w, full);
          }
        }
      T_SINCE(TL_TOTAL, t_start);
    }
  } else if (warp == MMA_WARP || warp == DOWN_WARP) {
    // ---------------------------------------------------------------- tensor-core issue
    {
      Issuer m;
      m.sbase = smem_u32(smem);
      m.bars = smem_u32(bars);
      m.tmem = uniform(tmem_base);
      m.elected = elect_one();
      m.full_par = 0;
      m.op_par = 0;
      m.aborted = s_aborted;
#ifdef BNB_TRACE
      trace_init(m.tr, args.status, warp == MMA_WARP ? 1 : 3);
      if ((tid & 31) != 0) m.tr.n = 1500;
#endif
      T_MARK(t_start);
      const bool down = warp == DOWN_WARP;
      if (down && passes > 0) {
        fill_table<MODE>(args, blockIdx.x, 0, smem + OFF_TAB);
        if (args.io_bf16) copy_tokens(args, smem + OFF_TAB, m.sbase + OFF_P);
        hand_over(m.bars + 8 * B_XFULL);
        __syncwarp();
      }
      int tile = blockIdx.x, t = 0;
      for (int pass = 0; pass < passes; ++pass) {
        const int this_t = t;
        if (++t == args.t_loop) {
          t = 0;
          tile += gridDim.x;
        }
        for (int si = 0; si < args.n_sub; ++si) {
          const int type = (int)uniform((uint32_t)s_sub[si].type);
          if (down) {
            if (si + 1 == args.n_sub && pass + 1 < passes) {
              wait_bar(m.bars + 8 * B_XFREE, pass & 1u, m.aborted, ST_TIMEOUT_OPERAND);
              fill_table<MODE>(args, tile, t, smem + OFF_TAB + (~pass & 1) * TAB_BYTES);
              prefetch_tokens(args, smem + OFF_TAB + (~pass & 1) * TAB_BYTES);
            }
            __syncwarp();
            const bool state_next = MODE != STEPS && this_t == 0 && type != SUB_TEMPORAL && si + 1 < args.n_sub && s_sub[si + 1].type == SUB_TEMPORAL;
            if (MODE != ANY || type != SUB_SPATIAL_PRE)
              issue_downs(m, state_next ? s_sub[si + 1].hid_in : nullptr, smem + OFF_TAB + (pass & 1) * TAB_BYTES);
            continue;
          }
          if (MODE == STEPS || type == SUB_TEMPORAL) {
            issue_temporal(m, args.has_fields != 0);
          } else {
            if (MODE != ANY || type != SUB_SPATIAL_POST) issue_qkv(m);
            if (MODE == ANY && type == SUB_SPATIAL_PRE) continue;
            issue_out_proj(m, MODE == ANY && type == SUB_SPATIAL_POST ? OFF_A : OFF_P);
          }
          issue_gate_up(m, type == SUB_TEMPORAL ? TEMPORAL_FFN_PAIR : SPATIAL_FFN_PAIR);
        }
        if (down && pass + 1 < passes) {
          if (args.io_bf16) copy_tokens(args, smem + OFF_TAB + (~pass & 1) * TAB_BYTES, m.sbase + OFF_P);
          hand_over(m.bars + 8 * B_XFULL);
          __syncwarp();
        }
      }
      // Nothing issued here may outlive the CTA: its tensor memory is freed and its barriers go
      // away at the end.  In a normal run the epilogue warps' last waits already imply this; after
      // a wait has run out nobody has waited for anything, so wait here, with the full limit.
      commit_one(m, B_DRAIN);
      for (int i = 0; i < DEFAULT_POLL_LIMIT && !mbar_try_wait(m.bars + 8 * B_DRAIN, 0); ++i) {
      }
      T_SINCE(TM_TOTAL, t_start);
    }
  } else {
    // ---------------------------------------------------------------- tile owners
    Epi e;
    e.smem = smem;
    e.sbase = smem_u32(smem);
    e.bars = smem_u32(bars);
    e.row = tid & (TILE - 1);
    e.part = tid >> 7;
    e.wide = args.wide != 0;
    e.lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    e.par = 0;
    e.aborted = s_aborted;
    e.ss_part = reinterpret_cast<float*>(smem + OFF_SS);
#ifdef BNB_TRACE
    trace_init(e.tr, args.status, 0);
    if (tid != 0) e.tr.n = 1500;
#endif
    T_MARK(t_start);
    const int row = e.row, lane = tid & 31;
    // Rows of bfloat16 tokens move through shared memory, so that a warp's access to global memory is two whole rows: 4
    // accesses of 512 bytes, where a thread per row took 2 that touch 32 lines each (a pass's last wait to its
    // first operand: 10 000 cycles, of a time walk's 45 000).  Row of this lane's i-th access, and its 16 bytes of the row:
    const auto io_row = [&](int i) { return 32 * (warp & 3) + 8 * e.part + 2 * i + (lane >> 4); };
    const uint32_t io_atom = ((lane & 15) >> 3) * CHUNK_BYTES;
    const auto own16 = [&](int area, int j) { return reinterpret_cast<uint4*>(smem + area + (e.part >> 1) * CHUNK_BYTES + swz(row, (e.part & 1) * 4 + j)); };

    int t = 0;
    for (int pass = 0; pass < passes; ++pass) {
      // ---- the pass: a tile of whole environments, ships first then fields in each
      T_MARK(t_io);
      const bool first_step = t == 0;
      if (++t == args.t_loop) t = 0;
      wait_other(e, B_XFULL, 12);
      T_RESET(t_io);
      e.tab = smem + OFF_TAB + (pass & 1) * TAB_BYTES;
      const int4 own = reinterpret_cast<const int4*>(e.tab)[row];
      const Place rs{own.x, (uint32_t)own.y, own.z, 0};
      const bool valid = rs.flags & P_VALID;
      // residual <- x (this thread: columns [32 part, 32 part + 32))
      {
        uint32_t v[32];
        if (args.io_bf16) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 w = valid ? *own16(OFF_P, j) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              v[j * 8 + 2 * k] = ws[k] << 16;              // a bfloat16 is the upper half of its float
              v[j * 8 + 2 * k + 1] = ws[k] & 0xFFFF0000u;
            }
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (valid) load8(f, args.x + (size_t)rs.trow * D + e.part * 32 + q * 8, e.wide);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[q * 8 + j] = __float_as_uint(f[j]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(e.bars + 8 * B_XFREE);
        tmem_st32(e.lane_addr + COL_RESID + e.part * 32, v);
      }
      T_SINCE(TE_IO, t_io);
      const int n_items = *reinterpret_cast<const int*>(e.tab + TAB_COUNT);
      for (int si = 0; si < args.n_sub; ++si) {
        const SubLayer& s = s_sub[si];
        const int type = s.type;
        const bool temporal = MODE == STEPS || type == SUB_TEMPORAL;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          if (MODE != ANY || half || type != SUB_SPATIAL_POST) {
            norm_to_A(e);
            post(e, B_OP0);
          }
          if (half) {
            ffn(e, temporal ? TEMPORAL_FFN_PAIR : SPATIAL_FFN_PAIR);
            break;
          }
          if (temporal) run_temporal<MODE == STEPS>(e, s, rs, args.has_fields != 0, first_step ? s.hid_in : s.hid_out, args.chunk);
          else if (MODE != ANY || type == SUB_SPATIAL) run_spatial(e, n_items, valid);
          else if (type == SUB_SPATIAL_POST) run_spatial_post(e, s, rs.trow, valid);
          else {
            run_spatial_pre(e, s, rs.trow, valid);
            break;
          }
          wait_round(e, temporal ? LINEAR_OUT_FLIPS : OUT_FLIPS);   // out_proj or linear_out accumulated into the residual
        }
      }
      // y <- residual
      T_RESET(t_io);
      {
        uint32_t v[32];
        tmem_ld32(e.lane_addr + COL_RESID + e.part * 32, v);
        if (args.io_bf16) {
#pragma unroll
          for (int j = 0; j < 4; ++j) *own16(OFF_A, j) = pack8(&v[8 * j]);
          asm volatile("bar.sync %0, 128;" ::"r"(3 + (warp & 3)) : "memory");   // the four warps of these rows
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int at = __shfl_sync(0xffffffffu, rs.trow, 8 * e.part + 2 * i + (lane >> 4));
            const uint4 w = *reinterpret_cast<const uint4*>(smem + OFF_A + io_atom + swz(io_row(i), lane & 7));
            if (at >= 0) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(args.y) + (size_t)at * (2 * D) + (lane & 15) * 16) = w;
          }
        } else if (valid) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[q * 8 + j]);
            store8(args.y + (size_t)rs.trow * D + e.part * 32 + q * 8, f, e.wide);
          }
        }
      }
      T_SINCE(TE_IO, t_io);
    }
    T_SINCE(TE_TOTAL, t_start);
  }
  tc_fence_before();
  __syncthreads();
#ifdef BNB_TIMING
  if (tid < 32) reinterpret_cast<long long*>(args.status)[32 + blockIdx.x * 32 + tid] = time_counters()[tid];
#endif
  if (s_aborted[0] && warp == LOAD_WARP) {
    // a wait ran out: copies may still be in flight towards this CTA's shared memory; give them
    // time to land before the CTA gives it up
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
    // the first code of the call is the one reported
    if ((tid & 31) == 0 && s_aborted[0] > 0 && atomicCAS(args.status, 0, s_aborted[0]) == 0 && args.host_status)
      *static_cast<volatile int*>(args.host_status) = s_aborted[0];
  }
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace pipe

int launch_pipelined(const TrunkArgs& a, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BNB_ERR_NO_DEVICE;
  if (!configured[dev]) {
    for (auto* k : {pipe::k_trunk_pipelined<pipe::ANY>, pipe::k_trunk_pipelined<pipe::WHOLE>, pipe::k_trunk_pipelined<pipe::STEPS>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, pipe::SMEM_BYTES) != cudaSuccess) return BNB_ERR_LAUNCH;
    configured[dev] = true;
  }
  const int grid = a.n_tiles < 148 ? a.n_tiles : 148;
  bool whole = !a.flat_rows;
  for (int i = 0; i < a.n_sub; ++i) whole = whole && (a.sub[i].type == SUB_SPATIAL || a.sub[i].type == SUB_TEMPORAL);
  const auto kernel = a.chunk ? pipe::k_trunk_pipelined<pipe::STEPS> : whole ? pipe::k_trunk_pipelined<pipe::WHOLE> : pipe::k_trunk_pipelined<pipe::ANY>;
  return launch_after(kernel, dim3(grid), pipe::THREADS, pipe::SMEM_BYTES, st, a);
}

}  // namespace tensor
}  // namespace bnb
