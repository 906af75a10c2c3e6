// Row tiles of 128 x 128 on one CTA: the roles, waits and data movement that the kernels with sixteen epilogue
// warps, one issuing and one fetching warp share (train_mlp.cu, split_kernels.cu).
#pragma once

#include "tensor_common.cuh"

namespace bnb {
namespace tensor {

constexpr int EPI_WARPS = 16, EPI_THREADS = 512, MMA_WARP = 16, LOAD_WARP = 17, THREADS = 576;
enum : int { TIMEOUT_FULL = 101, TIMEOUT_FREE = 102, TIMEOUT_ACC = 103, TIMEOUT_OPERAND = 104 };

// What every role needs for its waits.
struct Sync {
  uint32_t bars;           // shared address of the barrier array
  int* status;
  volatile int* aborted;
  __device__ __forceinline__ void wait(int bar, uint32_t parity, int code) const { mbar_wait(bars + 8 * bar, parity & 1u, status, aborted, code); }
};

// The epilogue warps' arrival on an operand barrier.
__device__ __forceinline__ void post(const Sync& s, int bar) {
  fence_proxy_async();
  tc_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(s.bars + 8 * bar);
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory"); }
// Rows move between global memory and the warps in a layout of their own: warp w owns rows 32 (w % 4) .. and
// columns 32 (w / 4) .., and in its i-th request (i < 8) lane l takes the sixteen bytes at row 4 i + l / 8,
// columns 4 (l % 8).. : a request touches four lines.  (With a thread per tile row, as tensor memory has it, each
// request touched 32 lines, and the loads and stores alone took 25 000 of a tile's 67 000 cycles.)
struct RowMap {
  int lane, row0, col;     // first tile row and this lane's first column
  __device__ __forceinline__ int row(int i) const { return row0 + 4 * i + (lane >> 3); }
};
__device__ __forceinline__ RowMap row_map() {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  return {lane, 32 * (warp & 3), 32 * (warp >> 2) + 4 * (lane & 7)};
}
__device__ __forceinline__ void rows_in(float4 (&v)[8], const float* src, const RowMap& m, int first, int rows) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = first + m.row(i);
    v[i] = r < rows ? *reinterpret_cast<const float4*>(src + (size_t)r * D + m.col) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
// Asks L2 for the rows of a tile, `bytes` each, one behind the other (a multiple of 16): their loads, a tile later, then
// find them there.  One thread.
__device__ __forceinline__ void prefetch_rows(const void* src, int tile, int rows, uint32_t bytes) {
  const int first = tile * TILE, n = rows - first < TILE ? rows - first : TILE;
  if (n <= 0) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(static_cast<const uint8_t*>(src) + (size_t)first * bytes), "r"((uint32_t)n * bytes) : "memory");
}
// Per-row sums of one value per request: over the eight lanes of a row here, over the four column parts
// through shared memory.  Returns the totals of this lane's rows; two barriers of the four warps of these rows.
__device__ __forceinline__ void row_sums(float (&v)[8], float* part_sums, const RowMap& m) {
  const int part = threadIdx.x >> 7, bar = 3 + ((threadIdx.x >> 5) & 3);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  if ((m.lane & 7) == 0)
#pragma unroll
    for (int i = 0; i < 8; ++i) part_sums[part * TILE + m.row(i)] = v[i];
  asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float* p = part_sums + m.row(i);
    v[i] = (p[0] + p[TILE]) + (p[2 * TILE] + p[3 * TILE]);
  }
  asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");   // before the next use
}
// 32 accumulator columns from the thread-per-row layout of tensor memory to the row layout, through 4 KB of
// shared memory of the warp's own: in with stage_rows, out with staged_row (i-th request) behind a __syncwarp.
__device__ __forceinline__ void stage_rows(uint32_t taddr, uint8_t* stage, int lane) {
  uint32_t t[32];
  tmem_ld32(taddr, t);
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<uint4*>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_uint4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
}
__device__ __forceinline__ float4 staged_row(const uint8_t* stage, int i, int lane) {
  const int r = 4 * i + (lane >> 3);
  return *reinterpret_cast<const float4*>(stage + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
}
__device__ __forceinline__ void transpose_rows(float4 (&v)[8], uint32_t taddr, uint8_t* stage, const RowMap& m) {
  stage_rows(taddr, stage, m.lane);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = staged_row(stage, i, m.lane);
}
// swz(m.row(i), c8): a row is four further per request and its swizzle alternates, so that the addresses of a loop over i are
// two registers and constants.  (From the row's number the compiler kept eight for each use, and spilled them.)
__device__ __forceinline__ uint32_t row_swz(const RowMap& m, int i, int c8) {
  const int l = m.lane >> 3;
  return (uint32_t)((((m.row0 + l) * 128 + ((c8 ^ l) << 4)) ^ ((i & 1) << 6)) + 512 * i);
}
// this lane's four values of its i-th row as bfloat16 into an operand tile
__device__ __forceinline__ void put_row4(uint8_t* tile, const RowMap& m, int i, const float4& v) {
  *reinterpret_cast<uint2*>(tile + (m.col >> 6) * CHUNK_BYTES + row_swz(m, i, (m.col & 63) >> 3) + ((m.col >> 2) & 1) * 8) =
      make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
}
// The descriptor of an MN-major operand (two 64-wide atoms CHUNK_BYTES apart): see mma_one for the rest.
__device__ __forceinline__ uint32_t desc_mn(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | ((CHUNK_BYTES >> 4) << 16); }
constexpr uint32_t BOTH_MN = (1u << 15) | (1u << 16);

// MMAs over a 128-deep operand pair of K-major tiles: A at a, B at b (low descriptor words), B's second K
// atom b_atom units further.
__device__ __forceinline__ void product128(uint32_t el, uint32_t d, uint32_t a, uint32_t b, uint32_t b_atom, uint32_t idesc) {
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) mma_one<false>(el, d, a + 2 * k, b + 2 * k, idesc, k ? 1u : 0u);
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) mma_one<false>(el, d, a + 1024 + 2 * k, b + b_atom + 2 * k, idesc, 1u);
}


// Kernel frame: barriers (counts given), tensor memory, status.  smem is the dynamic array itself, on a
// 1024-byte boundary because nothing static stands in front of it.
struct Frame {
  uint64_t* bars;
  uint32_t* tmem_slot;
  int* aborted;            // four ints, see mbar_wait
};
template <int N>
__device__ __forceinline__ Frame open_frame(uint8_t* at, int* status, int* host_status, const int (&counts)[N]) {
  static_assert(N <= 28, "barrier area");
  Frame f{reinterpret_cast<uint64_t*>(at), reinterpret_cast<uint32_t*>(at + 8 * 28), reinterpret_cast<int*>(at + 8 * 29)};
  if (threadIdx.x == 0) {
    f.aborted[0] = 0;
    f.aborted[1] = DEFAULT_POLL_LIMIT;
    *reinterpret_cast<int**>(&f.aborted[2]) = host_status;
#pragma unroll
    for (int i = 0; i < N; ++i) mbar_init(smem_u32(&f.bars[i]), counts[i]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    __syncwarp();
    tmem_alloc(smem_u32(f.tmem_slot), 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  let_next_start();
  wait_for_previous();
  if (threadIdx.x == 0 && *status != 0) *static_cast<volatile int*>(f.aborted) = 1;
  return f;
}
constexpr int FRAME_BYTES = 256;
__device__ __forceinline__ void close_frame(const Frame& f, uint32_t tmem) {
  tc_fence_before();
  __syncthreads();
  if (f.aborted[0] && threadIdx.x >= 32 * LOAD_WARP)   // copies may still be on their way here
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  __syncthreads();
  if (threadIdx.x < 32) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace tensor
}  // namespace bnb
