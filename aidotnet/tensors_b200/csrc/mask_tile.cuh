// The explicit mask of a warp's 32 rows for kernels whose threads own a row each: a lane takes a key, so that memory is read along rows
// in whole lines, and the lane that owns a row gets its part as bits (keep-masks) or through shared memory (a bias).  A thread that
// walked its own row touched 32 lines an instruction, and where rows are not a multiple of 16 bytes, with 64 of them a block: the
// forward pass of B2 H3 251 x 268 D128 with a keep-mask took 35 us, the training step of B1 H28 S523 D64 with a bias 300.
#pragma once

#include <stdint.h>

#include "ffma2.cuh"

namespace aidn {
namespace masktile {

constexpr int kBytes = 32 * 32 * 4;   // shared memory of a warp's tile: 32 rows and 32 keys of a bias

// Where in a tile key k of row r lies: 16-byte chunks swizzled, so that neither lanes along a row nor lanes down a column of chunks meet
// in a bank.
__device__ __forceinline__ uint32_t at(int r, int k) { return (uint32_t)(r * 128 + (((k >> 2) ^ (r & 7)) << 4) + (k & 3) * 4); }

// One value of each of 32 rows at the lane's key.  `src` is row 0, key 0; of rows >= `rows` and keys >= `keys`, which are not read, the
// value is another one's (loads that depend on the lane would each be a branch).
// WHOLE: whole tiles apart, which advance without a look at `rows`.  fp32 forward passes with a keep-mask of bytes 254.0 -> 221.7 us (13 x 30 heads of 396, D 64,
// causal; by the row warps' predicated loads 245.8); the backward kernels only get larger by it (16 bits, small calls, up to 8 % slower).
template <bool WHOLE = false, typename E>
__device__ __forceinline__ void load_rows(const E* src, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane, E (&x)[32]) {
  if (rows <= 0 || keys <= 0) {
#pragma unroll
    for (int r = 0; r < 32; ++r) x[r] = E(0);
    return;
  }
  const E* p = src + (lane < keys ? lane : keys - 1) * key_stride;
  if (WHOLE && rows >= 32) {
#pragma unroll
    for (int r = 0; r < 32; ++r) x[r] = p[r * row_stride];
    return;
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    x[r] = *p;
    p += r + 1 < rows ? row_stride : 0;
  }
}

// Bit k of the lane's row: key k is kept (32 keys).
template <bool WHOLE = false, typename E>
__device__ __forceinline__ uint32_t keep_bits(const E* src, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  if (row_stride == 0) return __ballot_sync(0xffffffffu, lane < keys && src[lane * key_stride] != E(0));   // one row of the mask for all
  E x[32];
  load_rows<WHOLE>(src, row_stride, key_stride, rows, keys, lane, x);
  uint32_t mine = 0;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const uint32_t w = __ballot_sync(0xffffffffu, x[r] != E(0));
    if (r == lane) mine = w;
  }
  return keys >= 32 ? mine : (keys <= 0 ? 0u : mine & ((1u << keys) - 1u));
}

// The same of a mask of either type (AIDN_MASK_KEEP_U8, AIDN_MASK_KEEP_F32), `first` elements into it.
template <bool WHOLE = false>
__device__ __forceinline__ uint32_t keep_bits_of(const SdpaParams& p, int64_t first, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  if (p.mask_kind == AIDN_MASK_KEEP_U8) return keep_bits<WHOLE>(static_cast<const uint8_t*>(p.mask) + first, row_stride, key_stride, rows, keys, lane);
  return keep_bits<WHOLE>(static_cast<const float*>(p.mask) + first, row_stride, key_stride, rows, keys, lane);
}

// Bit r: row r is kept at the lane's key.
template <typename E>
__device__ __forceinline__ uint32_t keep_column(const E* src, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  E x[32];
  load_rows(src, row_stride, key_stride, rows, keys, lane, x);
  uint32_t mine = 0;
#pragma unroll
  for (int r = 0; r < 32; ++r) mine |= x[r] != E(0) ? 1u << r : 0u;
  return rows >= 32 ? mine : (rows <= 0 ? 0u : mine & ((1u << rows) - 1u));
}
__device__ __forceinline__ uint32_t keep_column_of(const SdpaParams& p, int64_t first, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  if (p.mask_kind == AIDN_MASK_KEEP_U8) return keep_column(static_cast<const uint8_t*>(p.mask) + first, row_stride, key_stride, rows, keys, lane);
  return keep_column(static_cast<const float*>(p.mask) + first, row_stride, key_stride, rows, keys, lane);
}

// 32 rows and 32 keys of a bias on their way into the tile (cp.async; the caller waits for them and then for its warp).
__device__ __forceinline__ void request(uint32_t tile, const float* src, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  const float* p = src + lane * key_stride;
  const bool in = lane < keys;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const bool ok = in && r < rows;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tile + at(r, lane)), "l"(ok ? p : src), "r"(ok ? 4u : 0u) : "memory");
    p += row_stride;
  }
  cp_async_commit_f();
}

// The same for rows that are keys: the lane's key is the tile's row, the mask's row the tile's column.
__device__ __forceinline__ void request_columns(uint32_t tile, const float* src, int64_t row_stride, int64_t key_stride, int rows, int keys, int lane) {
  const float* p = src + lane * key_stride;
  const bool in = lane < keys;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const bool ok = in && r < rows;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tile + at(lane, r)), "l"(ok ? p : src), "r"(ok ? 4u : 0u) : "memory");
    p += row_stride;
  }
  cp_async_commit_f();
}

// ... and out of registers (load_rows).
__device__ __forceinline__ void put(uint32_t tile, const float (&x)[32], int lane) {
#pragma unroll
  for (int r = 0; r < 32; ++r) asm volatile("st.shared.f32 [%0], %1;" ::"r"(tile + at(r, lane)), "f"(x[r]) : "memory");
}

// Keys 4 c .. 4 c + 3 of the lane's row.
__device__ __forceinline__ float4 row4(uint32_t tile, int c, int lane) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(tile + at(lane, 4 * c)) : "memory");
  return v;
}

__device__ __forceinline__ int clamp32(int64_t n) { return n < 0 ? 0 : (n > 32 ? 32 : (int)n); }

}  // namespace masktile
}  // namespace aidn
