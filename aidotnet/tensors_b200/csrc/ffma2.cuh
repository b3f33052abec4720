// Building blocks of the fp32 kernels: two fused multiply-adds per instruction on a register pair, and 16-byte
// asynchronous copies into shared memory.
//
// `fma.rn.f32x2` (sm_100) does the two roundings of two scalar fmaf.  It saves issue slots, which the shared-memory loads
// that feed it need: measured on register operands 109 multiply-adds per SM and cycle against 92 for scalar fmaf.
#pragma once

#include <stdint.h>

#include "common.cuh"

namespace aidn {

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ float sum2(uint64_t v) {
  const float2 f = unpack2(v);
  return f.x + f.y;
}

struct Pair2 { uint64_t a, b; };   // four consecutive floats
__device__ __forceinline__ Pair2 lds_pairs(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}

// 16 bytes global -> shared; `valid` false writes zeros and reads nothing.
__device__ __forceinline__ void cp_async16_f(float* dst, const void* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const uint32_t n = valid ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit_f() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_f() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One 16-byte chunk of a row as floats: 4 of fp32, 8 of a 16-bit type.
template <typename T>
struct Chunk16 { static constexpr int N = 16 / sizeof(T); };

template <typename T>
__device__ __forceinline__ void store_chunk(float* dst, const uint4& u) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<uint4*>(dst) = u;
  } else {
    T t[8];
    *reinterpret_cast<uint4*>(t) = u;
#pragma unroll
    for (int i = 0; i < 8; i += 4)
      *reinterpret_cast<float4*>(dst + i) = make_float4(to_float<T>(t[i]), to_float<T>(t[i + 1]), to_float<T>(t[i + 2]), to_float<T>(t[i + 3]));
  }
}

// What the explicit mask contributes to a block of R x K logits, fetched before the products that the logits come from.
template <int R, int K>
struct MaskBlock { float v[R][K]; };

// `origin` is the mask offset of the tile's first row and key; row(i) and key(k) count from there.  `seen(i, k)` says
// which elements are read at all (a masked-out or padded position of the mask tensor is not touched).
template <int R, int K, typename Row, typename Key, typename Seen>
__device__ __forceinline__ void fetch_mask(const SdpaParams& p, int64_t origin, Row row, Key key, Seen seen, MaskBlock<R, K>& m) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int64_t base = origin + row(i) * p.mask_stride[2];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t at = base + key(k) * p.mask_stride[3];
      m.v[i][k] = 0.f;
      if (seen(i, k)) {
        if (p.mask_kind == AIDN_MASK_KEEP_U8) m.v[i][k] = static_cast<const uint8_t*>(p.mask)[at] ? 1.f : 0.f;
        else m.v[i][k] = static_cast<const float*>(p.mask)[at];
      }
    }
  }
}

// Which (row, key) of a tile may be visible, in tile coordinates: row < rows, key < keys and, under a causal mask,
// key - row <= diag.  `span` is anything above both extents of the tile.
struct TileBounds {
  int rows, keys, diag;
  __device__ __forceinline__ TileBounds(const SdpaParams& p, int64_t row0, int64_t key0, int64_t kv_limit, int span) {
    auto clamp = [span](int64_t x) { return (int)(x < -span ? -span : (x > span ? span : x)); };
    rows = clamp(p.seq_q - row0);
    keys = clamp(kv_limit - key0);
    diag = p.causal ? clamp(row0 + p.causal_offset - key0) : span;
  }
  __device__ __forceinline__ bool seen(int row, int key) const { return row < rows && key < keys && key - row <= diag; }
};

// The rule of finish_logit on a scaled logit whose mask value is at hand.
__device__ __forceinline__ float finish_logit_with(const SdpaParams& p, float s, bool seen, float mask) {
  if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
  if (!seen) return -INFINITY;
  if (p.mask_kind == AIDN_MASK_NONE) return s;
  if (p.mask_kind == AIDN_MASK_ADD_F32) return s + mask;
  return mask == 0.f ? -INFINITY : s;
}

// 16-byte vector access to rows of `elem` bytes per element: base and every stride must allow it.
inline bool rows_aligned16(const void* ptr, const int64_t* st, int elem) {
  if (reinterpret_cast<uintptr_t>(ptr) % 16) return false;
  for (int i = 0; i < 3; ++i)
    if ((st[i] * elem) % 16) return false;
  return true;
}

}  // namespace aidn
