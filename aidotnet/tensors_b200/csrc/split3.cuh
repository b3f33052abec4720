// fp32 operands on the 16-bit tensor cores: x = t0 + t1 + t2 with bf16 terms (8 significant bits each, round to nearest), which is
// exact where bf16's exponents reach: of an x below 2^-110 (7.7e-34) the bits under bf16's smallest number, 2^-133, are lost; above the
// largest bf16 (3.39e38) t0 is an infinity, as for an infinity, and the kernels form such sums again with multiply-adds.  A product of
// two operands is the sum of the six products of terms whose weights together are at least 2^-16 of the whole; the ones left out are
// below 2^-26 of it.  bf16 products are exact in fp32, so what remains is the rounding of
// the accumulation, and for that the leading products t0 * t0 are summed apart from the small ones where it matters.
#pragma once

#include <stdint.h>

#include "ffma2.cuh"
#include "sm100_ptx.cuh"

namespace aidn {
namespace split3 {

constexpr int kTerms = 3;
constexpr int kSmall = 5;   // products besides t0 * t0
__host__ __device__ constexpr int small_a(int i) { return i == 0 ? 0 : (i == 1 ? 1 : (i == 2 ? 0 : (i == 3 ? 2 : 1))); }
__host__ __device__ constexpr int small_b(int i) { return i == 0 ? 1 : (i == 1 ? 0 : (i == 2 ? 2 : (i == 3 ? 0 : 1))); }

// The next term of a pair of floats (packed, lo in bits 0-15), which is taken off the pair.
__device__ __forceinline__ uint32_t take_term(uint64_t& pair) {
  const float2 x = unpack2(pair);
  const uint32_t w = ptx::pack2<true>(x.x, x.y);
  pair = fma2(pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), 0xbf800000bf800000ull, pair);   // - 1 * term: exact
  return w;
}

// Eight neighbouring elements -> one 16-byte chunk of each term's image (128-byte swizzled rows of 64 elements); `addr` is the
// chunk in the image of the first term, the others lie `plane` bytes apart.
__device__ __forceinline__ void store_split8(uint32_t addr, uint32_t plane, ulonglong2 a, ulonglong2 b) {
  uint64_t x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
  for (int t = 0; t < kTerms; ++t) {
    const uint32_t w0 = take_term(x[0]), w1 = take_term(x[1]), w2 = take_term(x[2]), w3 = take_term(x[3]);
    ptx::st_shared_v4(addr + (uint32_t)t * plane, w0, w1, w2, w3);
  }
}

// Four floats in global memory, or zeros.
__device__ __forceinline__ ulonglong2 load4(const float* src, bool valid) {
  return valid ? *reinterpret_cast<const ulonglong2*>(src) : make_ulonglong2(0, 0);
}

// Offset of chunk c (eight elements) of row r in an image of 64-element rows.
__device__ __forceinline__ uint32_t chunk_at(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

}  // namespace split3
}  // namespace aidn
