// Attention forward for fp32 tensors on the fifth-generation tensor cores: both products from operands cut into three bf16
// terms (csrc/split3.cuh), softmax and all sums across key blocks in fp32 registers.  Results are as close to the exact ones as
// those of the fp32 multiply-adds of csrc/sdpa_f32.cu, which cannot leave the FP32 pipe's 74 TFLOP/s.
//
// A CTA owns 128 query rows and walks blocks of 64 keys:
//   warps 0-7   two threads per query row (32 keys and half of the output columns each): S out of TMEM, softmax, the three terms
//               of P back into TMEM over the scores, P V of the block before out of TMEM and added to the output in registers
//   warps 8-11  K and V from global memory through registers into swizzled images of their terms
//   warps 12-13 UMMA issuers (one elected lane each) of the scores and of P V; the first one owns TMEM
//   warps 14-15 a bias or a keep-mask of floats: asynchronous copies into the row warps' tiles
// S(j + 1) and P(j - 1) V are formed while the softmax of block j runs.  TMEM: two score buffers (leading products, small ones;
// P over them) and one pair of output accumulators that start afresh with every block, so that the tensor cores, which
// truncate when they accumulate, never add more than head_dim / 16 or four times into one cell.
// An infinity times a term that is 0 is not a number, and a value above the largest bf16 rounds to an infinity: a score that does
// not come out finite is formed again with multiply-adds, before the two threads of its row exchange their maxima (once they have,
// either may store P over the scores of both).  So is an output that is not finite in the end, from the keys that its row sees: the
// tensor cores multiply every key of a block with all 128 rows, and 0 times an infinity reaches rows that do not see it.
//
// A block is 48 products (24 at head sizes up to 32), so their issue counts: every number of k steps has its own instantiation,
// descriptors are a base plus a constant, and scores and P V have a warp each (with one warp that formed every descriptor anew
// B4 H16 S1024 D64 causal took 164 us, with one warp and constants 95).
//
// Launches with few tiles cut the keys over the CTAs of a cluster, which merge through distributed shared memory.
#include "common.cuh"
#include "ffma2.cuh"
#include "mask_tile.cuh"
#include "sm100_ptx.cuh"
#include "split3.cuh"

namespace aidn {
namespace {

using ptx::mbar_arrive;
using ptx::mbar_init;
using ptx::mbar_wait;
using ptx::smem_u32;
using ptx::tmem_ld16;
using ptx::tmem_ld32;

constexpr int kRows = 128, kKeys = 64, kHalf = 32;
constexpr int kIssuer = 12;   // warp
constexpr int kWorkers = 256, kLoaders = 128, kThreads = 512;   // row threads, loading threads, and a warpgroup with the issuer

// What becomes of a score: nothing, a bias or a keep-mask, the same behind a softcap (whose tanh, 32 times in the row loop, is kept
// out of the instructions of the others).
enum Mode { kPlain, kMask, kSoftcap };

// DP: columns that are loaded (32, 64 or 128); KS: k steps of 16 columns that are multiplied.
template <int DP, int KS, Mode MODE>
struct TCfg {
  static constexpr bool PLAIN = MODE == kPlain;
  static constexpr int kAtoms = (DP + 63) / 64;             // 128-byte columns of an image
  static constexpr int kOut = (KS * 16 + 31) / 32 * 32;     // output columns
  static constexpr int kQPlane = kAtoms * kRows * 128, kKPlane = kAtoms * kKeys * 128;
  static constexpr int kBufs = DP == 128 ? 1 : 2;           // of K, and of V
  static constexpr int kImage = split3::kTerms * kKPlane;
  static constexpr int kKOff = split3::kTerms * kQPlane, kVOff = kKOff + kBufs * kImage;
  static constexpr int kMaskOff = kVOff + kBufs * kImage;
  static constexpr int kXOff = kMaskOff + (PLAIN ? 0 : kWorkers / 32 * masktile::kBytes);
  static constexpr int kXBufs = DP == 128 && !PLAIN ? 1 : 2;   // row maxima: sets of [2 halves][128]
  static constexpr int kBarOff = kXOff + kXBufs * 2 * kRows * 4;
  static constexpr int kNumBars = 1 /*q*/ + 2 /*k_full*/ + 2 /*v_full*/ + 2 /*s_full*/ + 1 /*p_ready*/ + 2 /*o_full*/ + 4 /*pair*/ + 2 /*mask*/;
  static constexpr int kSmem = kBarOff + 8 * kNumBars + 8 + 1024;
  static_assert(kSmem <= 227 * 1024, "shared memory");
  static constexpr int kPartPitch = kOut + 4;               // floats per row of a CTA's partial output, over the images
  static_assert(kRows * (kPartPitch + 2) * 4 <= kMaskOff, "the partial output reuses the images");
  // registers of a row thread, and of the loading and issuing ones (the launch has 128 each)
  static constexpr int kRegRows = DP == 128 ? 160 : 144, kRegRest = 256 - kRegRows;
  static constexpr int kTmemO = 256;                        // leading, then small products
};

struct F32TcParams {
  int32_t splits, vec_out;
  int32_t withhold;   // test hook: the loaders load nothing, so that the bounded waits run out
  uint64_t wait_budget_ns;
};

// The largest of three; a NaN where any of them is one.
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {
  float y;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// What a CTA works on: 128 query rows of a head from row0 on, and n blocks of keys from blk0 on.
struct Place {
  int b, h, n;
  int64_t row0, kv_limit, blk0;
};
__device__ __forceinline__ int64_t visible_end(const SdpaParams& p, int64_t kv_limit, int64_t row) {   // keys [0, end) are visible to the row
  return p.causal && row + p.causal_offset + 1 < kv_limit ? row + p.causal_offset + 1 : kv_limit;
}
__device__ __forceinline__ Place place_of(const SdpaParams& p, int splits) {
  Place at;
  at.b = blockIdx.z;
  at.h = p.head_begin + blockIdx.y;
  const int rank = (int)blockIdx.x % splits, tiles = (int)gridDim.x / splits, at_x = (int)blockIdx.x / splits;
  // under a causal mask the last rows see the most keys: start them first
  at.row0 = (int64_t)(p.causal ? tiles - 1 - at_x : at_x) * kRows;
  at.kv_limit = kv_limit_of(p, at.b);
  const int64_t kend = visible_end(p, at.kv_limit, at.row0 + kRows < p.seq_q ? at.row0 + kRows - 1 : p.seq_q - 1);
  const int64_t blocks = kend > 0 ? (kend + kKeys - 1) / kKeys : 0;
  at.blk0 = rank * blocks / splits;
  at.n = (int)((rank + 1) * blocks / splits - at.blk0);
  return at;
}

// A score that the tensor cores could not form, as the row loop holds them: raw, or the finished logit with a bias or a softcap.
// (Called, not inlined, and two chains of maxima: either costs the row loop registers otherwise, 14.35 -> 14.8 us for B1 H8 S512 D64.)
__device__ __noinline__ float exact_score(const SdpaParams& p, int b, int h, int64_t row, int64_t key) {
  const float* q = static_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1] + row * p.qs[2];
  const float* k = static_cast<const float*>(p.k) + b * p.ks[0] + (h / p.group) * p.ks[1] + key * p.ks[2];
  float s = 0.f;
#pragma unroll 1
  for (int d = 0; d < p.head_dim; d += 4) {   // head sizes are multiples of 4, rows are 16-byte aligned
    const float4 x = *reinterpret_cast<const float4*>(q + d), y = *reinterpret_cast<const float4*>(k + d);
    s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
  }
  if (!(p.softcap > 0.f) && p.mask_kind != AIDN_MASK_ADD_F32) return s;
  return finish_logit(p, s * p.scale, b, h, row, key, key + 1);
}

// Columns col .. col + cols - 1 of `factor` times the output that the CTA's keys add to its row `lrow`, in y where that is not finite
// (m: the maximum that the weights are relative to).
__device__ __noinline__ void exact_output(const SdpaParams& p, int splits, int lrow, float m, float factor, int col, int cols, float* y) {
  const Place at = place_of(p, splits);   // (not handed over: the row loop would hold it in registers)
  const int b = at.b, h = at.h;
  const int64_t row = at.row0 + lrow, key0 = at.blk0 * kKeys, seen = visible_end(p, at.kv_limit, row);
  const int64_t end = (at.blk0 + at.n) * kKeys < seen ? (at.blk0 + at.n) * kKeys : seen;
  const bool raw = !(p.softcap > 0.f) && p.mask_kind != AIDN_MASK_ADD_F32;   // as in the row loop
  const float c = raw ? p.scale * kLog2e : kLog2e;
  if (m == -INFINITY) m = 0.f;
  for (int c0 = 0; c0 < cols; c0 += 16) {
    uint32_t bad = 0;
    for (int e = 0; e < 16; ++e)
      if (col + c0 + e < p.head_dim && !(fabsf(y[c0 + e]) < INFINITY)) bad |= 1u << e;
    if (!bad) continue;
    float s[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) s[e] = 0.f;
    const float* v = static_cast<const float*>(p.v) + b * p.vs[0] + (h / p.group) * p.vs[1] + key0 * p.vs[2] + col + c0;
    uint32_t open = bad;   // columns that are not NaN yet
    for (int64_t key = key0; key < end && open; ++key, v += p.vs[2]) {
      float x = exact_score(p, b, h, row, key);
      if (raw && p.mask_kind != AIDN_MASK_NONE && finish_logit(p, 0.f, b, h, row, key, end) == -INFINITY) x = -INFINITY;
      const float w = x == -INFINITY ? 0.f : ex2_approx((x - m) * c);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        if (!(open & (1u << e))) continue;
        s[e] = fmaf(w, v[e], s[e]);
        if (s[e] != s[e]) open &= ~(1u << e);
      }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e)
      if (bad & (1u << e)) y[c0 + e] = s[e] * factor;
  }
}

template <int DP, int KS, Mode MODE>
__global__ void __launch_bounds__(kThreads, 1) sdpa_f32_sm100_kernel(const __grid_constant__ SdpaParams p, const F32TcParams tp) {
  using C = TCfg<DP, KS, MODE>;
  constexpr bool PLAIN = C::PLAIN;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_q = smem_base + C::kBarOff, bar_k = bar_q + 8, bar_v = bar_k + 16, bar_s = bar_v + 16, bar_p = bar_s + 16, bar_o = bar_p + 8,
                 bar_pair = bar_o + 16, bar_mf = bar_pair + 32, bar_me = bar_mf + 8;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_gen + C::kBarOff + 8 * C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = p.head_dim;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_k + 8 * i, kLoaders / 32);
      mbar_init(bar_v + 8 * i, kLoaders / 32);
      mbar_init(bar_s + 8 * i, 1);
      mbar_init(bar_o + 8 * i, 1);
    }
    mbar_init(bar_q, kWorkers / 32);
    mbar_init(bar_p, kWorkers / 32);
    for (int i = 0; i < 4; ++i) mbar_init(bar_pair + 8 * i, 2);
    mbar_init(bar_mf, 2);
    mbar_init(bar_me, kWorkers / 32);
    ptx::fence_mbar_init();
  }
  if (warp == kIssuer) {
    ptx::tmem_alloc(smem_u32(tmem_ptr_smem), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_wait();   // the set-up above runs under the end of the launch before
  pdl_trigger();
  const Place at = place_of(p, tp.splits);
  const int b = at.b, h = at.h, kvh = h / p.group, rank = (int)blockIdx.x % tp.splits, n = at.n;
  const int64_t row0 = at.row0, kv_limit = at.kv_limit, blk0 = at.blk0;
  const int64_t kend = visible_end(p, kv_limit, row0 + kRows < p.seq_q ? row0 + kRows - 1 : p.seq_q - 1);
  const uint32_t q_s = smem_base, k_s = smem_base + C::kKOff, v_s = smem_base + C::kVOff;

  bool alive = true;
  auto wait = [&](uint32_t bar, int phase) {   // by whole warps
    alive = alive && mbar_wait(bar, (uint32_t)(phase & 1), abort_flag, tp.wait_budget_ns);
    alive = __all_sync(0xffffffffu, alive);
    ptx::tc_fence_after();
  };
  auto publish = [&](uint32_t bar) {   // shared memory written by this warp, for the tensor cores
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  constexpr int CPR = DP / 8;   // chunks of eight columns per row
  // Where the mask of rows 32 * quarter .. and keys 32 * half .. of block j lies, and how much of it there is.
  const bool add = !PLAIN && p.mask_kind == AIDN_MASK_ADD_F32;
  const bool tiles = add || (!PLAIN && p.mask_kind == AIDN_MASK_KEEP_F32 && p.mask_stride[2] != 0);   // floats: through the row warps' tiles
  auto mask_at = [&](int j, int quarter, int half, int& rows, int& keys) {
    const int64_t key = (blk0 + j) * kKeys + half * kHalf, r0 = row0 + quarter * 32;
    rows = masktile::clamp32(p.seq_q - r0);
    keys = masktile::clamp32(kv_limit - key);
    return b * p.mask_stride[0] + h * p.mask_stride[1] + r0 * p.mask_stride[2] + key * p.mask_stride[3];
  };
  if (warp < kWorkers / 32) {
    ptx::setmaxnreg_inc<C::kRegRows>();
    const int quarter = warp & 3, half = warp >> 2, lrow = quarter * 32 + lane;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int64_t row = row0 + lrow;
    const int64_t row_end = row < p.seq_q ? visible_end(p, kv_limit, row) : kend;
    constexpr int kCols = C::kOut / 2;                           // output columns of a half
    int pair_phase = 0;
    auto pair_sync = [&] {   // the two warps of the same rows
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_pair + 8 * quarter);
      wait(bar_pair + 8 * quarter, pair_phase++);
    };
    const bool masked = !PLAIN && p.mask_kind != AIDN_MASK_NONE, keeps = masked && !tiles;
    // The mask of the warp's 32 rows and its 32 keys of block j: floats in its tile, bytes (and one row of floats for all) as bits of the
    // thread's row, one block ahead; lanes take keys, so that either is read in whole lines.  Keep-masks of floats as bits, by the row warps
    // themselves, took B1 H12 S783 D64 46.7 -> 52.4 us, H60 511 x 352 49.2 -> 52.8.
    const uint32_t mask_s = smem_base + (uint32_t)(C::kMaskOff + warp * masktile::kBytes);
    uint32_t keep_next = 0;
    auto fetch_keep = [&](int j) {
      int rows, keys;
      const int64_t at0 = mask_at(j, quarter, half, rows, keys);
      keep_next = masktile::keep_bits_of<true>(p, at0, p.mask_stride[2], p.mask_stride[3], rows, keys, lane);
    };
    // p = 2^((s - m) c): s is the raw score and c = scale log2(e), or the finished logit and log2(e) with a bias or a softcap
    const bool raw = MODE != kSoftcap && !add;
    const float c = raw ? p.scale * kLog2e : kLog2e;
    const uint64_t c2 = pack2(c, c), scale2 = pack2(p.scale, p.scale);

    uint64_t acc[kCols / 2];
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) acc[i] = 0;
    float m = -INFINITY, l = 0.f;
    if (n > 0) {
      if (keeps) fetch_keep(0);
      const float* qb = static_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1];
      {
        constexpr int kPer = kRows * CPR / kWorkers;
        ulonglong2 v[kPer][2];   // all requested before the first is cut: one latency
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const int idx = tid + e * kWorkers, r = idx / CPR, d = idx % CPR * 8;
          const float* src = qb + (row0 + r) * p.qs[2] + d;
          const bool ok = row0 + r < p.seq_q;
          v[e][0] = split3::load4(src, ok && d < D);
          v[e][1] = split3::load4(src + 4, ok && d + 4 < D);
        }
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const int idx = tid + e * kWorkers, r = idx / CPR, ch = idx % CPR;
          split3::store_split8(q_s + (uint32_t)((ch >> 3) * kRows * 128) + split3::chunk_at(r, ch & 7), C::kQPlane, v[e][0], v[e][1]);
        }
      }
      publish(bar_q);
      auto x_of = [&](int j, int h) -> float& {   // what half h of the row exchanges at block j
        return reinterpret_cast<float*>(smem_gen + C::kXOff)[((C::kXBufs == 2 ? j & 1 : 0) * 2 + h) * kRows + lrow];
      };
      auto add_block = [&](int i) {   // P V of block i onto the output
        wait(bar_o + 8 * (i & 1), i >> 1);
        if (!alive) return;
        const uint32_t t_o = t_row + (uint32_t)(C::kTmemO + half * kCols);
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += 16) {
          uint64_t hi[8], lo[8];
          tmem_ld16(t_o + (uint32_t)c0, reinterpret_cast<uint32_t*>(hi));
          tmem_ld16(t_o + (uint32_t)(C::kOut + c0), reinterpret_cast<uint32_t*>(lo));
          ptx::tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[c0 / 2 + e] = add2(acc[c0 / 2 + e], add2(hi[e], lo[e]));
        }
      };

      for (int j = 0; j < n; ++j) {
        const uint32_t t_s = t_row + (uint32_t)((j & 1) * 128 + half * kHalf);
        wait(bar_s + 8 * (j & 1), j >> 1);
        if (!alive) break;
        uint64_t s[kHalf / 2];
        {
          uint64_t lo[kHalf / 2];
          tmem_ld32(t_s, reinterpret_cast<uint32_t*>(s));
          tmem_ld32(t_s + 64, reinterpret_cast<uint32_t*>(lo));
          ptx::tc_wait_ld();
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) s[k] = add2(s[k], lo[k]);
        }
        // keys of this half that the row sees
        const int64_t left = row_end - (blk0 + j) * kKeys - half * kHalf;
        int seen = left < 0 ? 0 : (left > kHalf ? kHalf : (int)left);
        if constexpr (PLAIN) {
          if (__any_sync(0xffffffffu, seen < kHalf)) {   // a block on the diagonal or at the end of the keys
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) {
              const float2 x = unpack2(s[k]);
              s[k] = pack2(2 * k < seen ? x.x : -INFINITY, 2 * k + 1 < seen ? x.y : -INFINITY);
            }
          }
        }
        uint32_t keep = seen < kHalf ? (1u << seen) - 1u : 0xffffffffu;
        if constexpr (!PLAIN) {
          if constexpr (MODE == kSoftcap) {
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) {
              const float2 x = unpack2(s[k]);
              s[k] = pack2(p.softcap * tanhf(x.x * p.scale / p.softcap), p.softcap * tanhf(x.y * p.scale / p.softcap));
            }
          }
          if (tiles) {
            wait(bar_mf, j);
            if (!alive) break;
            if (add) {
#pragma unroll
              for (int k = 0; k < kHalf / 2; k += 2) {
                const float4 m4 = masktile::row4(mask_s, k / 2, lane);
                const uint64_t b0 = pack2(m4.x, m4.y), b1 = pack2(m4.z, m4.w);
                s[k] = MODE == kSoftcap ? add2(s[k], b0) : fma2(s[k], scale2, b0);
                s[k + 1] = MODE == kSoftcap ? add2(s[k + 1], b1) : fma2(s[k + 1], scale2, b1);
              }
            } else {
              uint32_t w = 0;
#pragma unroll
              for (int k = 0; k < kHalf; k += 4) {
                const float4 m4 = masktile::row4(mask_s, k / 4, lane);
                w |= (m4.x != 0.f ? 1u << k : 0u) | (m4.y != 0.f ? 2u << k : 0u) | (m4.z != 0.f ? 4u << k : 0u) | (m4.w != 0.f ? 8u << k : 0u);
              }
              keep &= w;
            }
            __syncwarp();   // the values have been read
            if (lane == 0) mbar_arrive(bar_me);
          } else if (keeps) {
            keep &= keep_next;
          }
          if (__any_sync(0xffffffffu, keep != 0xffffffffu)) {
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) {
              const float2 x = unpack2(s[k]);
              s[k] = pack2(keep & (1u << (2 * k)) ? x.x : -INFINITY, keep & (2u << (2 * k)) ? x.y : -INFINITY);
            }
          }
        }
        float mt = -INFINITY, mt1 = -INFINITY;
#pragma unroll
        for (int k = 0; k < kHalf / 2; k += 2) {
          const float2 x = unpack2(s[k]), y = unpack2(s[k + 1]);
          mt = fmax3_nan(mt, x.x, x.y);
          mt1 = fmax3_nan(mt1, y.x, y.y);
        }
        mt = fmax3_nan(mt, mt1, mt1);
        if (!(mt < INFINITY) && row < p.seq_q) {
          uint32_t bad = 0;
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) {
            const float2 x = unpack2(s[k]);
            bad |= (fabsf(x.x) < INFINITY ? 0u : 1u << (2 * k)) | (fabsf(x.y) < INFINITY ? 0u : 2u << (2 * k));
          }
          for (bad &= keep; bad; bad &= bad - 1) {
            const int i = __ffs(bad) - 1;
            const float v = exact_score(p, b, h, row, (blk0 + j) * kKeys + half * kHalf + i);
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) {
              const float2 x = unpack2(s[k]);
              s[k] = pack2(2 * k == i ? v : x.x, 2 * k + 1 == i ? v : x.y);
            }
          }
          mt = -INFINITY;   // (what is not a number does not count: its weight is not a number either way)
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) {
            const float2 x = unpack2(s[k]);
            mt = fmaxf(mt, fmaxf(x.x, x.y));
          }
        }
        __syncwarp();
        x_of(j, half) = mt;
        pair_sync();   // the row's other thread has left its maximum, and has read its scores
        const float m_new = fmaxf(m, fmaxf(mt, x_of(j, 1 - half)));
        if (C::kXBufs == 1) pair_sync();
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        const float corr = ex2_approx((m - m_use) * c);
        m = m_new;
        uint64_t sums = 0;
        const uint64_t neg = pack2(-m_use, -m_use);
#pragma unroll
        for (int k = 0; k < kHalf / 2; ++k) {
          const float2 x = unpack2(mul2(add2(s[k], neg), c2));
          s[k] = pack2(ex2_approx(x.x), ex2_approx(x.y));
          sums = add2(sums, s[k]);
        }
        l = fmaf(l, corr, sum2(sums));
        if (keeps && j + 1 < n) fetch_keep(j + 1);
        if (j > 0) {
          add_block(j - 1);
          if (!alive) break;
          const uint64_t corr2 = pack2(corr, corr);
#pragma unroll
          for (int i = 0; i < kCols / 2; ++i) acc[i] = mul2(acc[i], corr2);
        }
#pragma unroll
        for (int t = 0; t < split3::kTerms; ++t) {
          uint32_t w[kHalf / 2];
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) w[k] = split3::take_term(s[k]);
          ptx::tmem_st16(t_row + (uint32_t)((j & 1) * 128 + t * 32 + half * 16), w);
        }
        ptx::tc_wait_st();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p);
      }
      if (alive) add_block(n - 1);
      // the row's sum is in two halves
      if (alive) {
        x_of(n, half) = l;
        pair_sync();
        l = half == 0 ? l + x_of(n, 1) : x_of(n, 0) + l;
      }
    }

    float inv = 1.f;
    float* dst;
    if (tp.splits > 1) {   // this CTA's partial, over the images (every product has read them)
      if (n > 0) asm volatile("bar.sync 1, 256;" ::: "memory");
      if (!alive) {   // the CTAs that merge it must not take it for a result
#pragma unroll
        for (int i = 0; i < kCols / 2; ++i) acc[i] = pack2(NAN, NAN);
      }
      float* part = reinterpret_cast<float*>(smem_gen);
      dst = part + lrow * C::kPartPitch + half * kCols;
#pragma unroll
      for (int i = 0; i < kCols; i += 4)
        *reinterpret_cast<ulonglong2*>(dst + i) = make_ulonglong2(acc[i / 2], acc[i / 2 + 1]);
      if (half == 0) {
        part[kRows * C::kPartPitch + lrow] = raw ? m * p.scale : m;
        part[kRows * (C::kPartPitch + 1) + lrow] = l;
      }
    } else if (alive && row < p.seq_q) {
      inv = l > 0.f ? 1.f / l : 0.f;
      const uint64_t inv2 = pack2(inv, inv);
      dst = static_cast<float*>(p.out) + b * p.os[0] + h * p.os[1] + row * p.os[2] + half * kCols;
#pragma unroll
      for (int i = 0; i < kCols; i += 4) {
        if (half * kCols + i >= D) continue;   // D is a multiple of 4
        const uint64_t x = mul2(acc[i / 2], inv2), y = mul2(acc[i / 2 + 1], inv2);
        if (tp.vec_out) {
          *reinterpret_cast<ulonglong2*>(dst + i) = make_ulonglong2(x, y);
        } else {
          const float2 f = unpack2(x), g = unpack2(y);
          dst[i] = f.x;
          dst[i + 1] = f.y;
          dst[i + 2] = g.x;
          dst[i + 3] = g.y;
        }
      }
      if (p.lse && half == 0) p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q + row] = l > 0.f ? (raw ? m * p.scale : m) + logf(l) : -INFINITY;
    }
    uint64_t chk = 0;
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) chk = add2(chk, acc[i]);
    // (a sum of weights that is not a number leaves nothing to save)
    if (!(fabsf(sum2(chk)) < INFINITY) && l == l && alive && row < p.seq_q) exact_output(p, tp.splits, lrow, m, inv, half * kCols, kCols, dst);
  } else if (warp < (kWorkers + kLoaders) / 32) {
    ptx::setmaxnreg_dec<C::kRegRest>();
    // Blocks go in pieces of up to four chunks a thread, in the order K(0), V(0), K(1), ..., the next piece requested before the
    // current one is stored.  Keys past kend (padding beyond kv_len, the causal future) and columns past head_dim are zeros and
    // are not read.
    constexpr int kPer = kKeys * CPR / kLoaders, kPiece = kPer < 4 ? kPer : 4, kPieces = kPer / kPiece, kRowsAt = kLoaders / CPR;
    const int lt = tid - kWorkers, ch = lt % CPR;
    const float* kb = static_cast<const float*>(p.k) + b * p.ks[0] + kvh * p.ks[1];
    const float* vb = static_cast<const float*>(p.v) + b * p.vs[0] + kvh * p.vs[1];
    const uint32_t at = (uint32_t)((ch >> 3) * kKeys * 128);
    auto load = [&](int q, ulonglong2 (&reg)[kPiece][2]) {
      if (q >= n * 2 * kPieces) return;
      const int j = q / (2 * kPieces), r = q % (2 * kPieces);
      const bool is_v = r >= kPieces;
      const int row0_at = lt / CPR + (is_v ? r - kPieces : r) * kPiece * kRowsAt;
      const int64_t stride = is_v ? p.vs[2] : p.ks[2], key = (blk0 + j) * kKeys + row0_at, left = kend - key;
      const float* src = (is_v ? vb : kb) + key * stride + ch * 8;
#pragma unroll
      for (int e = 0; e < kPiece; ++e) {
        const bool ok = e * kRowsAt < left;
        reg[e][0] = split3::load4(src, ok && ch * 8 < D);
        reg[e][1] = split3::load4(src + 4, ok && ch * 8 + 4 < D);
        src += kRowsAt * stride;
      }
    };
    auto store = [&](int q, const ulonglong2 (&reg)[kPiece][2]) {
      const int j = q / (2 * kPieces), r = q % (2 * kPieces), slot = j % C::kBufs;
      const bool is_v = r >= kPieces;
      const int piece = is_v ? r - kPieces : r;
      const int i = j - C::kBufs;   // the last block that used the buffer: its scores, its part of the output have been formed
      // (two barriers each for scores and outputs: a phase of one cannot pass unseen before its buffer is filled again)
      if (i >= 0 && piece == 0) wait((is_v ? bar_o : bar_s) + 8 * (i & 1), i >> 1);
      if (!alive) return;
      const uint32_t image = (is_v ? v_s : k_s) + (uint32_t)(slot * C::kImage) + at;
#pragma unroll
      for (int e = 0; e < kPiece; ++e)
        split3::store_split8(image + split3::chunk_at(lt / CPR + (piece * kPiece + e) * kRowsAt, ch & 7), C::kKPlane, reg[e][0], reg[e][1]);
      if (piece == kPieces - 1) publish((is_v ? bar_v : bar_k) + 8 * slot);
    };
    if (n > 0 && !tp.withhold) {
      ulonglong2 even[kPiece][2], odd[kPiece][2];
      load(0, even);
      for (int q = 0; q < n * 2 * kPieces && alive; q += 2) {
        load(q + 1, odd);
        store(q, even);
        load(q + 2, even);
        if (alive) store(q + 1, odd);
      }
    }
  } else {
    ptx::setmaxnreg_dec<C::kRegRest>();
    const bool leader = ptx::elect_one();
    auto given = [&](uint32_t bar, int phase) {
      alive = alive && mbar_wait(bar, (uint32_t)(phase & 1), abort_flag, tp.wait_budget_ns);
      ptx::tc_fence_after();
      return alive;
    };
    if (warp == kIssuer) {
      constexpr uint32_t idesc = ptx::make_idesc(kRows, kKeys, true, false);
      const uint64_t qd = ptx::make_smem_desc(q_s, 16, 1024);
      if (n > 0) given(bar_q, 0);
      for (int i = 0; i < n && alive; ++i) {
        const int slot = i % C::kBufs;
        if (!given(bar_k + 8 * slot, i / C::kBufs)) break;
        // the buffer of the scores of block i - 2, over which its P lies, has been read
        if (i >= 2 && !given(bar_o + 8 * (i & 1), (i - 2) >> 1)) break;
        const uint64_t kd = ptx::make_smem_desc(k_s + (uint32_t)(slot * C::kImage), 16, 1024);
        const uint32_t d = tmem_base + (uint32_t)((i & 1) * 128);
        auto product = [&](uint32_t dst, int ta, int tb, bool fresh) {
#pragma unroll
          for (int kk = 0; kk < KS; ++kk) {
            const uint64_t x = qd + (uint64_t)((ta * C::kQPlane + (kk >> 2) * kRows * 128 + (kk & 3) * 32) >> 4);
            const uint64_t y = kd + (uint64_t)((tb * C::kKPlane + (kk >> 2) * kKeys * 128 + (kk & 3) * 32) >> 4);
            if (leader) ptx::mma_ss(dst, x, y, idesc, !fresh || kk > 0 ? 1u : 0u);
          }
        };
        product(d, 0, 0, true);
#pragma unroll
        for (int t = 0; t < split3::kSmall; ++t) product(d + 64, split3::small_a(t), split3::small_b(t), t == 0);
        if (leader) ptx::tc_commit(bar_s + 8 * (i & 1));
      }
    } else if (warp == kIssuer + 1) {
      constexpr uint32_t idesc = ptx::make_idesc(kRows, C::kOut, true, true);
      for (int j = 0; j < n; ++j) {
        const int slot = j % C::kBufs;
        if (!given(bar_v + 8 * slot, j / C::kBufs) || !given(bar_p, j)) break;
        const uint64_t vd = ptx::make_smem_desc(v_s + (uint32_t)(slot * C::kImage), kKeys * 128, 1024);
        const uint32_t t_p = tmem_base + (uint32_t)((j & 1) * 128);
        auto product = [&](uint32_t dst, int ta, int tb, bool fresh) {
#pragma unroll
          for (int kk = 0; kk < kKeys / 16; ++kk) {
            const uint64_t y = vd + (uint64_t)((tb * C::kKPlane + kk * 2048) >> 4);
            if (leader) ptx::mma_ts(dst, t_p + (uint32_t)(ta * 32 + kk * 8), y, idesc, !fresh || kk > 0 ? 1u : 0u);
          }
        };
        product(tmem_base + C::kTmemO, 0, 0, true);
#pragma unroll
        for (int t = 0; t < split3::kSmall; ++t) product(tmem_base + C::kTmemO + C::kOut, split3::small_a(t), split3::small_b(t), t == 0);
        if (leader) ptx::tc_commit(bar_o + 8 * (j & 1));
      }
    } else if (tiles) {   // half of every row warp's tiles each
      const int half = warp - kIssuer - 2;
      for (int j = 0; j < n; ++j) {
        if (j > 0) wait(bar_me, j - 1);
        if (!alive) break;
#pragma unroll 1
        for (int quarter = 0; quarter < 4; ++quarter) {
          int rows, keys;
          const int64_t at0 = mask_at(j, quarter, half, rows, keys);
          masktile::request(smem_base + (uint32_t)(C::kMaskOff + (half * 4 + quarter) * masktile::kBytes), static_cast<const float*>(p.mask) + at0,
                            p.mask_stride[2], p.mask_stride[3], rows, keys, lane);
        }
        cp_async_wait_f<0>();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_mf);
      }
    }
  }

  // TMEM goes back before the CTAs of the cluster wait for one another: one of them may still be waiting for its columns behind
  // a CTA of another launch, which may be waiting for these.
  __syncwarp();
  ptx::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    ptx::abort_grace();
    if (tid == 0 && p.status) atomicOr(p.status, kStatusTimeout);
    __syncthreads();
  }
  if (warp == kIssuer) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
  if (tp.splits > 1) {
    __syncwarp();
    cluster_sync_all();   // every CTA's partial is written
    if (warp < kWorkers / 32 && !*abort_flag) {
      const uint32_t part = smem_base, pm = part + kRows * C::kPartPitch * 4, pl = pm + kRows * 4;
      const int d4s = D / 4;
      for (int idx = rank * kWorkers + tid; idx < kRows * d4s; idx += tp.splits * kWorkers) {
        const int r = idx / d4s, d = (idx - r * d4s) * 4;
        const int64_t row = row0 + r;
        if (row >= p.seq_q) continue;
        float ms[8], ls[8], M = -INFINITY, lsum = 0.f;
        float4 o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          ms[i] = -INFINITY;
          ls[i] = 0.f;
          o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (i < tp.splits) {
            ms[i] = ld_cluster_f32(pm + (uint32_t)(r * 4), (uint32_t)i);
            ls[i] = ld_cluster_f32(pl + (uint32_t)(r * 4), (uint32_t)i);
            o[i] = ld_cluster_f4(part + (uint32_t)((r * C::kPartPitch + d) * 4), (uint32_t)i);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) M = fmaxf(M, ms[i]);
        const float M_use = M == -INFINITY ? 0.f : M;
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= tp.splits) continue;
          const float w = expf(ms[i] - M_use);
          lsum = fmaf(w, ls[i], lsum);
          y[0] = fmaf(w, o[i].x, y[0]); y[1] = fmaf(w, o[i].y, y[1]); y[2] = fmaf(w, o[i].z, y[2]); y[3] = fmaf(w, o[i].w, y[3]);
        }
        const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
        float* out = static_cast<float*>(p.out) + b * p.os[0] + h * p.os[1] + row * p.os[2] + d;
        if (tp.vec_out) {
          *reinterpret_cast<float4*>(out) = make_float4(y[0] * inv, y[1] * inv, y[2] * inv, y[3] * inv);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) out[e] = y[e] * inv;
        }
        if (p.lse && d == 0) p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q + row] = lsum > 0.f ? M + logf(lsum) : -INFINITY;
      }
    }
    __syncwarp();
    cluster_sync_all();   // nobody reads this CTA's shared memory any more
  }
}

template <int DP, int KS, Mode MODE>
cudaError_t launch_t(const SdpaParams& p, F32TcParams tp, cudaStream_t stream) {
  auto kern = sdpa_f32_sm100_kernel<DP, KS, MODE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TCfg<DP, KS, MODE>::kSmem);
  if (e != cudaSuccess) return e;
  return launch_dependent_cluster(kern, dim3((unsigned)((p.seq_q + kRows - 1) / kRows * tp.splits), (unsigned)p.head_count, (unsigned)p.batch), kThreads,
                                  dim3((unsigned)tp.splits), TCfg<DP, KS, MODE>::kSmem, stream, p, tp);
}

template <int DP, int KS>
cudaError_t launch_mode(const SdpaParams& p, const F32TcParams& tp, Mode mode, cudaStream_t stream) {
  if (mode == kPlain) return launch_t<DP, KS, kPlain>(p, tp, stream);
  return mode == kMask ? launch_t<DP, KS, kMask>(p, tp, stream) : launch_t<DP, KS, kSoftcap>(p, tp, stream);
}

}  // namespace

// fp32 calls of the register-tiled kernel (f32_supported) that this one takes: those that give a tile of 128 rows enough to do.  A CTA
// takes the same time for 16 rows as for 128, about 7 us with its set-up and one block of keys (D 64; 6 at 32, 11 at 128), the
// multiply-adds work for the rows that are there.  Both sides measured, in us (multiply-adds -> this kernel):
//   more CTAs than SMs   16 x 32 heads 64 x 64: D 32 21 -> 25, D 64 29 -> 31, D 128 77 -> 43; 16 x 64: D 64 21 -> 29, D 128 42 -> 41;
//                        16 x 512: D 64 97 -> 90; 16 x 16 heads 100 x 100: D 32 27 -> 17, D 64 41 -> 21
//   fewer                2 heads 16 x 16: D 32 7.0 -> 8.7, D 128 10.8 -> 12.4; 4 x 8 heads 16 x 64: D 32 9.7 -> 8.7, D 64 12.7 -> 9.5;
//                        8 heads 100 x 100: D 64 15.2 -> 12.7, D 128 16.8 -> 18.8; 2 heads 100 x 300: D 80 27 -> 19
//   softcap              a tanh per score, the same on both sides: 16 x 32 heads 64 x 64: D 64 37 -> 54, D 128 84 -> 68; 8 x 16 heads
//                        197 x 197, causal: D 64 74 -> 80; 2 x 8 heads 333 x 333: D 64 39 -> 35; 8 heads 100 x 100: D 128 19 -> 25
// The error against 64 bits is below that of the multiply-adds in all of them (by a fifth to a half).  But where a log-sum-exp is
// asked for and its backward pass stays on the multiply-adds, so does the forward pass: the roundings of the one cancel against
// those of the other only in the same arithmetic (gradients of 4 x 8 heads of 333 rows: 3.9e-7 mixed, 3.6e-7 not).
bool f32_sm100_supported(const SdpaParams& p, int dtype) {
  const int64_t tiles = (p.seq_q + kRows - 1) / kRows;
  if (dtype != AIDN_F32 || p.no_tcgen05 || (p.lse && !backward_f32_sm100_fits(p)) || tiles == 0 || tiles * 8 > 0x7fffffff) return false;
  const bool many = tiles * p.head_count * p.batch > 148, wide = p.head_dim > 64;
  const int64_t pairs = p.seq_q / tiles * p.seq_kv;   // of a tile
  if (wide) return many ? pairs >= (p.softcap > 0.f ? 4096 : 2048) : p.seq_kv > (p.softcap > 0.f ? 256 : 128);
  if (p.softcap > 0.f) return p.seq_kv > 256;
  return pairs >= (many ? 8192 : 1024);
}

cudaError_t launch_f32_sm100(const SdpaParams& p, cudaStream_t stream) {
  F32TcParams tp;
  tp.vec_out = reinterpret_cast<uintptr_t>(p.out) % 16 == 0;
  for (int i = 0; i < 3; ++i) tp.vec_out = tp.vec_out && p.os[i] % 4 == 0;
  tp.withhold = p.expire;
  tp.wait_budget_ns = p.expire ? 20000000ull : ptx::kWaitBudgetNs;   // 20 ms in the time-out test
  const int64_t tiles = (p.seq_q + kRows - 1) / kRows * p.head_count * p.batch, blocks = (p.seq_kv + kKeys - 1) / kKeys;
  tp.splits = 1;
  while (tp.splits < 8 && tiles * tp.splits * 2 <= 148 && tp.splits * 2 <= blocks) tp.splits *= 2;
  const Mode mode = p.softcap > 0.f ? kSoftcap : (p.mask_kind == AIDN_MASK_NONE ? kPlain : kMask);
  if (p.head_dim <= 32) return launch_mode<32, 2>(p, tp, mode, stream);
  if (p.head_dim <= 64) return launch_mode<64, 4>(p, tp, mode, stream);
  if (p.head_dim <= 96) return launch_mode<128, 6>(p, tp, mode, stream);
  return launch_mode<128, 8>(p, tp, mode, stream);
}

}  // namespace aidn
