// Attention backward of fp32 tensors on the fifth-generation tensor cores (head_dim <= 64): dQ and dK / dV as two launches of one
// kernel, every operand as three bf16 terms (csrc/split3.cuh).  The formulas and the mask rules are those of
// sdpa_backward.cu, and the accuracy is that of the fp32 multiply-adds of sdpa_backward_f32.cu.
//
// A CTA keeps 128 rows of one sequence ("own") in shared memory and walks blocks of 64 rows of the other past them:
//   KEYS = true  (dK, dV): X = its K rows, Y = its V rows; a block is U = Q rows, W = dO rows of one query head of the group.
//   KEYS = false (dQ):     X = its Q rows, Y = its dO rows; a block is U = K rows, W = V rows.
//   S = X U^T    dP = Y W^T    acc0 += dS U    KEYS: acc1 += P W      with P = exp(S scale - lse), dS = P (dP - delta)
//   warps 0-7   two threads per own row (32 rows of the block and half of the gradient's columns each): S and dP out of TMEM, the
//               terms of P and dS into it, and the gradients of the block before added up in registers
//   warps 8-11  the blocks from global memory through registers into swizzled images of their terms, two buffers
//   warps 12-13 UMMA issuers (one elected lane each) of the scores and of the gradients; the first one owns TMEM
//   warps 14-15 a bias: asynchronous copies into the row warps' tiles (by the row warps themselves they were half of a block's 6000 cycles)
// The scores of block j + 1 are formed while the row threads work on block j.  The gradient accumulators start afresh with every
// block, so that the tensor cores, which truncate when they accumulate, never add more than four times into one cell.
// An infinity times a term that is 0 is not a number, a value above the largest bf16 rounds to an infinity, and a block is multiplied
// with rows that take no part with one another: a score that does not come out finite is formed again with multiply-adds, and so
// is an element of a gradient that is not finite in the end.
//
// Launches with few tiles cut the walk over the CTAs of a cluster, which add their gradients in rank order through distributed
// shared memory: every gradient is summed in a fixed order (deterministic, no atomics).
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

constexpr int kOwn = 128, kStr = 64, kHalf = 32, kDP = 64;
constexpr int kIssuer = 12;   // warp
constexpr int kWorkers = 256, kLoaders = 128, kThreads = 512;   // row threads, loading threads, and a warpgroup with the issuer
constexpr int kOwnPlane = kOwn * 128, kStrPlane = kStr * 128;
constexpr int kStrImage = split3::kTerms * kStrPlane;             // U or W of one block
constexpr int kYOff = split3::kTerms * kOwnPlane, kUOff = 2 * kYOff;
constexpr int kRowOff = kUOff + 4 * kStrImage;                    // -lse and -delta of streamed query rows: [2 buffers][2][64]
constexpr int kMaskOff = kRowOff + 2 * 2 * kStr * 4;
constexpr int kBars = 10;                                         // full[2], g_full[2], s_full, s_empty, p_ready, xy_full, mask_full, mask_empty
constexpr int bar_off(bool plain) { return kMaskOff + (plain ? 0 : kWorkers * 32 * 4); }
constexpr int smem_bytes(bool plain) { return bar_off(plain) + 8 * kBars + 8 + 1024; }
static_assert(smem_bytes(false) <= 227 * 1024, "shared memory");
constexpr int kPartPitch = kDP + 4;   // floats per row of a CTA's partial gradient, over the images
static_assert(2 * kOwn * kPartPitch * 4 <= kRowOff, "the partial gradients reuse the images");
// TMEM columns: S, dP | terms of P | terms of dS | acc0 | acc1 (dV).  dQ and dV keep leading and small products apart; for dK
// there are no columns left.
constexpr int kTS = 0, kTdP = 64, kTP = 128, kTdS = 224, kTAcc0 = 320, kTAcc1 = 384;

struct BwdTcParams {
  int32_t splits;
  int32_t withhold;   // test hook: the loaders load nothing, so that the bounded waits run out
  uint64_t wait_budget_ns;
};

// The sum that the tensor cores could not form: an infinity times a term that is 0 is not a number.
__device__ __noinline__ float dot_rows(const float* x, const float* u, int n) {
  float s = 0.f;
  for (int i = 0; i < n; ++i) s = fmaf(x[i], u[i], s);
  return s;
}

// What a CTA works on: 128 own rows from own0 on, of which those before own_end take part, and n steps from s_begin on: blocks of
// streamed rows [first, last), per_head of them for each query head from h0 on (hl0 within the shard).
struct Place {
  int b, hl0, h0, per_head, s_begin, n;
  int64_t own0, own_end, kv_limit, first, last;
};
template <bool KEYS>
__device__ __forceinline__ Place place_of(const SdpaParams& p, int splits) {
  Place at;
  at.b = blockIdx.z;
  at.hl0 = KEYS ? blockIdx.y * p.group : blockIdx.y;
  at.h0 = p.head_begin + at.hl0;
  const int rank = (int)blockIdx.x % splits, tiles = (int)gridDim.x / splits, at_x = (int)blockIdx.x / splits;
  // under a causal mask the last query rows and the first keys have the most to do: start them first
  at.own0 = (int64_t)(!KEYS && p.causal ? tiles - 1 - at_x : at_x) * kOwn;
  at.kv_limit = kv_limit_of(p, at.b);
  // streamed rows [first, last) of one head that any of the CTA's own rows takes part with
  at.first = 0;
  at.last = KEYS ? p.seq_q : at.kv_limit;
  if (p.causal) {
    if constexpr (KEYS) {
      at.first = at.own0 - p.causal_offset;              // query rows that see the CTA's first key
      at.first = at.first > 0 ? at.first / kStr * kStr : 0;
    } else {
      int64_t last_row = at.own0 + kOwn - 1;
      if (last_row > p.seq_q - 1) last_row = p.seq_q - 1;
      if (last_row + p.causal_offset + 1 < at.last) at.last = last_row + p.causal_offset + 1;
    }
  }
  if (KEYS && at.own0 >= at.kv_limit) at.last = 0;
  at.own_end = KEYS ? at.kv_limit : p.seq_q;
  at.per_head = at.last > at.first ? (int)((at.last - at.first + kStr - 1) / kStr) : 0;
  const int64_t steps = (int64_t)at.per_head * (KEYS ? p.group : 1);
  at.s_begin = (int)(rank * steps / splits);
  at.n = (int)((rank + 1) * steps / splits) - at.s_begin;
  return at;
}

// Columns col .. col + cols - 1 (at most 32) of `factor` times what the CTA's blocks add to the gradient of its own row `lrow` - dQ
// or dK, or with of_v dV - in y where that is not finite: from the rows that take part with it.
template <bool KEYS>
__device__ __noinline__ void exact_gradient(const BwdParams& bp, int splits, int lrow, bool of_v, float factor, int col, int cols, float* y) {
  const SdpaParams& p = bp.p;
  const Place at = place_of<KEYS>(p, splits);   // (not handed over: the row loop would hold it in registers)
  const int D = p.head_dim, kvh = at.h0 / p.group;
  const int64_t own = at.own0 + lrow;
  uint32_t bad = 0;
  for (int e = 0; e < cols; ++e)
    if (col + e < D && !(fabsf(y[e]) < INFINITY)) bad |= 1u << e;
  float s[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) s[e] = 0.f;
  uint32_t open = own < at.own_end ? bad : 0;   // columns that are not NaN yet
  for (int j = 0; j < at.n && open; ++j) {
    const int g = KEYS ? (at.s_begin + j) / at.per_head : 0, h = at.h0 + g;
    const int64_t base = at.first + (int64_t)(at.s_begin + j - g * at.per_head) * kStr;
    const float* qb = static_cast<const float*>(p.q) + at.b * p.qs[0] + h * p.qs[1];
    const float* gb = static_cast<const float*>(bp.dout) + at.b * bp.dos[0] + h * bp.dos[1];
    const float* kb = static_cast<const float*>(p.k) + at.b * p.ks[0] + kvh * p.ks[1];
    const float* vb = static_cast<const float*>(p.v) + at.b * p.vs[0] + kvh * p.vs[1];
    for (int64_t r = base; r < base + kStr && r < at.last && open; ++r) {
      const int64_t query = KEYS ? r : own, key = KEYS ? own : r;
      if (p.causal && key > query + p.causal_offset) continue;
      const float val = finish_logit(p, dot_rows(qb + query * p.qs[2], kb + key * p.ks[2], D) * p.scale, at.b, h, query, key, at.kv_limit);
      const float lse = p.lse[((int64_t)at.b * p.num_q_heads + h) * p.seq_q + query];
      float w = val == -INFINITY || lse == -INFINITY ? 0.f : ex2_approx((val - lse) * kLog2e);
      if (!of_v)
        w *= dot_rows(gb + query * bp.dos[2], vb + key * p.vs[2], D) - bp.delta[((int64_t)at.b * p.head_count + at.hl0 + g) * p.seq_q + query];
      const float* u = (of_v ? gb + query * bp.dos[2] : (KEYS ? qb + query * p.qs[2] : kb + key * p.ks[2])) + col;
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        if (!(open & (1u << e))) continue;
        s[e] = fmaf(w, u[e], s[e]);
        if (s[e] != s[e]) open &= ~(1u << e);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 32; ++e)
    if (bad & (1u << e)) y[e] = s[e] * factor;
}

// One block's gradient (N column pairs of the thread's row) onto the registers; APART: small products kDP columns on.
template <bool APART, int N>
__device__ __forceinline__ void add_gradient(uint32_t t_acc, uint64_t (&acc)[N]) {
#pragma unroll
  for (int c0 = 0; c0 < 2 * N; c0 += 16) {
    uint64_t hi[8], lo[8];
    tmem_ld16(t_acc + (uint32_t)c0, reinterpret_cast<uint32_t*>(hi));
    if (APART) tmem_ld16(t_acc + (uint32_t)(kDP + c0), reinterpret_cast<uint32_t*>(lo));
    ptx::tc_wait_ld();
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[c0 / 2 + e] = add2(acc[c0 / 2 + e], APART ? add2(hi[e], lo[e]) : hi[e]);
  }
}
template <int N>
__device__ __forceinline__ bool all_finite(const uint64_t (&acc)[N]) {   // (or their sum is not)
  uint64_t chk = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) chk = add2(chk, acc[i]);
  return fabsf(sum2(chk)) < INFINITY;
}

// KS: k steps of 16 columns (2: head sizes up to 32).
// dQ waits for the kernel that formed delta.  dK / dV, which follows on the stream, needs nothing of dQ: it starts when all of dQ's CTAs
// have begun - by then every launch before dQ is complete, and what it reads of theirs dQ hands over - and takes the SMs that dQ leaves idle; it
// ends only after dQ has, so that what comes next on the stream may rely on both.
template <int KS, bool KEYS, bool PLAIN>
__global__ void __launch_bounds__(kThreads, 1) bwd_f32_sm100_kernel(const __grid_constant__ BwdParams bp, const BwdTcParams tp) {
  const SdpaParams& p = bp.p;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_full = smem_base + bar_off(PLAIN), bar_g = bar_full + 16, bar_s = bar_g + 16, bar_se = bar_s + 8, bar_p = bar_se + 8, bar_xy = bar_p + 8, bar_mf = bar_xy + 8, bar_me = bar_mf + 8;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_gen + bar_off(PLAIN) + 8 * kBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = p.head_dim;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_full + 8 * i, kLoaders / 32);
      mbar_init(bar_g + 8 * i, 1);
    }
    mbar_init(bar_xy, kWorkers / 32);
    mbar_init(bar_s, 1);
    mbar_init(bar_se, kWorkers / 32);
    mbar_init(bar_p, kWorkers / 32);
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
  if (!KEYS) {
    pdl_wait();
    if (warp == kIssuer + 1) pdl_hand_over();   // (a warp that has to wait first; it speaks for the CTA)
  } else {   // waits at its end
    pdl_take_over();
    pdl_trigger();
  }
  const Place at = place_of<KEYS>(p, tp.splits);
  const int b = at.b, hl0 = at.hl0, h0 = at.h0, kvh = h0 / p.group, kv_heads = p.head_count / p.group, rank = (int)blockIdx.x % tp.splits;
  const int per_head = at.per_head, s_begin = at.s_begin, n = at.n;
  const int64_t own0 = at.own0, own_end = at.own_end, kv_limit = at.kv_limit, first = at.first, last = at.last;
  const uint32_t x_s = smem_base, y_s = smem_base + kYOff, u_s = smem_base + kUOff;   // buffer i: U at u_s + 2 i images, W behind it

  const float* kb = static_cast<const float*>(p.k) + b * p.ks[0] + (int64_t)kvh * p.ks[1];
  const float* vb = static_cast<const float*>(p.v) + b * p.vs[0] + (int64_t)kvh * p.vs[1];
  const float* qb = static_cast<const float*>(p.q) + b * p.qs[0] + (int64_t)h0 * p.qs[1];
  const float* gb = static_cast<const float*>(bp.dout) + b * bp.dos[0] + (int64_t)h0 * bp.dos[1];
  const int64_t ustr = KEYS ? p.qs[2] : p.ks[2], wstr = KEYS ? bp.dos[2] : p.vs[2];
  constexpr int CPR = KS * 2;   // chunks of eight columns per row
  struct Block {   // of step s: its head within the group, its first streamed row
    int g;
    int64_t base;
  };
  auto block_of = [&](int j) {
    const int s = s_begin + j, g = KEYS ? s / per_head : 0;
    return Block{g, first + (int64_t)(s - g * per_head) * kStr};
  };
  // Where the mask of own rows 32 * quarter .. and rows 32 * half .. of block j lies, and how much of it there is.
  const bool add = !PLAIN && p.mask_kind == AIDN_MASK_ADD_F32;
  auto mask_at = [&](int j, int quarter, int half, int& rows, int& keys) {
    const Block bk = block_of(j);
    const int64_t o0 = own0 + quarter * 32, s0 = bk.base + half * kHalf, key = KEYS ? o0 : s0, query = KEYS ? s0 : o0;
    rows = masktile::clamp32(p.seq_q - query);
    keys = masktile::clamp32(kv_limit - key);
    return b * p.mask_stride[0] + (h0 + bk.g) * p.mask_stride[1] + query * p.mask_stride[2] + key * p.mask_stride[3];
  };
  bool alive = true;
  auto wait = [&](uint32_t bar, int phase) {   // by whole warps
    alive = alive && mbar_wait(bar, (uint32_t)(phase & 1), abort_flag, tp.wait_budget_ns);
    alive = __all_sync(0xffffffffu, alive);
    ptx::tc_fence_after();
  };
  if (warp < kWorkers / 32) {
    ptx::setmaxnreg_inc<168>();
    const int quarter = warp & 3, half = warp >> 2, lrow = quarter * 32 + lane;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int64_t own = own0 + lrow;
    constexpr int kCols = KS * 8;           // gradient columns of a half
    const float* xb = KEYS ? kb : qb;
    const float* yb = KEYS ? vb : gb;
    const int64_t xstr = KEYS ? p.ks[2] : p.qs[2], ystr = KEYS ? p.vs[2] : bp.dos[2];
    // The mask of the warp's 32 own rows and its 32 rows of block j: a bias in its tile, a keep-mask as bits of the thread's row, one block
    // ahead; lanes take keys, so that either is read in whole lines.
    const uint32_t mask_s = smem_base + (uint32_t)(kMaskOff + warp * masktile::kBytes);
    uint32_t keep = ~0u;
    auto fetch_keep = [&](int j) {
      int rows, keys;
      const int64_t at0 = mask_at(j, quarter, half, rows, keys);
      keep = KEYS ? masktile::keep_column_of(p, at0, p.mask_stride[2], p.mask_stride[3], rows, keys, lane)
                  : masktile::keep_bits_of(p, at0, p.mask_stride[2], p.mask_stride[3], rows, keys, lane);
    };

    uint64_t acc0[kCols / 2], acc1[KEYS ? kCols / 2 : 1];
#pragma unroll
    for (int c = 0; c < kCols / 2; ++c) {
      acc0[c] = 0;
      if constexpr (KEYS) acc1[c] = 0;
    }
    if (n > 0) {
      {
        constexpr int kPer = kOwn * CPR / kWorkers;
        ulonglong2 xv[kPer][2], yv[kPer][2];   // all requested before the first is cut: one latency
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const int idx = tid + e * kWorkers, r = idx / CPR, d = idx % CPR * 8;
          const bool lo = own0 + r < own_end && d < D, hi = own0 + r < own_end && d + 4 < D;
          const float* xr = xb + (own0 + r) * xstr + d;
          const float* yr = yb + (own0 + r) * ystr + d;
          xv[e][0] = split3::load4(xr, lo);
          xv[e][1] = split3::load4(xr + 4, hi);
          yv[e][0] = split3::load4(yr, lo);
          yv[e][1] = split3::load4(yr + 4, hi);
        }
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const int idx = tid + e * kWorkers;
          split3::store_split8(x_s + split3::chunk_at(idx / CPR, idx % CPR), kOwnPlane, xv[e][0], xv[e][1]);
          split3::store_split8(y_s + split3::chunk_at(idx / CPR, idx % CPR), kOwnPlane, yv[e][0], yv[e][1]);
        }
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_xy);
      if (!PLAIN && !add) fetch_keep(0);
      float nl_own = -INFINITY, nd_own = 0.f;   // -lse (-inf where no key is visible, which makes every P 0) and -delta
      if (!KEYS && own < p.seq_q) {
        const float lse = p.lse[((int64_t)b * p.num_q_heads + h0) * p.seq_q + own];
        nl_own = lse == -INFINITY ? -INFINITY : -lse;
        nd_own = -bp.delta[((int64_t)b * p.head_count + hl0) * p.seq_q + own];
      }
      const uint64_t scale2 = pack2(p.scale, p.scale), log2e2 = pack2(kLog2e, kLog2e);

      auto add_block = [&](int j) {
        wait(bar_g + 8 * (j & 1), j >> 1);
        if (!alive) return;
        add_gradient<!KEYS>(t_row + (uint32_t)(kTAcc0 + half * kCols), acc0);
        if constexpr (KEYS) add_gradient<true>(t_row + (uint32_t)(kTAcc1 + half * kCols), acc1);
      };

      for (int j = 0; j < n; ++j) {
        const Block bk = block_of(j);
        const int64_t s0 = bk.base + half * kHalf;   // the thread's first streamed row
        if constexpr (KEYS) wait(bar_full + 8 * (j & 1), j >> 1);   // (for the rows' -lse and -delta)
        wait(bar_s, j);
        if (!alive) break;
        uint64_t pr[kHalf / 2], ds[kHalf / 2];
        tmem_ld32(t_row + (uint32_t)(kTS + half * kHalf), reinterpret_cast<uint32_t*>(pr));
        tmem_ld32(t_row + (uint32_t)(kTdP + half * kHalf), reinterpret_cast<uint32_t*>(ds));
        ptx::tc_wait_ld();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_se);
        const float* row_s = reinterpret_cast<const float*>(smem_gen + kRowOff) + (j & 1) * 128 + half * kHalf;
        {
          uint64_t chk = 0;
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) chk = add2(chk, add2(pr[k], ds[k]));
          if (__any_sync(0xffffffffu, !(fabsf(sum2(chk)) < INFINITY))) {
            const float* us = KEYS ? qb + (int64_t)bk.g * p.qs[1] : kb;
            const float* ws = KEYS ? gb + (int64_t)bk.g * bp.dos[1] : vb;
#pragma unroll
            for (int k = 0; k < kHalf; ++k) {
              const int64_t r = s0 + k;
              const bool in = r < last && own < own_end;
              float2 x = unpack2(pr[k / 2]), y = unpack2(ds[k / 2]);
              float& sv = k & 1 ? x.y : x.x;
              float& dv = k & 1 ? y.y : y.x;
              if (in && !(fabsf(sv) < INFINITY)) {
                sv = dot_rows(xb + own * xstr, us + r * ustr, D);
                if ((KEYS ? row_s[k] : nl_own) == -INFINITY) sv = 0.f;   // P is 0 whatever the logit is
              }
              if (in && !(fabsf(dv) < INFINITY)) dv = dot_rows(yb + own * ystr, ws + r * wstr, D);
              pr[k / 2] = pack2(x.x, x.y);
              ds[k / 2] = pack2(y.x, y.y);
            }
          }
          __syncwarp();
        }
        // streamed rows [lo, hi) of this half take part with the own row
        int64_t from = 0, to = last - s0;
        if (own >= own_end) to = 0;
        if (KEYS && p.causal) from = own - p.causal_offset - s0;
        if (!KEYS && p.causal && own + p.causal_offset + 1 - s0 < to) to = own + p.causal_offset + 1 - s0;
        const int lo = from < 0 ? 0 : (from > kHalf ? kHalf : (int)from), hi = to < 0 ? 0 : (to > kHalf ? kHalf : (int)to);
        const bool whole = !__any_sync(0xffffffffu, lo > 0 || hi < kHalf);
        if constexpr (!PLAIN) {   // the finished logits
          if (add) {
            wait(bar_mf, j);
            if (!alive) break;
#pragma unroll
            for (int k = 0; k < kHalf / 2; k += 2) {
              const float4 m4 = masktile::row4(mask_s, k / 2, lane);
              pr[k] = fma2(pr[k], scale2, pack2(m4.x, m4.y));
              pr[k + 1] = fma2(pr[k + 1], scale2, pack2(m4.z, m4.w));
            }
            __syncwarp();   // the values have been read
            if (lane == 0) mbar_arrive(bar_me);
          } else {
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) {
              const float2 x = unpack2(mul2(pr[k], scale2));
              pr[k] = pack2(keep & (1u << (2 * k)) ? x.x : -INFINITY, keep & (2u << (2 * k)) ? x.y : -INFINITY);
            }
          }
        }
#pragma unroll
        for (int k4 = 0; k4 < kHalf; k4 += 4) {
          ulonglong2 nl = make_ulonglong2(pack2(nl_own, nl_own), pack2(nl_own, nl_own)), nd = make_ulonglong2(pack2(nd_own, nd_own), pack2(nd_own, nd_own));
          if constexpr (KEYS) {
            nl = *reinterpret_cast<const ulonglong2*>(row_s + k4);
            nd = *reinterpret_cast<const ulonglong2*>(row_s + 64 + k4);
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int k = k4 / 2 + e;
            const uint64_t nlk = e ? nl.y : nl.x;
            uint64_t t;
            if constexpr (PLAIN) {
              t = fma2(pr[k], scale2, nlk);
            } else {
              const float2 x = unpack2(pr[k]), q = unpack2(nlk);
              t = add2(pack2(q.x == -INFINITY ? -INFINITY : x.x, q.y == -INFINITY ? -INFINITY : x.y), nlk);
            }
            const float2 y = unpack2(mul2(t, log2e2));
            pr[k] = pack2(ex2_approx(y.x), ex2_approx(y.y));
            if (!whole) {
              const float2 x = unpack2(pr[k]);
              pr[k] = pack2(2 * k >= lo && 2 * k < hi ? x.x : 0.f, 2 * k + 1 >= lo && 2 * k + 1 < hi ? x.y : 0.f);
            }
            ds[k] = mul2(pr[k], add2(ds[k], e ? nd.y : nd.x));
            if (!whole) {
              const float2 x = unpack2(ds[k]);
              ds[k] = pack2(2 * k >= lo && 2 * k < hi ? x.x : 0.f, 2 * k + 1 >= lo && 2 * k + 1 < hi ? x.y : 0.f);
            }
          }
        }
        if constexpr (!PLAIN) {
          if (!add && j + 1 < n) fetch_keep(j + 1);
        }
        if (j > 0) add_block(j - 1);   // the terms of P and dS of block j - 1 have been read, and so have its gradients
        if (!alive) break;
#pragma unroll
        for (int t = 0; t < split3::kTerms; ++t) {
          uint32_t w[kHalf / 2];
          if constexpr (KEYS) {
#pragma unroll
            for (int k = 0; k < kHalf / 2; ++k) w[k] = split3::take_term(pr[k]);
            ptx::tmem_st16(t_row + (uint32_t)(kTP + t * 32 + half * 16), w);
          }
#pragma unroll
          for (int k = 0; k < kHalf / 2; ++k) w[k] = split3::take_term(ds[k]);
          ptx::tmem_st16(t_row + (uint32_t)(kTdS + t * 32 + half * 16), w);
        }
        ptx::tc_wait_st();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p);
      }
      if (alive) add_block(n - 1);
    }

    const int64_t out_rows = KEYS ? p.seq_kv : p.seq_q;
    const bool out_of_range = !all_finite(acc0) || (KEYS && !all_finite(acc1));
    float *dst0, *dst1 = nullptr;
    if (tp.splits > 1) {   // this CTA's partial gradients, over the images (every product has read them)
      if (n > 0) asm volatile("bar.sync 1, 256;" ::: "memory");
      if (!alive) {   // the CTAs that add it up must not take it for a result
#pragma unroll
        for (int c = 0; c < kCols / 2; ++c) {
          acc0[c] = pack2(NAN, NAN);
          if constexpr (KEYS) acc1[c] = pack2(NAN, NAN);
        }
      }
      dst0 = reinterpret_cast<float*>(smem_gen) + lrow * kPartPitch + half * kCols;
      dst1 = dst0 + kOwn * kPartPitch;
#pragma unroll
      for (int c = 0; c < kCols; c += 4) {
        *reinterpret_cast<ulonglong2*>(dst0 + c) = make_ulonglong2(acc0[c / 2], acc0[c / 2 + 1]);
        if constexpr (KEYS) *reinterpret_cast<ulonglong2*>(dst1 + c) = make_ulonglong2(acc1[c / 2], acc1[c / 2 + 1]);
      }
    } else if (alive && own < out_rows) {
      const int64_t base = KEYS ? ((int64_t)b * kv_heads + blockIdx.y) * out_rows : ((int64_t)b * p.head_count + hl0) * out_rows;
      const int64_t to = (base + own) * D + half * kCols;
      const uint64_t scale2 = pack2(p.scale, p.scale);
      dst0 = (KEYS ? bp.dk : bp.dq) + to;
      if constexpr (KEYS) dst1 = bp.dv + to;
#pragma unroll
      for (int c = 0; c < kCols; c += 4) {
        if (half * kCols + c >= D) continue;   // D is a multiple of 4
        *reinterpret_cast<ulonglong2*>(dst0 + c) = make_ulonglong2(mul2(acc0[c / 2], scale2), mul2(acc0[c / 2 + 1], scale2));
        if constexpr (KEYS) *reinterpret_cast<ulonglong2*>(dst1 + c) = make_ulonglong2(acc1[c / 2], acc1[c / 2 + 1]);
      }
    }
    if (out_of_range && alive && own < out_rows) {
      exact_gradient<KEYS>(bp, tp.splits, lrow, false, tp.splits > 1 ? 1.f : p.scale, half * kCols, kCols, dst0);
      if constexpr (KEYS) exact_gradient<KEYS>(bp, tp.splits, lrow, true, 1.f, half * kCols, kCols, dst1);
    }
  } else if (warp < (kWorkers + kLoaders) / 32) {
    ptx::setmaxnreg_dec<104>();
    const int lt = tid - kWorkers;
    constexpr int kPer = kStr * CPR / kLoaders;
    ulonglong2 ureg[kPer][2], wreg[kPer][2];
    float rowreg = 0.f;
    auto load = [&](int j) {
      const Block bk = block_of(j);
      const int d = lt % CPR * 8;
      const int64_t r0 = bk.base + lt / CPR;
      const float* us = (KEYS ? qb + (int64_t)bk.g * p.qs[1] : kb) + r0 * ustr + d;
      const float* ws = (KEYS ? gb + (int64_t)bk.g * bp.dos[1] : vb) + r0 * wstr + d;
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const bool ok = r0 + e * (kLoaders / CPR) < last;
        ureg[e][0] = split3::load4(us, ok && d < D);
        ureg[e][1] = split3::load4(us + 4, ok && d + 4 < D);
        wreg[e][0] = split3::load4(ws, ok && d < D);
        wreg[e][1] = split3::load4(ws + 4, ok && d + 4 < D);
        us += (kLoaders / CPR) * ustr;
        ws += (kLoaders / CPR) * wstr;
      }
      if constexpr (KEYS) {   // -lse (threads 0-63; -inf where no key is visible, which makes every P 0) and -delta
        const int64_t r = bk.base + (lt & 63);
        if (lt < 64) {
          const float v = r < p.seq_q ? p.lse[((int64_t)b * p.num_q_heads + h0 + bk.g) * p.seq_q + r] : -INFINITY;
          rowreg = v == -INFINITY ? -INFINITY : -v;
        } else {
          rowreg = r < p.seq_q ? -bp.delta[((int64_t)b * p.head_count + hl0 + bk.g) * p.seq_q + r] : 0.f;
        }
      }
    };
    if (n > 0) load(0);
    for (int j = 0; j < n && !tp.withhold; ++j) {
      if (j >= 2) wait(bar_g + 8 * (j & 1), (j - 2) >> 1);   // the gradients of block j - 2 have read the buffer
      if (!alive) break;
      const uint32_t u = u_s + (uint32_t)((j & 1) * 2 * kStrImage);
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const uint32_t at = u + split3::chunk_at(lt / CPR + e * (kLoaders / CPR), lt % CPR);
        split3::store_split8(at, kStrPlane, ureg[e][0], ureg[e][1]);
        split3::store_split8(at + (uint32_t)kStrImage, kStrPlane, wreg[e][0], wreg[e][1]);
      }
      if (KEYS) reinterpret_cast<float*>(smem_gen + kRowOff)[(j & 1) * 128 + lt] = rowreg;
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_full + 8 * (j & 1));
      if (j + 1 < n) load(j + 1);
    }
  } else {
    ptx::setmaxnreg_dec<72>();
    const bool leader = ptx::elect_one();
    auto given = [&](uint32_t bar, int phase) {
      alive = alive && mbar_wait(bar, (uint32_t)(phase & 1), abort_flag, tp.wait_budget_ns);
      ptx::tc_fence_after();
      return alive;
    };
    // (a block is up to 96 products: descriptors are a base plus a constant)
    if (warp == kIssuer) {
      constexpr uint32_t idesc = ptx::make_idesc(kOwn, kStr, true, false);
      const uint64_t xd = ptx::make_smem_desc(x_s, 16, 1024);
      if (n > 0) given(bar_xy, 0);
      for (int j = 0; j < n && alive; ++j) {
        if (!given(bar_full + 8 * (j & 1), j >> 1) || (j > 0 && !given(bar_se, j - 1))) break;
        const uint64_t ud = ptx::make_smem_desc(u_s + (uint32_t)((j & 1) * 2 * kStrImage), 16, 1024);
        auto product = [&](int which, int ta, int tb, bool fresh) {
#pragma unroll
          for (int kk = 0; kk < KS; ++kk) {
            const uint64_t x = xd + (uint64_t)((which * kYOff + ta * kOwnPlane + kk * 32) >> 4);
            const uint64_t y = ud + (uint64_t)((which * kStrImage + tb * kStrPlane + kk * 32) >> 4);
            if (leader) ptx::mma_ss(tmem_base + (which ? kTdP : kTS), x, y, idesc, !fresh || kk > 0 ? 1u : 0u);
          }
        };
        // the small products first: what they lose when the leading ones are added is below the last bit of the sum
#pragma unroll
        for (int which = 0; which < 2; ++which) {
#pragma unroll
          for (int t = 0; t < split3::kSmall; ++t) product(which, split3::small_a(t), split3::small_b(t), t == 0);
          product(which, 0, 0, false);
        }
        if (leader) ptx::tc_commit(bar_s);
      }
    } else if (warp == kIssuer + 1) {
      constexpr uint32_t idesc = ptx::make_idesc(kOwn, KS * 16, true, true);
      for (int j = 0; j < n; ++j) {
        if (!given(bar_p, j)) break;
        const uint64_t ud = ptx::make_smem_desc(u_s + (uint32_t)((j & 1) * 2 * kStrImage), kStrPlane, 1024);
        auto product = [&](uint32_t dst, int which, int ta, int tb, bool fresh) {
#pragma unroll
          for (int kk = 0; kk < kStr / 16; ++kk) {
            const uint64_t y = ud + (uint64_t)((which * kStrImage + tb * kStrPlane + kk * 2048) >> 4);
            if (leader) ptx::mma_ts(tmem_base + dst, tmem_base + (uint32_t)((which ? kTP : kTdS) + ta * 32 + kk * 8), y, idesc, !fresh || kk > 0 ? 1u : 0u);
          }
        };
#pragma unroll
        for (int which = 0; which < (KEYS ? 2 : 1); ++which) {
          const uint32_t dst = which ? kTAcc1 : kTAcc0;
          const bool apart = !KEYS || which;
#pragma unroll
          for (int t = 0; t < split3::kSmall; ++t) product(apart ? dst + kDP : dst, which, split3::small_a(t), split3::small_b(t), t == 0);
          product(dst, which, 0, 0, apart);
        }
        if (leader) ptx::tc_commit(bar_g + 8 * (j & 1));
      }
    } else if (add) {   // half of every row warp's tiles each
      const int half = warp - kIssuer - 2;
      for (int j = 0; j < n; ++j) {
        if (j > 0) wait(bar_me, j - 1);
        if (!alive) break;
#pragma unroll 1
        for (int quarter = 0; quarter < 4; ++quarter) {
          int rows, keys;
          const int64_t at0 = mask_at(j, quarter, half, rows, keys);
          const uint32_t tile = smem_base + (uint32_t)(kMaskOff + (half * 4 + quarter) * masktile::kBytes);
          const float* src = static_cast<const float*>(p.mask) + at0;
          if (KEYS) masktile::request_columns(tile, src, p.mask_stride[2], p.mask_stride[3], rows, keys, lane);
          else masktile::request(tile, src, p.mask_stride[2], p.mask_stride[3], rows, keys, lane);
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
      const int64_t out_rows = KEYS ? p.seq_kv : p.seq_q;
      const int64_t base = KEYS ? ((int64_t)b * kv_heads + blockIdx.y) * out_rows : ((int64_t)b * p.head_count + hl0) * out_rows;
      // Eight vectors in flight, and nothing divided (one at a time, the sums of two CTAs took 8000 cycles): four of a thread's own from two CTAs, or
      // where it has fewer one from all (four whatever it has, the missing ones read again, took B2 H1 S512 D64 causal 34 -> 38 us; this 28).
      // All numbers here are powers of two: four times their distance divides the vectors, or there are fewer.
      constexpr int kVecs = KS * 4, kItems = kOwn * kVecs * (KEYS ? 2 : 1);   // (of a row; those past head_dim are not stored)
      const int hop = tp.splits * kWorkers;
      auto at = [&](int idx) { return smem_base + (uint32_t)((idx / kVecs * kPartPitch + idx % kVecs * 4) * 4); };
      auto put = [&](int idx, const float4& y) {
        const int which = idx / (kOwn * kVecs), r = idx / kVecs % kOwn, d = idx % kVecs * 4;
        if (own0 + r >= out_rows || d >= D) return;
        const float f = which ? 1.f : p.scale;
        float* out = (which ? bp.dv : (KEYS ? bp.dk : bp.dq)) + (base + own0 + r) * D + d;
        *reinterpret_cast<float4*>(out) = make_float4(y.x * f, y.y * f, y.z * f, y.w * f);
      };
      if (kItems >= 4 * hop) {
        for (int idx = rank * kWorkers + tid; idx < kItems; idx += 4 * hop) {
          float4 y[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
          for (int i = 0; i < tp.splits; ++i) {
            float4 u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) u[e] = ld_cluster_f4(at(idx + e * hop), (uint32_t)i);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e].x += u[e].x, y[e].y += u[e].y, y[e].z += u[e].z, y[e].w += u[e].w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) put(idx + e * hop, y[e]);
        }
      } else {
        for (int idx = rank * kWorkers + tid; idx < kItems; idx += hop) {
          float4 u[8], y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 8; ++i) u[i] = i < tp.splits ? ld_cluster_f4(at(idx), (uint32_t)i) : y;
#pragma unroll
          for (int i = 0; i < 8; ++i) y.x += u[i].x, y.y += u[i].y, y.z += u[i].z, y.w += u[i].w;
          put(idx, y);
        }
      }
    }
    __syncwarp();
    cluster_sync_all();   // nobody reads this CTA's shared memory any more
  }
  if (KEYS) pdl_wait();
}

// dK / dV laid over K or V, which a CTA has read by the time it stores its own rows: not beside dQ, whose CTAs still read them.
bool gradients_over_keys(const BwdParams& bp) {
  const SdpaParams& p = bp.p;
  const int64_t heads = p.num_kv_heads, count = (int64_t)p.batch * (p.head_count / p.group) * p.seq_kv * p.head_dim;
  auto over = [&](const float* grad, const void* in, const int64_t* stride) {
    const uintptr_t g = reinterpret_cast<uintptr_t>(grad), i = reinterpret_cast<uintptr_t>(in);
    const int64_t last = (p.batch - 1) * stride[0] + (heads - 1) * stride[1] + (p.seq_kv - 1) * stride[2] + p.head_dim;
    return g < i + (uintptr_t)last * sizeof(float) && i < g + (uintptr_t)count * sizeof(float);
  };
  return over(bp.dk, p.k, p.ks) || over(bp.dk, p.v, p.vs) || over(bp.dv, p.k, p.ks) || over(bp.dv, p.v, p.vs);
}

template <int KS, bool KEYS, bool PLAIN>
cudaError_t launch_one(const BwdParams& bp, cudaStream_t stream) {
  const SdpaParams& p = bp.p;
  auto kern = bwd_f32_sm100_kernel<KS, KEYS, PLAIN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(PLAIN));
  if (e != cudaSuccess) return e;
  const int64_t rows = KEYS ? p.seq_kv : p.seq_q, heads = KEYS ? p.head_count / p.group : p.head_count;
  const int64_t tiles = (rows + kOwn - 1) / kOwn, steps = ((KEYS ? p.seq_q : p.seq_kv) + kStr - 1) / kStr * (KEYS ? p.group : 1);
  BwdTcParams tp;
  tp.withhold = bp.expire;
  tp.wait_budget_ns = bp.expire ? 20000000ull : ptx::kWaitBudgetNs;   // 20 ms in the time-out test
  tp.splits = 1;
  while (tp.splits < 8 && tiles * heads * p.batch * tp.splits * 2 <= 148 && tp.splits * 2 <= steps) tp.splits *= 2;
  return launch_cluster(!KEYS || !gradients_over_keys(bp), kern, dim3((unsigned)(tiles * tp.splits), (unsigned)heads, (unsigned)p.batch), kThreads,
                        dim3((unsigned)tp.splits), smem_bytes(PLAIN), stream, bp, tp);
}

template <int KS>
cudaError_t launch_both(const BwdParams& bp, cudaStream_t stream) {
  const bool plain = bp.p.mask_kind == AIDN_MASK_NONE;
  const cudaError_t e = plain ? launch_one<KS, false, true>(bp, stream) : launch_one<KS, false, false>(bp, stream);
  if (e != cudaSuccess) return e;
  return plain ? launch_one<KS, true, true>(bp, stream) : launch_one<KS, true, false>(bp, stream);
}

}  // namespace

// Calls that backward_f32_supported accepts and this kernel takes.  Both sides measured, multiply-adds against this kernel, dQ, dK
// and dV: B1 H4 S333 D64 64 -> 44 us, B4 H8 S333 189 -> 64, B2 H8 S509 with a bias 151 -> 72, B4 H16 S1024 causal 1092 -> 332.
// Shorter sequences would often gain as well (8 x 16 heads of 100 rows 88 -> 39 us, 2 heads of 64 rows 27 -> 32), but there the
// multiply-adds' sums are as short as a block's and the truncation of four additions weighs more than their rounding: error
// against 64 bits 2.9e-7 -> 3.2e-7 at 8 x 4 heads of 64 rows, 3.3e-7 -> 3.5e-7 at 197, 3.6e-7 -> 3.5e-7 at 333, 3.9e-7 -> 3.6e-7
// at 509.  (With the roundings of t log2(e) made up for, here or in the forward kernel too, none of these is smaller: the
// log-sum-exp carries the same ones, and they cancel.)
bool backward_f32_sm100_supported(const BwdParams& bp) {
  const SdpaParams& p = bp.p;
  const int64_t longer = p.seq_q > p.seq_kv ? p.seq_q : p.seq_kv;
  return !bp.no_tcgen05 && backward_f32_sm100_fits(p) && (longer + kOwn) / kStr * 8 * (int64_t)p.group <= 0x7fffffff;
}

cudaError_t launch_backward_f32_sm100(const BwdParams& bp, cudaStream_t stream) {
  return bp.p.head_dim <= 32 ? launch_both<2>(bp, stream) : launch_both<4>(bp, stream);
}

}  // namespace aidn
