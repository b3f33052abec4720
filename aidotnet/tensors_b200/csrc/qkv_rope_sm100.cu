// Decode-step projection of several tokens with bf16 weights on the fifth-generation tensor cores: the packed Q/K/V
// product of csrc/qkv_rope_cache.cu (same contract: bias, interleaved RoPE on Q and K, rows written into the cache).
//
// The work is one pass over W: `rows * model * 2` bytes for at most 64 tokens, so the kernel is a weight stream.  W is the
// M operand of tcgen05.mma (128 output rows per tile, K-major as it lies) and arrives by TMA, so that what is in flight
// does not depend on registers or on how many warps an SM holds; the tokens are N.  The fp32 activations travel through
// the same ring, and eight warps turn each 64-wide slice into three bf16 terms (x = hi + mid + lo to 2^-27), which become
// 3 * T columns of one B operand: D[:, t] + D[:, T + t] + D[:, 2 T + t] is the fp32 product.
//
//   warp 0      TMA producer: per 64-wide K block one W box (128 x 64, 128-byte swizzle) and one X box (T x 64 fp32)
//   warp 1      UMMA issuer and owner of TMEM
//   warps 2-9   split of the activations; then TMEM -> shared memory (four of them), and the finish (bias, rotation, stores)
//
// The tensor cores truncate when they accumulate.  The products with hi therefore go to six accumulators in turn (chains of
// model / splits / 96 additions), those with mid and lo, 2^-8 of the whole, to one.
//
// There are fewer row tiles than SMs, so K is cut over the CTAs of a cluster; every CTA leaves its partial tile in its
// own shared memory and the cluster's CTAs finish one share of the tile each, reading the others' partials through
// distributed shared memory in rank order: no scratch memory, no atomics, the same bits every time.
//
// Hq32 / Hkv8 D128 (50 MB of weights, 7.8 us at the copy bandwidth), against one mma.sync pass per eight tokens:
// 16 tokens 35.5 -> 15.5 us, 2 tokens 19.0 -> 14.2, 64 tokens 133 -> 33.4; Hq64 / Hkv8 D128 (168 MB) with 16 tokens 255 -> 33.
// Error of fp32 outputs against 64 bits 2.5e-6 -> 1.3e-7 (3.2e-7 with 64 tokens, Hq64 2.6e-7 to 4.2e-7).  What is left is the latency of set-up, first
// bytes and finish (a launch over 3 MB of weights takes 5 us).
#include <cuda.h>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "split3.cuh"
#include "tensor_map.hpp"

namespace aidn {
namespace {

using namespace ptx;

constexpr int kTileRows = 128;
constexpr int kBK = 64;
constexpr int kSplitters = 256, kThreads = 64 + kSplitters;
constexpr int kWBytes = kTileRows * kBK * 2;
constexpr int kBStages = 2;
constexpr int kMaxStages = 4;
constexpr int kMaxTokens = 64;
constexpr int kAccs = 6;

struct QkvTcMaps {
  CUtensorMap w;   // (model, rows), box 64 x 128, bf16, 128-byte swizzle
  CUtensorMap x;   // (model, tokens), box 64 x T, fp32
};

struct QkvTcParams {
  int32_t t_base, ntok, tpad;   // tokens of this pass, padded to a multiple of 16
  int32_t stages;
  int32_t tmem_cols;
  int32_t k_blocks, splits;
  int32_t withhold;             // test hook: the producer withholds its loads, so that the bounded waits run out
  uint64_t wait_budget_ns;
};

// Set when a bounded wait gave up (this entry point has no handle whose status word could say so); aidn_qkv_rope_poll reads it.
__device__ int32_t g_qkv_status;

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void store_as(void* base, int64_t idx, float x, int dtype) {
  if (dtype == AIDN_F32) static_cast<float*>(base)[idx] = x;
  else if (dtype == AIDN_F16) static_cast<__half*>(base)[idx] = __float2half_rn(x);
  else static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(x);
}

// What is left of x after its leading term (exact); nothing of an infinity or a NaN, which the leading term carries alone.
__device__ __forceinline__ float rest(float x, float lead) {
  const float r = x - lead;
  return fabsf(r) < INFINITY ? r : 0.f;
}

// The wait for the last products gave up: what was already issued gets a bounded chance to complete before tensor and shared memory are
// released, and the thread's row of the partial tile becomes NaN, for the cluster's other CTAs may finish their shares: what they
// store is then not a number, rather than a sum over whatever lay here.  (Looking at this CTA's flag for every sum and storing nothing
// costs a projection of 2 to 32 tokens 0.3 to 0.9 us of 14 to 18.)
__device__ __forceinline__ void give_up(float* part_row, int ntok) {
  abort_grace();
  for (int t = 0; t < ntok; ++t) part_row[t * kTileRows] = NAN;
}

__global__ void __launch_bounds__(kThreads) qkv_rope_cache_sm100_kernel(const __grid_constant__ QkvTcMaps maps, const QkvRopeParams p,
                                                                        const QkvTcParams tp) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const int tpad = tp.tpad, stages = tp.stages;
  const uint32_t b_bytes = (uint32_t)(split3::kTerms * tpad * 128), x_bytes = (uint32_t)(tpad * kBK * 4);
  const uint32_t b_off = (uint32_t)(stages * kWBytes), x_off = b_off + kBStages * b_bytes;
  const uint32_t bar_off = x_off + stages * x_bytes;
  const uint32_t bar_full = smem_base + bar_off;            // [stages]: W and X have landed
  const uint32_t bar_empty = bar_full + 8 * kMaxStages;     // [stages]: the products that read them have completed
  const uint32_t bar_bfull = bar_empty + 8 * kMaxStages;    // [kBStages]: the three terms are written
  const uint32_t bar_bempty = bar_bfull + 8 * kBStages;     // [kBStages]
  const uint32_t bar_acc = bar_bempty + 8 * kBStages;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_gen + (bar_acc - smem_base) + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  float* part = reinterpret_cast<float*>(smem_gen);   // [tpad][128], over the ring once every product has completed

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)blockIdx.x % tp.splits, tile = (int)blockIdx.x / tp.splits;   // a cluster is `splits` CTAs of one tile
  const int kb0 = (int)((int64_t)rank * tp.k_blocks / tp.splits), kb1 = (int)((int64_t)(rank + 1) * tp.k_blocks / tp.splits);
  const int nkb = kb1 - kb0;

  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < kBStages; ++s) {
      mbar_init(bar_bfull + 8 * s, kSplitters / 32);
      mbar_init(bar_bempty + 8 * s, 1);
    }
    mbar_init(bar_acc, 1);
    fence_mbar_init();
    prefetch_tensormap(&maps.w);
    prefetch_tensormap(&maps.x);
  }
  const uint32_t tmem_cols = (uint32_t)tp.tmem_cols;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_ptr_smem), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_wait();      // nothing above touches memory that an earlier kernel writes
  pdl_trigger();   // the attention that follows may be set up while this kernel runs

  const int D = p.head_dim, half = D / 2;
  const int q_rows = p.heads * D, kv_rows = p.kv_heads * D, rows = q_rows + 2 * kv_rows;

  if (warp == 0) {
    // ============================================ TMA producer ============================================
    const bool leader = elect_one();
    for (int i = 0; i < nkb; ++i) {
      const int s = i % stages;
      if (tp.withhold) break;
      if (!mbar_wait(bar_empty + 8 * s, (uint32_t)((i / stages) & 1) ^ 1u, abort_flag, tp.wait_budget_ns)) break;
      if (leader) {
        const uint32_t bar = bar_full + 8 * s;
        mbar_expect_tx(bar, kWBytes + x_bytes);
        tma_load_4d(smem_base + s * kWBytes, &maps.w, bar, (kb0 + i) * kBK, tile * kTileRows, 0, 0);
        tma_load_4d(smem_base + x_off + s * x_bytes, &maps.x, bar, (kb0 + i) * kBK, tp.t_base, 0, 0);
      }
    }
  } else if (warp == 1) {
    // ============================================ UMMA issuer =============================================
    const bool leader = elect_one();
    const uint32_t idesc_hi = make_idesc(kTileRows, tpad, true, false), idesc_low = make_idesc(kTileRows, 2 * tpad, true, false);
    bool alive = true;
    for (int i = 0; i < nkb; ++i) {
      const int s = i % stages, bs = i % kBStages;
      if (!mbar_wait(bar_full + 8 * s, (uint32_t)((i / stages) & 1), abort_flag, tp.wait_budget_ns) ||
          !mbar_wait(bar_bfull + 8 * bs, (uint32_t)((i / kBStages) & 1), abort_flag, tp.wait_budget_ns)) {
        alive = false;
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)((2 + i % kAccs) * tpad);   // behind the columns of mid and lo
      const uint64_t wd = make_smem_desc(smem_base + s * kWBytes, 16, 1024), hd = make_smem_desc(smem_base + b_off + bs * b_bytes, 16, 1024);
      const uint64_t ld = hd + (uint64_t)(tpad * 128 >> 4);
#pragma unroll
      for (int kk = 0; kk < kBK / 16; ++kk) {
        if (leader) mma_ss(d, wd + 2 * kk, hd + 2 * kk, idesc_hi, (i >= kAccs || kk > 0) ? 1u : 0u);
        if (leader) mma_ss(tmem_base, wd + 2 * kk, ld + 2 * kk, idesc_low, (i > 0 || kk > 0) ? 1u : 0u);
      }
      if (leader) {
        tc_commit(bar_empty + 8 * s);
        tc_commit(bar_bempty + 8 * bs);
      }
    }
    if (alive && leader) tc_commit(bar_acc);
  } else {
    // ========================================== split of X ================================================
    const int etid = tid - 64;
    bool alive = true;
    for (int i = 0; i < nkb && alive; ++i) {
      const int s = i % stages, bs = i % kBStages;
      alive = mbar_wait(bar_full + 8 * s, (uint32_t)((i / stages) & 1), abort_flag, tp.wait_budget_ns) &&
              mbar_wait(bar_bempty + 8 * bs, (uint32_t)((i / kBStages) & 1) ^ 1u, abort_flag, tp.wait_budget_ns);
      alive = __all_sync(0xffffffffu, alive);
      if (!alive) break;
      const uint8_t* xs = smem_gen + x_off + s * x_bytes;
      const uint32_t b_s = smem_base + b_off + bs * b_bytes;
      for (int item = etid; item < tpad * 8; item += kSplitters) {   // eight activations: one 16-byte chunk of each term
        const int t = item >> 3, c = item & 7;
        const float4 a = *reinterpret_cast<const float4*>(xs + t * 256 + c * 32);
        const float4 b = *reinterpret_cast<const float4*>(xs + t * 256 + c * 32 + 16);
        float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int term = 0; term < split3::kTerms; ++term) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            w[e] = pack2<true>(f[2 * e], f[2 * e + 1]);
            f[2 * e] = rest(f[2 * e], __uint_as_float(w[e] << 16));
            f[2 * e + 1] = rest(f[2 * e + 1], __uint_as_float(w[e] & 0xffff0000u));
          }
          // row term * tpad + t of the operand (tpad is a multiple of 8: the swizzle is that of row t)
          st_shared_v4(b_s + (uint32_t)(term * tpad * 128) + split3::chunk_at(t, c), w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_bfull + 8 * bs);
    }
    // ================================ accumulators -> this CTA's partial tile ================================
    if (alive) alive = mbar_wait(bar_acc, 0u, abort_flag, tp.wait_budget_ns);
    alive = __all_sync(0xffffffffu, alive);
    if (alive && warp < 6) {
      tc_fence_after();
      const int quarter = warp & 3;   // the TMEM lanes a warp may read: 32 * (warp % 4) ...
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
      const int row = quarter * 32 + lane;
      const int accs = kAccs < nkb ? kAccs : nkb;
      for (int t0 = 0; t0 < tp.ntok; t0 += 8) {
        float y[8], low[8], mid[8];
        tmem_ld8(t_row + (uint32_t)t0, mid);
        tmem_ld8(t_row + (uint32_t)(tpad + t0), low);
        tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          y[e] = 0.f;
          low[e] += mid[e];
        }
        for (int a = 0; a < accs; ++a) {
          float hi[8];
          tmem_ld8(t_row + (uint32_t)((2 + a) * tpad + t0), hi);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] += hi[e];
        }
        // an infinite weight times a term that is 0 is not a number: the leading terms alone say what the sum is then
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (fabsf(y[e]) < INFINITY) y[e] += low[e];
#pragma unroll
        for (int e = 0; e < 8; ++e) part[(t0 + e) * kTileRows + row] = y[e];   // t0 + 8 <= tpad
      }
      tc_fence_before();
    }
    if (!alive && warp < 6) give_up(part + (warp & 3) * 32 + lane, tp.ntok);
  }

  // ------------------------------------------ finish: one share of the tile ------------------------------------------
  // Item: (token, rotation pair); pairs run fastest, so that a warp stores neighbouring elements.  What the first items need
  // besides the sums is requested before the cluster meets.
  constexpr int kPairs = kTileRows / 2, kAhead = 2;
  const int items = kPairs * tp.ntok, stride = tp.splits * kThreads;
  struct Extra { int64_t crow; float b0, b1, c, s; };
  auto extra_of = [&](int item) {
    Extra x = {-1, 0.f, 0.f, 1.f, 0.f};
    const int r0 = tile * kTileRows + 2 * (item & (kPairs - 1));
    if (item >= items || r0 >= rows) return x;
    const int tok = tp.t_base + item / kPairs;
    const int64_t pos = p.positions ? p.positions[tok] : (int64_t)p.position + tok;
    x.crow = p.cache_rows ? p.cache_rows[tok] : pos;
    if (p.bias) { x.b0 = p.bias[r0]; x.b1 = p.bias[r0 + 1]; }
    if (r0 < q_rows + kv_rows && pos >= 0 && pos < p.max_position) {
      const int i = ((r0 < q_rows ? r0 : r0 - q_rows) % D) >> 1;
      x.c = p.cosine[pos * half + i];
      x.s = p.sine[pos * half + i];
    }
    return x;
  };
  const int first = rank * kThreads + tid;
  Extra ahead[kAhead];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) ahead[u] = extra_of(first + u * stride);

  // TMEM goes back before the CTAs of the cluster wait for one another: one of them may still be waiting for its columns behind
  // a CTA of another launch, which may be waiting for these.
  __syncwarp();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
  __syncwarp();
  cluster_sync_all();   // every CTA's partial tile is written
  if (!*abort_flag) {
    int u = 0;
    for (int item = first; item < items; item += stride, ++u) {
      const int pr = item & (kPairs - 1), t = item / kPairs;
      const int r0 = tile * kTileRows + 2 * pr;
      if (r0 >= rows) continue;
      const Extra x = u == 0 ? ahead[0] : (u == 1 ? ahead[1] : extra_of(item));
      float y0 = 0.f, y1 = 0.f;
#pragma unroll 4
      for (int r = 0; r < tp.splits; ++r) {
        const float2 v = ld_cluster_f2(smem_base + (uint32_t)((t * kTileRows + 2 * pr) * 4), (uint32_t)r);
        y0 += v.x;
        y1 += v.y;
      }
      y0 += x.b0;
      y1 += x.b1;
      const bool is_q = r0 < q_rows;
      const bool is_k = !is_q && r0 < q_rows + kv_rows;
      if (is_q || is_k) {   // interleaved RoPE: (x_even, x_odd) -> (x_even c - x_odd s, x_even s + x_odd c)
        const float e = y0 * x.c - y1 * x.s, o = y0 * x.s + y1 * x.c;
        y0 = e;
        y1 = o;
      }
      if (is_q) {
        const int64_t at = (int64_t)(tp.t_base + t) * q_rows + r0;
        store_as(p.query, at, y0, p.query_dtype);
        store_as(p.query, at + 1, y1, p.query_dtype);
      } else if (x.crow >= 0 && x.crow < p.cache_capacity) {   // a row outside the cache is not written
        const int64_t at = x.crow * kv_rows + (is_k ? r0 - q_rows : r0 - q_rows - kv_rows);
        void* dst = is_k ? p.key_cache : p.value_cache;
        store_as(dst, at, y0, p.cache_dtype);
        store_as(dst, at + 1, y1, p.cache_dtype);
      }
    }
  }
  __syncwarp();
  cluster_sync_all();   // nobody reads this CTA's shared memory any more
  if (*abort_flag) {
    if (tid == 0) atomicOr(&g_qkv_status, kStatusTimeout);
    __syncthreads();
  }
}

struct QkvTcPlan {
  int tpad, stages, tmem_cols, splits;
  size_t smem;
};

QkvTcPlan plan_of(int tokens, int tiles, int k_blocks, int num_sms) {
  QkvTcPlan pl;
  pl.tpad = (tokens + 15) / 16 * 16;
  pl.stages = pl.tpad <= 32 ? 3 : 4;
  pl.tmem_cols = 128;
  while (pl.tmem_cols < (2 + kAccs) * pl.tpad) pl.tmem_cols *= 2;
  const int resident = pl.tpad <= 16 ? 3 : (pl.tpad <= 32 ? 2 : 1);   // CTAs per SM, by shared memory
  // As many CTAs as are resident at once hide one another's latencies (measured with four splitting warps, whose times are not those
  // above: 16 tokens, 48 tiles of 64 K blocks 18.0 us with 3 splits, 15.8 with 4, 13.3 with 8); a second wave costs as much as the first (80 tiles of 128: 5 splits = 400 CTAs 30.6 us,
  // 6 = 480 CTAs 41), and clusters of three or more do not pack the SMs to the last one (48 tiles with 64 tokens, one CTA per
  // SM: 2 splits 37 us, 3 splits = 144 CTAs 53).
  pl.splits = 1;
  int64_t best = INT64_MAX;
  for (int ks = 1; ks <= 8 && ks <= k_blocks; ++ks) {
    const int64_t room = ks > 2 ? (int64_t)num_sms * resident * 92 / 100 : (int64_t)num_sms * resident;
    const int64_t waves = ((int64_t)tiles * ks + room - 1) / room;
    const int64_t cost = waves * ((k_blocks + ks - 1) / ks + 6);
    if (cost < best) { best = cost; pl.splits = ks; }
  }
  pl.smem = (size_t)pl.stages * (kWBytes + pl.tpad * kBK * 4) + (size_t)kBStages * split3::kTerms * pl.tpad * 128 + 8 * (2 * kMaxStages + 2 * kBStages + 1) + 16 + 1024;
  return pl;
}

}  // namespace

// One token stays on the GEMV of qkv_rope_cache.cu: 11.7 us over 50 MB of weights, where this kernel takes 13.9 with two.
bool qkv_rope_sm100_supported(const QkvRopeParams& p, int weight_dtype) {
  return weight_dtype == AIDN_BF16 && p.tokens >= 2;
}

int32_t* qkv_rope_sm100_status() {
  void* addr = nullptr;
  if (cudaGetSymbolAddress(&addr, g_qkv_status) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<int32_t*>(addr);
}

cudaError_t launch_qkv_rope_sm100(const QkvRopeParams& p, int num_sms, cudaStream_t stream, int* launches, bool expire) {
  cudaError_t e = tmap::resolve_encode();
  if (e != cudaSuccess) return e;
  const int64_t rows = (int64_t)(p.heads + 2 * p.kv_heads) * p.head_dim;
  const int tiles = (int)((rows + kTileRows - 1) / kTileRows), k_blocks = (p.model + kBK - 1) / kBK;
  *launches = 0;
  for (int t_base = 0; t_base < p.tokens; t_base += kMaxTokens) {
    QkvTcParams tp;
    tp.t_base = t_base;
    tp.ntok = p.tokens - t_base < kMaxTokens ? p.tokens - t_base : kMaxTokens;
    const QkvTcPlan pl = plan_of(tp.ntok, tiles, k_blocks, num_sms);
    tp.tpad = pl.tpad;
    tp.stages = pl.stages;
    tp.tmem_cols = pl.tmem_cols;
    tp.k_blocks = k_blocks;
    tp.splits = pl.splits;
    tp.withhold = expire ? 1 : 0;
    tp.wait_budget_ns = expire ? 20000000ull : kWaitBudgetNs;   // 20 ms in the time-out test
    QkvTcMaps maps;
    const int64_t ws[3] = {rows * p.model, rows * p.model, p.model};
    const int64_t xs[3] = {(int64_t)p.tokens * p.model, (int64_t)p.tokens * p.model, p.model};
    if (!tmap::encode_bhsd(&maps.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, CU_TENSOR_MAP_SWIZZLE_128B, p.weights, p.model, rows, 1, 1, ws, kBK, kTileRows) ||
        !tmap::encode_bhsd(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, CU_TENSOR_MAP_SWIZZLE_NONE, p.input, p.model, p.tokens, 1, 1, xs, kBK, pl.tpad))
      return cudaErrorInvalidValue;
    e = cudaFuncSetAttribute(qkv_rope_cache_sm100_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
    if (e != cudaSuccess) return e;
    e = launch_dependent_cluster(qkv_rope_cache_sm100_kernel, dim3((unsigned)(tiles * pl.splits)), kThreads, dim3((unsigned)pl.splits), pl.smem, stream, maps, p, tp);
    if (e != cudaSuccess) return e;
    ++*launches;
  }
  return cudaSuccess;
}

}  // namespace aidn
