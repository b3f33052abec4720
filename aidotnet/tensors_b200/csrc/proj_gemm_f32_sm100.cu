// fp32 projection GEMM of the fused multi-head-attention forward on the fifth-generation tensor cores:
//   C[row, n] = sum_k A[row, k] * W[k, n], fp32 operands, results as close to the exact sum as fp32 multiply-adds give them.
// Every operand is cut into three bf16 terms (csrc/split3.cuh), and a block of 64 of K is six products.
// Against the FP32 pipe (74 TFLOP/s, and shared-memory reads per multiply-add on top) six 16-bit products leave 375 TFLOP/s.
//
// proj_split_f32_kernel cuts the weights once, into images that the GEMM copies as they are: per tile of BN columns, block of K and
// term one run of BN rows of 128 bytes (row = column of W, the 64 of K along it, swizzled).  Every row tile cutting them anew was
// the larger part of a block's 2.3 us.
//
// proj_gemm_f32_sm100_kernel, one CTA per 128 rows and BN columns:
//   warps 0-15  each owns 32 rows (its TMEM lanes) and 16 of a block's K: cp.async into a ring of its own, three terms into TMEM as
//               the A operand - from shared memory it would be read 24 times a block, on top of W's terms more than the 128 bytes
//               a cycle there are.  The same warps add up the blocks (a quarter of the columns each) and store the result
//   warps 16-17 UMMA issuers (one elected lane each) of the small and of the leading products; the first one owns TMEM.  An issuer's
//               barrier tests cost 570 cycles a block in which the tensor cores would stand still: they run under the other's products
//   warp 18     W: bulk copies into a ring of single terms
// With few row tiles (CUT_W) a launch of its own for the terms of W costs more than it saves: there warps 0-15 cut W too, into images
// whose rows are K, as the row-major weight has them (the MN-major B operand).
//
// The tensor cores truncate when they accumulate (one accumulator over K = 768 was 1.3e-6 off, always towards zero), so the
// leading products of a K block, four additions, are added to the sum in registers, which rounds to nearest; the small products
// keep one accumulator.  The leading ones of a block are read while the next block's small ones run.  A result that is not finite is formed again with multiply-adds by the thread that holds it, because
// an infinity times a term that is 0 is not a number.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "split3.cuh"

namespace aidn {
namespace {

using namespace ptx;

constexpr int kBM = 128, kBK = 64;
constexpr int kWorkerWarps = 16, kIssuer = 16, kLeadIssuer = 17, kThreads = 608;
constexpr int kXStages = 3, kXStage = 32 * 64;   // of a warp: 32 rows of 16 floats

template <int BN>
struct FCfg {
  static constexpr int kCols = BN / 4;                    // columns that a warp adds up
  static constexpr int kWOff = kWorkerWarps * kXStages * kXStage, kWSlot = BN * 128;
  // Narrow tiles multiply a term of A with two neighbouring terms of W at once: 16 products a block instead of 24, of which the issuer
  // hands out one in 35 cycles.  They keep a block's terms together; wide tiles have no room for three blocks and a ring of terms.
  static constexpr bool kPairs = BN <= 96;
  static constexpr int kFit = (227 * 1024 - 2048 - kWOff) / kWSlot, kSlots = kPairs ? (kFit < 12 ? kFit / 3 * 3 : 12) : kFit;
  static constexpr int kFullBars = (kSlots + 2) / 3 + 1;   // of a block: when its first term goes into a slot, the block as many before has been used
  static constexpr int kBarOff = kWOff + kSlots * kWSlot;
  static constexpr int kNumBars = 2 /*a_full*/ + 2 /*done*/ + 1 /*lead_free*/ + kFullBars + kSlots;
  static constexpr int kSmem = kBarOff + 8 * kNumBars + 8 + 1024;
  static constexpr int kLead = 0, kSmall = BN, kA = kSmall + (kPairs ? 2 * BN : BN);   // TMEM columns; A: two buffers of three terms of 32
  // the result on its way out, over the warp's ring: floats per row (an odd number of 16-byte chunks), then where rows and columns go
  static constexpr int kPitch = kCols + (kCols / 4 % 2 ? 8 : 4), kQuads = kCols / 4;
  static_assert(BN % 16 == 0 && kA + 192 <= 512 && kSlots >= split3::kTerms && kSmem <= 227 * 1024, "tile");
  static_assert(32 * kPitch * 4 + (32 + kQuads) * 8 <= kXStages * kXStage, "staging");
};

struct F32GemmParams {
  const float* a;
  const uint8_t* image;   // the terms of W
  const float* w[3];
  float* c[3];
  int64_t cs[3];
  int64_t rows;
  int32_t seq, k, n, head_dim;
  int32_t cols;           // of all matrices together
  int32_t col_tiles;
  int32_t row_tiles;      // where these run fastest, else 0
  int32_t splits;         // CTAs of a cluster that share a tile's K
  int32_t vec_out;
  int32_t* status;
  int32_t withhold;       // test hook: the issuer waits for operands that are never given, so that the bounded waits run out
  uint64_t wait_budget_ns;
};

__device__ __noinline__ float dot_f32(const float* a, const float* w, int k, int64_t n) {
  float s = 0.f;
  for (int i = 0; i < k; ++i) s = fmaf(a[i], w[i * n], s);
  return s;
}

// The weights of one GEMM: where they are and where their terms go.
struct SplitGroup {
  const float* w[3];
  uint8_t* image;
  int32_t k, n, cols, bn, col_tiles, k_blocks;
  int32_t col_units, units;   // of 16 columns; of 16 columns and 64 of K
};
struct SplitParams {
  SplitGroup g[2];
};

// A block of 128 threads takes 16 columns and 64 of K: a thread eight neighbours of K in one column, a warp the whole rows of four
// columns in the image (whole lines out; the lines of W that its four columns do not use are read by the other warps).
__global__ void __launch_bounds__(128) proj_split_f32_kernel(const __grid_constant__ SplitParams p) {
  pdl_wait();
  pdl_trigger();
  const bool second = (int)blockIdx.x >= p.g[0].units;
  const SplitGroup& g = second ? p.g[1] : p.g[0];
  const int unit = (int)blockIdx.x - (second ? p.g[0].units : 0);
  const int kb = unit / g.col_units, chunk = threadIdx.x & 7, k0 = kb * kBK + chunk * 8;
  const int col = (unit - kb * g.col_units) * 16 + (int)(threadIdx.x >> 3);
  const int tile = col / g.bn, row = col - tile * g.bn;
  float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < g.cols) {
    const int mat = col / g.n;
    const float* src = (mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2])) + (int64_t)k0 * g.n + (col - mat * g.n);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k0 + i < g.k) x[i] = src[(int64_t)i * g.n];
  }
  uint64_t v[4] = {pack2(x[0], x[1]), pack2(x[2], x[3]), pack2(x[4], x[5]), pack2(x[6], x[7])};
  const int64_t plane = (int64_t)g.bn * 128;
  uint8_t* dst = g.image + ((int64_t)tile * g.k_blocks + kb) * split3::kTerms * plane + split3::chunk_at(row, chunk);
#pragma unroll
  for (int t = 0; t < split3::kTerms; ++t) {
    uint4 w;
    w.x = split3::take_term(v[0]); w.y = split3::take_term(v[1]); w.z = split3::take_term(v[2]); w.w = split3::take_term(v[3]);
    *reinterpret_cast<uint4*>(dst + t * plane) = w;
  }
}

template <int BN, bool CUT_W>
__global__ void __launch_bounds__(kThreads, 1) proj_gemm_f32_sm100_kernel(const F32GemmParams g) {
  using C = FCfg<BN>;
  constexpr int kCutSlots = C::kSlots / split3::kTerms * split3::kTerms, kCutChunks = kBK * BN / 8 / (kWorkerWarps * 32);
  static_assert(!CUT_W || (BN % 64 == 0 && kCutSlots >= 2 * split3::kTerms && kCutChunks >= 1), "whole 64-column blocks and buffers of K blocks");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_a = smem_base + C::kBarOff, bar_done = bar_a + 16, bar_lead = bar_done + 16, bar_w = bar_lead + 8, bar_free = bar_w + 8 * C::kFullBars;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_gen + C::kBarOff + 8 * C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_a + 8 * i, kWorkerWarps);
      mbar_init(bar_done + 8 * i, 2);
    }
    mbar_init(bar_lead, kWorkerWarps);
    for (int i = 0; i < C::kFullBars; ++i) mbar_init(bar_w + 8 * i, 1);
    for (int i = 0; i < C::kSlots; ++i) mbar_init(bar_free + 8 * i, 2);
    fence_mbar_init();
  }
  if (warp == kIssuer) {
    tmem_alloc(smem_u32(tmem_ptr_smem), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_wait();      // A, and the terms of W, may come from the launches before
  pdl_trigger();

  // The larger of A and W is read once: column tiles run fastest (the CTAs in flight share rows of A, W stays in L2), or row tiles.
  const int rank = (int)blockIdx.x % g.splits, tile = (int)blockIdx.x / g.splits;
  const int ct = g.row_tiles ? tile / g.row_tiles : tile % g.col_tiles;
  const int64_t row0 = (int64_t)(g.row_tiles ? tile % g.row_tiles : tile / g.col_tiles) * kBM;
  const int all_blocks = (g.k + kBK - 1) / kBK, first = rank * all_blocks / g.splits, k_blocks = (rank + 1) * all_blocks / g.splits - first;
  const int quarter = warp & 3, part = warp >> 2;   // of a worker: the TMEM lanes that it may touch, 32 * (warp % 4) ..., and its columns
  float* stage = reinterpret_cast<float*>(smem_gen + warp * kXStages * kXStage);
  int64_t* row_to = reinterpret_cast<int64_t*>(stage + 32 * C::kPitch);
  float** col_to = reinterpret_cast<float**>(row_to + 32);
  const int c_first = ct * BN + part * C::kCols;
  auto column = [&](int col) {   // n is a multiple of 4: four columns belong to one matrix, and to one head where head_dim is one too
    const int mat = col / g.n, n = col - mat * g.n, h = n / g.head_dim;
    return (mat == 0 ? g.c[0] : (mat == 1 ? g.c[1] : g.c[2])) + (int64_t)h * g.cs[1] + (n - h * g.head_dim);
  };
  // Row r and columns 4 q .. of the warp's part of the tile.
  auto store = [&](int r, int q, float4 y) {
    const int64_t to = row_to[r];
    float* dst = col_to[q];
    if (to < 0 || !dst) return;
    if (g.vec_out) {
      *reinterpret_cast<float4*>(dst + to) = y;
    } else {
      dst[to] = y.x;
#pragma unroll
      for (int e = 1; e < 4; ++e) column(c_first + q * 4 + e)[to] = e == 1 ? y.y : (e == 2 ? y.z : y.w);
    }
  };
  auto exact = [&](int r, int q, float4& y) {   // what is not finite, formed again
    const int col = c_first + q * 4, mat = col / g.n;
    const int64_t row = row0 + quarter * 32 + r;
    if (row >= g.rows || col >= g.cols) return;
    const float* a = g.a + row * g.k;
    const float* w = (mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2])) + (col - mat * g.n);
    if (!(fabsf(y.x) < INFINITY)) y.x = dot_f32(a, w, g.k, g.n);
    if (!(fabsf(y.y) < INFINITY)) y.y = dot_f32(a, w + 1, g.k, g.n);
    if (!(fabsf(y.z) < INFINITY)) y.z = dot_f32(a, w + 2, g.k, g.n);
    if (!(fabsf(y.w) < INFINITY)) y.w = dot_f32(a, w + 3, g.k, g.n);
  };

  if (warp < kWorkerWarps) {
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t ring = smem_base + (uint32_t)(warp * kXStages * kXStage);
    const int64_t row_first = row0 + quarter * 32;
    auto chunk = [](int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); };   // 16 bytes: no bank conflicts by rows
    // the warp's 32 rows, 16 of K each: four lanes per row (what does not change from block to block is kept: the loop is bound by issue)
    const float* x_src = g.a + (row_first + (lane >> 2)) * g.k + first * kBK + part * 16 + (lane & 3) * 4;
    const int64_t x_step = (int64_t)8 * g.k;
    const uint32_t x_dst = ring + chunk(lane >> 2, lane & 3);   // 8 rows further down the chunk is the same
    const int64_t x_left = g.rows - row_first - (lane >> 2);
    int x_k = g.k - (first * kBK + part * 16 + (lane & 3) * 4), x_stage = 0;   // K is a multiple of 4
    auto request = [&](int kb) {
      if (kb < k_blocks) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool ok = e * 8 < x_left && x_k > 0;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                       ::"r"(x_dst + (uint32_t)(x_stage + e * 512)), "l"(ok ? x_src + e * x_step : g.a), "r"(ok ? 16u : 0u) : "memory");
        }
        x_src += kBK;
        x_k -= kBK;
        x_stage = x_stage == (kXStages - 1) * kXStage ? 0 : x_stage + kXStage;
      }
      cp_async_commit_f();
    };
    // CUT_W: chunks of eight columns, requested one or two blocks ahead (a block of 64 columns is shorter than the latency)
    constexpr int kAhead = BN == 64 ? 2 : 1;
    struct WChunks { ulonglong2 v[kCutChunks ? kCutChunks : 1][2]; } w_even, w_odd;
    const float* w_src[2];
    int w_k[2];   // rows of W that are left, or none
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int col = ct * BN + tid % (BN / 8) * 8 + q * 4, mat = col / g.n;   // n is a multiple of 4: four columns belong to one matrix
      const int k = first * kBK + tid / (BN / 8);
      w_src[q] = (mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2])) + (int64_t)k * g.n + (col - mat * g.n);
      w_k[q] = col < g.cols ? (g.k < (first + k_blocks) * kBK ? g.k : (first + k_blocks) * kBK) - k : 0;
    }
    constexpr int kCutRows = kWorkerWarps * 32 / (BN / 8);   // rows of W from one chunk of a thread to its next
    auto request_w = [&](WChunks& wn) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int e = 0; e < kCutChunks; ++e) wn.v[e][q] = split3::load4(w_src[q] + (int64_t)e * kCutRows * g.n, w_k[q] > e * kCutRows);
        w_src[q] += (int64_t)kBK * g.n;
        w_k[q] -= kBK;
      }
    };
    if (CUT_W) {
      request_w(w_even);
      if (kAhead == 2) request_w(w_odd);
    }
    float acc[C::kCols];
#pragma unroll
    for (int c = 0; c < C::kCols; ++c) acc[c] = 0.f;
    bool alive = true;
    auto add = [&](uint32_t at) {   // all loads at once: one wait
      uint32_t y[C::kCols];
#pragma unroll
      for (int c = 0; c < C::kCols; c += 8) {
        if (c + 8 <= C::kCols) tmem_ld8(at + (uint32_t)c, y + c);
        else tmem_ld4(at + (uint32_t)c, y + c);
      }
      tc_wait_ld();
#pragma unroll
      for (int c = 0; c < C::kCols; ++c) acc[c] += __uint_as_float(y[c]);
    };
    auto add_block = [&](int kb) {   // the products of block kb are complete
      alive = mbar_wait(bar_done + 8 * (kb & 1), (uint32_t)((kb >> 1) & 1), abort_flag, g.wait_budget_ns);
      alive = __all_sync(0xffffffffu, alive);
      tc_fence_after();
      if (!alive) return;
      add(t_row + (uint32_t)(C::kLead + part * C::kCols));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_lead);
    };
#pragma unroll
    for (int kb = 0; kb < kXStages - 1; ++kb) request(kb);
    auto give_block = [&](int kb, WChunks& wn) {
      cp_async_wait_f<kXStages - 2>();
      __syncwarp();   // every lane's copies are there, and the stage before has been read
      request(kb + kXStages - 1);
      uint64_t x[8];
      const uint32_t at = ring + (uint32_t)((kb % kXStages) * kXStage);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x[2 * c]), "=l"(x[2 * c + 1]) : "r"(at + chunk(lane, c)) : "memory");
      // (its buffer was last read by the products of block kb - 2, which add_block has waited for)
#pragma unroll
      for (int t = 0; t < split3::kTerms; ++t) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = split3::take_term(x[i]);
        tmem_st8(t_row + (uint32_t)(C::kA + (kb & 1) * 96 + t * 32 + part * 8), w);
      }
      if (CUT_W) {   // the slots of block kb - 2 or before: read by products that add_block has waited for
        const uint32_t w_s = smem_base + (uint32_t)(C::kWOff + kb * split3::kTerms % kCutSlots * C::kWSlot);
#pragma unroll
        for (int e = 0; e < kCutChunks; ++e) {
          const int idx = tid + e * kWorkerWarps * 32, c = idx % (BN / 8);
          split3::store_split8(w_s + (uint32_t)((c >> 3) * kBK * 128) + split3::chunk_at(idx / (BN / 8), c & 7), C::kWSlot, wn.v[e][0], wn.v[e][1]);
        }
        fence_proxy_async_smem();
        request_w(wn);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && !g.withhold) mbar_arrive(bar_a + 8 * (kb & 1));
      if (kb > 0) add_block(kb - 1);
    };
    for (int kb = 0; kb < k_blocks && alive; kb += 2) {
      give_block(kb, w_even);
      if (alive && kb + 1 < k_blocks) give_block(kb + 1, kAhead == 2 ? w_odd : w_even);
    }
    if (alive) add_block(k_blocks - 1);
    cp_async_wait_f<0>();
    if (alive) {
      add(t_row + (uint32_t)(C::kSmall + part * C::kCols));
      if (C::kPairs) add(t_row + (uint32_t)(C::kSmall + BN + part * C::kCols));
      // Through shared memory, so that lanes store neighbours; where a row and a group of four columns go is worked out once each
      // (in the loop the divisions made it 11000 cycles of 34000 at 144 columns).
      __syncwarp();
#pragma unroll
      for (int c = 0; c < C::kCols; c += 4)
        *reinterpret_cast<float4*>(stage + lane * C::kPitch + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      const int64_t row = row_first + lane, b = row / g.seq;
      row_to[lane] = row < g.rows ? b * g.cs[0] + (row - b * g.seq) * g.cs[2] : -1;
      if (lane < C::kQuads) col_to[lane] = c_first + lane * 4 < g.cols ? column(c_first + lane * 4) : nullptr;
      if (g.splits == 1) {
        float chk = 0.f;
#pragma unroll
        for (int c = 0; c < C::kCols; ++c) chk += fabsf(acc[c]);
        if (!(chk < INFINITY)) {
          for (int q = 0; q < C::kQuads; ++q) {
            float4 y = *reinterpret_cast<const float4*>(stage + lane * C::kPitch + q * 4);
            exact(lane, q, y);
            *reinterpret_cast<float4*>(stage + lane * C::kPitch + q * 4) = y;
          }
        }
        __syncwarp();
#pragma unroll 4
        for (int i = lane; i < 32 * C::kQuads; i += 32) {
          const int r = i / C::kQuads, q = i % C::kQuads;
          store(r, q, *reinterpret_cast<const float4*>(stage + r * C::kPitch + q * 4));
        }
      }
    }
  } else if (warp == kIssuer || warp == kLeadIssuer) {
    const bool leader = elect_one(), lead = warp == kLeadIssuer;
    bool alive = true;
    auto given = [&](uint32_t bar, uint32_t phase) {
      alive = alive && mbar_wait(bar, phase & 1, abort_flag, g.wait_budget_ns);
      tc_fence_after();
      return alive;
    };
    for (int kb = 0; kb < k_blocks; ++kb) {
      const uint32_t t_a = tmem_base + (uint32_t)(C::kA + (kb & 1) * 96), small = tmem_base + C::kSmall;
      if (!given(bar_a + 8 * (kb & 1), (uint32_t)(kb >> 1))) break;
      if (!CUT_W && !given(bar_w + 8 * (kb % C::kFullBars), (uint32_t)(kb / C::kFullBars))) break;
      // the block's terms of W, in the order that they are copied in: 0, 1, 2 in pairs, else 2, 1, 0
      auto slot_of = [&](int tb) { return (kb * split3::kTerms + (C::kPairs || CUT_W ? tb : 2 - tb)) % (CUT_W ? kCutSlots : C::kSlots); };
      auto product = [&](uint32_t d, int ta, int tb, int terms, bool fresh) {
        const uint64_t wd = make_smem_desc(smem_base + (uint32_t)(C::kWOff + slot_of(tb) * C::kWSlot), kBK * 128, 1024);   // (64 columns to the next block, with CUT_W)
        const uint32_t idesc = make_idesc(kBM, terms * BN, true, CUT_W);
#pragma unroll
        for (int kk = 0; kk < kBK / 16; ++kk)
          if (leader) mma_ts(d, t_a + (uint32_t)(ta * 32 + kk * 8), wd + (uint64_t)((kk * (CUT_W ? 2048 : 32)) >> 4), idesc, !fresh || kk > 0 ? 1u : 0u);
      };
      auto used = [&](int tb) {
        if (leader) tc_commit(bar_free + 8 * slot_of(tb));
      };
      if (lead) {
        if (!C::kPairs && leader) {   // (terms that this warp does not use)
          mbar_arrive(bar_free + 8 * slot_of(2));
          mbar_arrive(bar_free + 8 * slot_of(1));
        }
        if (kb > 0 && !given(bar_lead, (uint32_t)(kb - 1))) break;   // the leading products of the block before have been read
        product(tmem_base + C::kLead, 0, 0, 1, true);
      } else if constexpr (C::kPairs) {
        product(small, 0, 1, 2, kb == 0);   // with terms 1 and 2
        product(small, 1, 0, 2, false);     // with terms 0 and 1
        product(small, 2, 0, 1, false);
      } else {
        product(small, 0, 2, 1, kb == 0);
        used(2);
        product(small, 0, 1, 1, false);
        product(small, 1, 1, 1, false);
        used(1);
        product(small, 1, 0, 1, false);
        product(small, 2, 0, 1, false);
      }
      used(0);   // in pairs: the whole block
      if (leader) tc_commit(bar_done + 8 * (kb & 1));
    }
  } else if (!CUT_W && elect_one() && !g.withhold) {
    const uint8_t* src = g.image + ((int64_t)ct * all_blocks + first) * split3::kTerms * C::kWSlot;
    bool alive = true;
    for (int kb = 0, i = 0; kb < k_blocks && alive; ++kb) {
      const uint32_t full = bar_w + 8 * (kb % C::kFullBars);
#pragma unroll
      for (int t = 0; t < split3::kTerms; ++t, ++i) {
        const int slot = i % C::kSlots, tb = C::kPairs ? t : 2 - t;
        if (i >= C::kSlots && (!C::kPairs || t == 0))
          alive = alive && mbar_wait(bar_free + 8 * slot, (uint32_t)((i / C::kSlots - 1) & 1), abort_flag, g.wait_budget_ns);
        if (!alive) break;
        if (t == 0) mbar_expect_tx(full, split3::kTerms * C::kWSlot);
        bulk_load(smem_base + (uint32_t)(C::kWOff + slot * C::kWSlot), src + (int64_t)(kb * split3::kTerms + tb) * C::kWSlot, C::kWSlot, full);
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && tid == 0 && g.status) atomicOr(g.status, kStatusTimeout);
  if (warp == kIssuer) {   // (shared memory stays until this warp ends; a barrier for all in a branch of its own costs 0.4 us a launch)
    if (*abort_flag) abort_grace();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (g.splits > 1) {
    __syncwarp();
    cluster_sync_all();   // every CTA's sums are staged
    bool whole = true;    // where a CTA gave up, nothing is stored
    for (int i = 0; i < g.splits; ++i) whole = whole && __float_as_int(ld_cluster_f32(smem_u32(tmem_ptr_smem + 1), (uint32_t)i)) == 0;
    if (warp < kWorkerWarps && whole) {
      const int r_count = 32 / g.splits, r_first = rank * r_count;
#pragma unroll 2
      for (int i = lane; i < r_count * C::kQuads; i += 32) {
        const int r = i / C::kQuads + r_first, q = i % C::kQuads;
        float4 u[8], y = make_float4(0.f, 0.f, 0.f, 0.f);   // all requested before the first is used
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = j < g.splits ? ld_cluster_f4(smem_u32(stage + r * C::kPitch + q * 4), (uint32_t)j) : y;
#pragma unroll
        for (int j = 0; j < 8; ++j) y.x += u[j].x, y.y += u[j].y, y.z += u[j].z, y.w += u[j].w;
        if (!(fabsf(y.x) + fabsf(y.y) + fabsf(y.z) + fabsf(y.w) < INFINITY)) exact(r, q, y);
        store(r, q, y);
      }
    }
    __syncwarp();
    cluster_sync_all();   // nobody reads this CTA's shared memory any more
  }
}

template <int BN, bool CUT_W = false>
cudaError_t launch_t(F32GemmParams& f, int splits, cudaStream_t stream) {
  f.col_tiles = (f.cols + BN - 1) / BN;
  f.splits = splits;
  const int64_t row_tiles = (f.rows + kBM - 1) / kBM, ctas = row_tiles * f.col_tiles * splits;
  f.row_tiles = f.cols >= f.rows ? (int)row_tiles : 0;
  if (ctas > 0x7fffffff) return cudaErrorInvalidValue;
  auto kern = proj_gemm_f32_sm100_kernel<BN, CUT_W>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FCfg<BN>::kSmem);
  if (e != cudaSuccess) return e;
  return launch_dependent_cluster(kern, dim3((unsigned)ctas), kThreads, dim3((unsigned)splits), FCfg<BN>::kSmem, stream, f);
}

}  // namespace

// Columns of a tile, CTAs that share its K, and whether they cut W themselves: what has the shortest time by waves of CTAs, in cycles.
// A block of K takes 1190 at 32 and 2330 at 160 columns, with W cut in place 1950 and 3300 at 64 and 128; the rest 7600 at 48 and 10000
// at 144 columns, the merge of a cluster 7000 to 12000, a launch for the terms of W 5000 and an element 1 / 220 (they are written and
// read again).  Clusters only where all of a launch's CTAs are resident at once.  Layers, in us, before -> with these rules:
//   rows x width  16 x 512 35 -> 25, 100 x 1024 57 -> 46, 256 x 2048 123 -> 93, 384 x 3072 256 -> 215, 1024 x 1024 127 -> 101,
//   2048 x 3072 1294 -> 1124; 1576 x 512 (143 tiles of 144 and of 48 columns) 83 -> 57
// (The instantiations that cut W have 96 registers a thread and keep 24 and 40 bytes of stack at 64 and 128 columns.)
// (`launched`: the launch for the terms is there for another GEMM of the layer already, and costs this one nothing.)
ProjPlanF32 proj_gemm_f32_sm100_plan(int64_t rows, int64_t k, int64_t n, int mats, int num_sms, bool images, bool launched) {
  const int64_t cols = n * mats, launch = launched ? 0 : 5000;
  ProjPlanF32 best = {0, 0, false};
  int64_t best_cost = 0;
  const int64_t blocks = (k + kBK - 1) / kBK;
  auto consider = [&](int bn, bool cut, int64_t block, int64_t once) {
    for (int s = 1; s <= 8 && (s == 1 || s * 2 <= blocks); s *= 2) {
      const int64_t ctas = (rows + kBM - 1) / kBM * ((cols + bn - 1) / bn) * s, waves = (ctas + num_sms - 1) / num_sms;
      if (s > 1 && ctas * 100 > num_sms * 89) break;
      const int64_t cost = once + waves * (6500 + 24 * bn + (s > 1 ? 5500 + 15 * bn + 500 * s : 0) + (blocks + s - 1) / s * block);
      if (!best.width || cost < best_cost) best = {bn, s, cut}, best_cost = cost;
    }
  };
  consider(64, true, 1950, 0);
  consider(128, true, 3300, 0);
  if (images)
    for (int bn : {32, 48, 64, 96, 128, 144, 160}) consider(bn, false, bn <= 96 ? 900 + 9 * bn : 1050 + 8 * bn, launch + cols * k / 220);
  return best;
}

// Whole layers, the attention unchanged, multiply-adds against these kernels' first form: 64 rows x 3072 and 1024 x 1024
// 211 -> 138 and 336 -> 181 us (the latter 125 with the fp32 attention on the tensor cores, 101 with the kernels above).  Error of a whole layer against
// 64 bits 7.2e-7 -> 4.0e-7 at K = 768, 5.4e-7 -> 3.8e-7 at 512; below K = 256 the truncation of four additions weighs more than the
// rounding of K (2.5e-7 -> 3.4e-7 at 64) and the times are equal: there the multiply-adds stay.
bool proj_gemm_f32_sm100_fits(int64_t k, int64_t n) { return k >= 256 && k % 4 == 0 && n % 4 == 0 && n * 3 + 160 <= 0x7fffffff; }

bool proj_gemm_f32_sm100_supported(const ProjGemm& g) {
  bool ok = proj_gemm_f32_sm100_fits(g.k, g.n) && reinterpret_cast<uintptr_t>(g.a) % 16 == 0;
  for (int i = 0; i < g.num_mats; ++i) ok = ok && reinterpret_cast<uintptr_t>(g.w[i]) % 16 == 0;
  return ok;
}

int64_t proj_gemm_f32_sm100_bytes(const ProjPlanF32& plan, int64_t k, int64_t n, int mats) {
  if (plan.cut_w) return 0;
  return (n * mats + plan.width - 1) / plan.width * plan.width * ((k + kBK - 1) / kBK) * 128 * split3::kTerms;
}

cudaError_t launch_proj_split_f32(const ProjGemm* gemms, int count, cudaStream_t stream) {
  SplitParams p = {};
  int64_t units = 0;
  for (int i = 0; i < count; ++i) {
    const ProjGemm& g = gemms[i];
    SplitGroup& s = p.g[i];
    for (int j = 0; j < 3; ++j) s.w[j] = static_cast<const float*>(g.w[j < g.num_mats ? j : 0]);
    s.image = static_cast<uint8_t*>(g.image);
    s.k = (int)g.k;
    s.n = (int)g.n;
    s.cols = (int)(g.n * g.num_mats);
    s.bn = g.f32_plan.width;
    s.col_tiles = (s.cols + s.bn - 1) / s.bn;
    s.k_blocks = (int)((g.k + kBK - 1) / kBK);
    s.col_units = s.col_tiles * (s.bn / 16);
    const int64_t u = (int64_t)s.col_units * s.k_blocks;
    units += u;
    if (units > 0x7fffffff) return cudaErrorInvalidValue;
    s.units = (int)u;
  }
  return launch_dependent(proj_split_f32_kernel, dim3((unsigned)units), 128, 0, stream, p);
}

cudaError_t launch_proj_gemm_f32_sm100(const ProjGemm& p, cudaStream_t stream, int32_t* status, bool expire) {
  F32GemmParams f;
  f.a = static_cast<const float*>(p.a);
  f.image = static_cast<const uint8_t*>(p.image);
  bool vec = p.head_dim % 4 == 0;
  for (int i = 0; i < 3; ++i) {
    const int j = i < p.num_mats ? i : 0;
    f.w[i] = static_cast<const float*>(p.w[j]);
    f.c[i] = static_cast<float*>(p.c[j]);
    f.cs[i] = p.c_stride[i];
    vec = vec && p.c_stride[i] % 4 == 0 && reinterpret_cast<uintptr_t>(f.c[i]) % 16 == 0;
  }
  f.rows = p.batch * p.seq;
  f.seq = (int)p.seq;
  f.k = (int)p.k;
  f.n = (int)p.n;
  f.cols = (int)(p.n * p.num_mats);
  f.head_dim = p.head_dim;
  f.vec_out = vec ? 1 : 0;
  f.status = status;
  f.withhold = expire ? 1 : 0;
  f.wait_budget_ns = expire ? 20000000ull : kWaitBudgetNs;   // 20 ms in the time-out test
  const ProjPlanF32& plan = p.f32_plan;
  if (plan.cut_w) return plan.width == 64 ? launch_t<64, true>(f, plan.splits, stream) : launch_t<128, true>(f, plan.splits, stream);
  switch (plan.width) {
    case 32: return launch_t<32>(f, plan.splits, stream);
    case 48: return launch_t<48>(f, plan.splits, stream);
    case 64: return launch_t<64>(f, plan.splits, stream);
    case 96: return launch_t<96>(f, plan.splits, stream);
    case 128: return launch_t<128>(f, plan.splits, stream);
    case 144: return launch_t<144>(f, plan.splits, stream);
    default: return launch_t<160>(f, plan.splits, stream);
  }
}

}  // namespace aidn
