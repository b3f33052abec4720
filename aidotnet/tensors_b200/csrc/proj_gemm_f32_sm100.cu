// fp32 projection GEMM of the fused multi-head-attention forward on the fifth-generation tensor cores:
//   C[row, n] = sum_k A[row, k] * W[k, n], fp32 operands, results as close to the exact sum as fp32 multiply-adds give them.
// Every operand is cut into three bf16 terms (csrc/split3.cuh) on its way into shared memory, and a K block is six products.
// Against the FP32 pipe (74 TFLOP/s, and shared-memory reads per multiply-add on top) six 16-bit products leave 375 TFLOP/s.
//
//   warps 0-7   per 64-wide K block: 128 x 64 of A (K-major image) and 64 x BN of W (MN-major B operand: its rows are K, so the
//               row-major weight needs no transpose) from global memory to registers - requested one block ahead - and as
//               three swizzled images each into one of two buffers; two threads per row add up the blocks; epilogue
//   warp 8      UMMA issuer (one elected lane) and owner of TMEM
//
// The tensor cores truncate when they accumulate (one accumulator over K = 768 was 1.3e-6 off, always towards zero), so the
// leading products of a K block, four additions, are added to the sum in registers, which rounds to nearest; the small products
// keep one accumulator.  A result that is not finite is formed again with multiply-adds by the thread that stores it, because
// an infinity times a term that is 0 is not a number.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "split3.cuh"

namespace aidn {
namespace {

using namespace ptx;

constexpr int kBM = 128, kBK = 64, kBufs = 2;
constexpr int kWorkers = 256, kThreads = 384;   // two warpgroups of workers, one with the issuer

template <int BN>
struct FCfg {
  static constexpr int kAPlane = kBM * 128, kWBlock = kBK * 128, kWPlane = (BN / 64) * kWBlock;
  static constexpr int kBuf = split3::kTerms * (kAPlane + kWPlane);
  static constexpr int kBarOff = kBufs * kBuf;
  static constexpr int kSmem = kBarOff + 8 * 2 * kBufs + 8 + 1024;
  static constexpr int kTmemCols = BN == 64 ? 256 : 512;   // two block accumulators and that of the small products
};

struct F32GemmParams {
  const float* a;
  const float* w[3];
  float* c[3];
  int64_t cs[3];
  int64_t rows;
  int32_t seq, k, n, head_dim;
  int32_t col_tiles;      // of one matrix
  int32_t all_col_tiles;  // of all of them
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

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) proj_gemm_f32_sm100_kernel(const F32GemmParams g) {
  using C = FCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_full = smem_base + C::kBarOff, bar_done = bar_full + 8 * kBufs;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_gen + C::kBarOff + 8 * 2 * kBufs);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(bar_full + 8 * i, kWorkers / 32);
      mbar_init(bar_done + 8 * i, 1);
    }
    fence_mbar_init();
  }
  if (warp == kWorkers / 32) {
    tmem_alloc(smem_u32(tmem_ptr_smem), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  // column tiles run fastest: the CTAs in flight share rows of A, and all of W stays in L2
  const int ct = (int)blockIdx.x % g.all_col_tiles;
  const int mat = ct / g.col_tiles;
  const int64_t row0 = (int64_t)((int)blockIdx.x / g.all_col_tiles) * kBM;
  const int col0 = (ct - mat * g.col_tiles) * BN;
  const int k_blocks = (g.k + kBK - 1) / kBK;
  const float* w = mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2]);   // no indexed copy of the parameters

  if (warp < kWorkers / 32) {
    setmaxnreg_inc<208>();
    constexpr int kAChunks = kBM * 8 / kWorkers, kWChunks = kBK * (BN / 8) / kWorkers, kChunks = kAChunks + kWChunks;
    ulonglong2 next[kChunks][2];
    auto request = [&](int kb) {
#pragma unroll
      for (int e = 0; e < kAChunks; ++e) {
        const int idx = tid + e * kWorkers, r = idx >> 3, k = kb * kBK + (idx & 7) * 8;
        const float* src = g.a + (row0 + r) * g.k + k;
        const bool ok = row0 + r < g.rows;
        next[e][0] = split3::load4(src, ok && k < g.k);
        next[e][1] = split3::load4(src + 4, ok && k + 4 < g.k);
      }
#pragma unroll
      for (int e = 0; e < kWChunks; ++e) {
        const int idx = tid + e * kWorkers, r = idx / (BN / 8), n = col0 + (idx % (BN / 8)) * 8, k = kb * kBK + r;
        const float* src = w + (int64_t)k * g.n + n;
        const bool ok = k < g.k;
        next[kAChunks + e][0] = split3::load4(src, ok && n < g.n);
        next[kAChunks + e][1] = split3::load4(src + 4, ok && n + 4 < g.n);
      }
    };
    const int quarter = warp & 3;   // the TMEM lanes a warp may read: 32 * (warp % 4) ...
    const int c_begin = (warp >> 2) * (BN / 2);
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_begin;
    float acc[BN / 2];
#pragma unroll
    for (int c = 0; c < BN / 2; ++c) acc[c] = 0.f;
    bool alive = true;
    auto add = [&](uint32_t at) {
#pragma unroll
      for (int c0 = 0; c0 < BN / 2; c0 += 32) {
        uint32_t y[32];
        tmem_ld32(at + (uint32_t)c0, y);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c0 + c] += __uint_as_float(y[c]);
      }
    };
    auto add_block = [&](int kb) {   // the products of K block kb are complete (and its buffer is free)
      alive = mbar_wait(bar_done + 8 * (kb % kBufs), (uint32_t)((kb / kBufs) & 1), abort_flag, g.wait_budget_ns);
      alive = __all_sync(0xffffffffu, alive);
      tc_fence_after();
      if (alive) add(t_row + (uint32_t)((kb & 1) * BN));
      tc_fence_before();
    };
    request(0);
    for (int kb = 0; kb < k_blocks; ++kb) {
      const uint32_t a_s = smem_base + (kb % kBufs) * C::kBuf, w_s = a_s + split3::kTerms * C::kAPlane;
#pragma unroll
      for (int e = 0; e < kAChunks; ++e) {
        const int idx = tid + e * kWorkers;
        split3::store_split8(a_s + split3::chunk_at(idx >> 3, idx & 7), C::kAPlane, next[e][0], next[e][1]);
      }
#pragma unroll
      for (int e = 0; e < kWChunks; ++e) {
        const int idx = tid + e * kWorkers, r = idx / (BN / 8), cn = idx % (BN / 8);
        split3::store_split8(w_s + (uint32_t)((cn >> 3) * C::kWBlock) + split3::chunk_at(r, cn & 7), C::kWPlane, next[kAChunks + e][0], next[kAChunks + e][1]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && !g.withhold) mbar_arrive(bar_full + 8 * (kb % kBufs));
      if (kb + 1 < k_blocks) request(kb + 1);
      if (kb > 0) add_block(kb - 1);   // block kb + 1 goes into its buffer
      if (!alive) break;
    }
    if (alive) add_block(k_blocks - 1);
    if (alive) {
      add(t_row + 2 * BN);
      const int64_t row = row0 + quarter * 32 + lane;
      const int64_t b = row / g.seq, s = row - b * g.seq;
      float* c = mat == 0 ? g.c[0] : (mat == 1 ? g.c[1] : g.c[2]);
      float* dst = c + b * g.cs[0] + s * g.cs[2];
      if (row < g.rows) {
#pragma unroll
        for (int c4 = 0; c4 < BN / 2; c4 += 4) {
          const int n = col0 + c_begin + c4;
          if (n >= g.n) continue;   // n is a multiple of 4: the group of four columns is inside or outside as a whole
          float y[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            y[e] = acc[c4 + e];
            if (!(fabsf(y[e]) < INFINITY)) y[e] = dot_f32(g.a + row * g.k, w + n + e, g.k, g.n);
          }
          if (g.vec_out) {   // head_dim % 4 == 0: the four columns belong to one head
            const int h = n / g.head_dim;
            *reinterpret_cast<float4*>(dst + (int64_t)h * g.cs[1] + (n - h * g.head_dim)) = make_float4(y[0], y[1], y[2], y[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int h = (n + e) / g.head_dim;
              dst[(int64_t)h * g.cs[1] + (n + e - h * g.head_dim)] = y[e];
            }
          }
        }
      }
    }
  } else {
    setmaxnreg_dec<88>();
    if (warp == kWorkers / 32) {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc(kBM, BN, true, true);
      for (int kb = 0; kb < k_blocks; ++kb) {
        const int buf = kb % kBufs;
        if (!mbar_wait(bar_full + 8 * buf, (uint32_t)((kb / kBufs) & 1), abort_flag, g.wait_budget_ns)) break;
        tc_fence_after();
        const uint32_t a_s = smem_base + buf * C::kBuf, w_s = a_s + split3::kTerms * C::kAPlane;
        // (a descriptor is its base plus a constant: one warp issues 24 products a block)
        const uint64_t ad = make_smem_desc(a_s, 16, 1024), wd = make_smem_desc(w_s, C::kWBlock, 1024);
        auto product = [&](uint32_t d, int ta, int tb, bool fresh) {
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk) {
            const uint64_t x = ad + (uint64_t)((ta * C::kAPlane + kk * 32) >> 4), y = wd + (uint64_t)((tb * C::kWPlane + kk * 2048) >> 4);
            if (leader) mma_ss(d, x, y, idesc, !fresh || kk > 0 ? 1u : 0u);
          }
        };
        product(tmem_base + (uint32_t)((kb & 1) * BN), 0, 0, true);
#pragma unroll
        for (int i = 0; i < split3::kSmall; ++i) product(tmem_base + 2 * BN, split3::small_a(i), split3::small_b(i), kb == 0 && i == 0);
        if (leader) tc_commit(bar_done + 8 * buf);
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && tid == 0 && g.status) atomicOr(g.status, kStatusTimeout);
  if (warp == kWorkers / 32) {   // (shared memory stays until this warp ends; a barrier for all in a branch of its own costs 0.4 us a launch)
    if (*abort_flag) abort_grace();
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int BN>
cudaError_t launch_t(F32GemmParams& f, int mats, cudaStream_t stream) {
  f.col_tiles = (f.n + BN - 1) / BN;
  f.all_col_tiles = f.col_tiles * mats;
  const int64_t tiles = (f.rows + kBM - 1) / kBM * f.all_col_tiles;
  if (tiles > 0x7fffffff) return cudaErrorInvalidValue;
  auto kern = proj_gemm_f32_sm100_kernel<BN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FCfg<BN>::kSmem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)tiles, kThreads, FCfg<BN>::kSmem, stream>>>(f);
  return cudaGetLastError();
}

}  // namespace

// Whole layers, the attention unchanged: 64 rows x 3072 and 1024 x 1024 211 -> 138 and 336 -> 181 us.  Error of a whole layer against
// 64 bits 7.2e-7 -> 4.0e-7 at K = 768, 5.4e-7 -> 3.8e-7 at 512; below K = 256 the truncation of four additions weighs more than the
// rounding of K (2.5e-7 -> 3.4e-7 at 64) and the times are equal: there the multiply-adds stay.
bool proj_gemm_f32_sm100_supported(const ProjGemm& g) {
  bool ok = g.k >= 256 && g.k % 4 == 0 && g.n % 4 == 0 && reinterpret_cast<uintptr_t>(g.a) % 16 == 0;
  for (int i = 0; i < g.num_mats; ++i) ok = ok && reinterpret_cast<uintptr_t>(g.w[i]) % 16 == 0;
  return ok;
}

cudaError_t launch_proj_gemm_f32_sm100(const ProjGemm& p, cudaStream_t stream, int num_sms, int32_t* status, bool expire) {
  F32GemmParams f;
  f.a = static_cast<const float*>(p.a);
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
  f.head_dim = p.head_dim;
  f.vec_out = vec ? 1 : 0;
  f.status = status;
  f.withhold = expire ? 1 : 0;
  f.wait_budget_ns = expire ? 20000000ull : kWaitBudgetNs;   // 20 ms in the time-out test
  auto waves = [&](int bn) {
    const int64_t tiles = (f.rows + kBM - 1) / kBM * ((f.n + bn - 1) / bn) * p.num_mats;
    return (tiles + num_sms - 1) / num_sms;
  };
  if (waves(128) * 4 <= waves(64) * 3) return launch_t<128>(f, p.num_mats, stream);
  return launch_t<64>(f, p.num_mats, stream);
}

}  // namespace aidn
