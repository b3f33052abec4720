// Projection GEMM of the fused multi-head-attention forward for the shapes and types the tcgen05 kernel does not take
// (fp32 operands, head sizes other than 64 / 128, model widths that are not a multiple of 128):
//   C[b, s, n] = sum_k A[b, s, k] * W[k, n]
// fp32 FFMA arithmetic, any sizes, the same head-major scatter in the epilogue (column n lands in head n / head_dim).
// The first kernel takes anything: a 64 x 64 tile per CTA of 256 threads, 16-wide K slices through shared memory, a 4 x 4
// micro-tile per thread.  The second one takes fp32 operands whose rows allow 16-byte access.
//
// This is the exact route of the engine's MultiHeadAttentionForward: with fp32 tensors it meets the 1e-4 bound of the
// reference's own tests of the fused call (tests/AiDotNet.Tensors.Tests/Engines/MultiHeadAttentionForwardTests.cs:123),
// including their head sizes of 2 to 8 (src/AiDotNet.Tensors/Engines/CpuEngine.MultiHeadAttention.cs:155-338).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ffma2.cuh"

namespace aidn {
namespace {

constexpr int kTile = 64;
constexpr int kSlice = 16;

template <typename T>
__device__ __forceinline__ float to_f32(T v) {
  return static_cast<float>(v);
}

template <typename T>
__device__ __forceinline__ void store_as(void* base, int64_t off, float v, bool f32) {
  if (f32) static_cast<float*>(base)[off] = v;
  else static_cast<T*>(base)[off] = static_cast<T>(v);
}
template <>
__device__ __forceinline__ void store_as<float>(void* base, int64_t off, float v, bool) {
  static_cast<float*>(base)[off] = v;
}

struct GenericGemmParams {
  const void* a;
  const void* w[3];
  void* c[3];
  int64_t cs[3];
  int64_t rows;   // batch * seq
  int32_t seq, k, n, head_dim;
  int32_t out_f32;
};

template <typename T>
__global__ void __launch_bounds__(256) proj_gemm_generic_kernel(const GenericGemmParams g) {
  __shared__ float a_s[kSlice][kTile + 4];   // a_s[kk][row]: transposed on the way in
  __shared__ float w_s[kSlice][kTile + 4];
  const int mat = blockIdx.z;
  const T* a = static_cast<const T*>(g.a);
  const T* w = static_cast<const T*>(mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2]));   // no indexed copy of the parameters
  const int64_t row0 = (int64_t)blockIdx.y * kTile;
  const int col0 = blockIdx.x * kTile;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < g.k; k0 += kSlice) {
    // A slice: 64 rows x 16 k; thread t reads row t / 4, k offsets 4 * (t % 4) ..
    {
      const int r = threadIdx.x >> 2, kq = (threadIdx.x & 3) * 4;
      const int64_t row = row0 + r;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int kk = k0 + kq + i;
        a_s[kq + i][r] = (row < g.rows && kk < g.k) ? to_f32(a[row * g.k + kk]) : 0.f;
      }
    }
    // W slice: 16 k x 64 columns; thread t reads k row t / 16, columns 4 * (t % 16) ..
    {
      const int kr = threadIdx.x >> 4, cq = (threadIdx.x & 15) * 4;
      const int kk = k0 + kr;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = col0 + cq + i;
        w_s[kr][cq + i] = (kk < g.k && col < g.n) ? to_f32(w[(int64_t)kk * g.n + col]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kSlice; ++kk) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[i] = a_s[kk][ty * 4 + i];
        wv[i] = w_s[kk][tx * 4 + i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
  void* c = mat == 0 ? g.c[0] : (mat == 1 ? g.c[1] : g.c[2]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t row = row0 + ty * 4 + i;
    if (row >= g.rows) continue;
    const int64_t b = row / g.seq, s = row - b * g.seq;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + tx * 4 + j;
      if (col >= g.n) continue;
      const int h = col / g.head_dim;
      const int64_t off = b * g.cs[0] + (int64_t)h * g.cs[1] + s * g.cs[2] + (col - h * g.head_dim);
      store_as<T>(c, off, acc[i][j], g.out_f32 != 0);
    }
  }
}

// ---- fp32 operands with 16-byte rows: register-tiled packed multiply-adds -------------------------------------------------
// Shared memory hands 128 bytes per cycle to the registers whether lanes read the same words or not, so an a x b block per
// lane is bound by it unless (a + b) / (a b) <= 1 / 4: a warp owns 32 rows x 64 columns, 8 x 8 per lane (4 x 8 lanes).
// A is staged as it lies ([row][k]), W as it lies ([k][column]); column pairs are the packed dimension and A's values are
// duplicated in registers.  (W transposed on the way in, with k as the packed dimension and 8 x 4 blocks, needs no
// duplicates but took 127 us for three 1576 x 512 x 512 products against 82 here and 130 for the kernel above.)
// Three cp.async stages of 32 k.  KG > 1: the warps of one output tile split each stage's k and their sums are added
// through shared memory in warp order, so results do not depend on timing.
template <int WM, int KG>
struct GCfg {
  static constexpr int kThreads = WM * KG * 32;
  static constexpr int kBM = WM * 32, kBN = 64, kBK = 32, kStages = 3;
  static constexpr int kAPitch = kBK + 4, kWPitch = kBN;
  static constexpr int kAFloats = kBM * kAPitch, kStageFloats = kAFloats + kBK * kWPitch;
  static constexpr size_t kSmem = sizeof(float) * kStages * kStageFloats;
};

template <int WM, int KG>
__global__ void __launch_bounds__(WM* KG * 32, 2) proj_gemm_f32_kernel(const GenericGemmParams g, const int vec_out) {
  using C = GCfg<WM, KG>;
  extern __shared__ __align__(16) float gsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ty = lane >> 3, tx = lane & 7;
  const int wm = warp % WM, kg = warp / WM;
  const int mat = blockIdx.z;
  const float* a = static_cast<const float*>(g.a);
  const float* w = static_cast<const float*>(mat == 0 ? g.w[0] : (mat == 1 ? g.w[1] : g.w[2]));   // no indexed copy of the parameters
  const int64_t row0 = (int64_t)blockIdx.y * C::kBM;
  const int64_t col0 = (int64_t)blockIdx.x * C::kBN;

  auto fetch = [&](int s) {
    float* as = gsm + (s % C::kStages) * C::kStageFloats;
    float* ws = as + C::kAFloats;
    const int64_t k0 = (int64_t)s * C::kBK;
#pragma unroll
    for (int e = 0; e < C::kBM * 8 / C::kThreads; ++e) {
      const int idx = tid + e * C::kThreads;
      const int r = idx >> 3, kk = (idx & 7) * 4;
      const bool ok = row0 + r < g.rows && k0 + kk < g.k;
      cp_async16_f(as + r * C::kAPitch + kk, a + (ok ? (row0 + r) * g.k + k0 + kk : 0), ok);
    }
#pragma unroll
    for (int e = 0; e < C::kBK * C::kBN / 4 / C::kThreads; ++e) {
      const int idx = tid + e * C::kThreads;
      const int kk = idx / (C::kBN / 4), c = (idx - kk * (C::kBN / 4)) * 4;
      const bool ok = k0 + kk < g.k && col0 + c < g.n;
      cp_async16_f(ws + kk * C::kWPitch + c, w + (ok ? (k0 + kk) * g.n + col0 + c : 0), ok);
    }
  };
  uint64_t acc[8][4];   // rows ty + 4 i; columns tx * 4 + {0, 1}, {2, 3}, 32 + {0, 1}, 32 + {2, 3}
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0;

  const int steps = (g.k + C::kBK - 1) / C::kBK;
#pragma unroll
  for (int s = 0; s < C::kStages - 1; ++s) {
    if (s < steps) fetch(s);
    cp_async_commit_f();
  }
  for (int s = 0; s < steps; ++s) {
    cp_async_wait_f<C::kStages - 2>();
    __syncthreads();   // stage s has landed, and every warp has left the stage that is filled next
    if (s + C::kStages - 1 < steps) fetch(s + C::kStages - 1);
    cp_async_commit_f();
    const float* as = gsm + (s % C::kStages) * C::kStageFloats + (wm * 32 + ty) * C::kAPitch;
    const float* ws = gsm + (s % C::kStages) * C::kStageFloats + C::kAFloats + tx * 4;
#pragma unroll
    for (int kq = 0; kq < C::kBK / KG; kq += 4) {
      const int k = kg * (C::kBK / KG) + kq;
      float4 av[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const float4*>(as + 4 * i * C::kAPitch + k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const Pair2 w0 = lds_pairs(ws + (k + e) * C::kWPitch), w1 = lds_pairs(ws + (k + e) * C::kWPitch + 32);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float x = e == 0 ? av[i].x : (e == 1 ? av[i].y : (e == 2 ? av[i].z : av[i].w));
          const uint64_t x2 = pack2(x, x);
          acc[i][0] = fma2(x2, w0.a, acc[i][0]);
          acc[i][1] = fma2(x2, w0.b, acc[i][1]);
          acc[i][2] = fma2(x2, w1.a, acc[i][2]);
          acc[i][3] = fma2(x2, w1.b, acc[i][3]);
        }
      }
    }
  }

  if constexpr (KG > 1) {   // lane-major images of the other groups' sums: conflict-free both ways
    cp_async_wait_f<0>();
    __syncthreads();
    ulonglong2* all = reinterpret_cast<ulonglong2*>(gsm);
    if (kg > 0) {
      ulonglong2* mine = all + ((kg - 1) * WM + wm) * 16 * 32 + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        mine[(2 * i) * 32] = make_ulonglong2(acc[i][0], acc[i][1]);
        mine[(2 * i + 1) * 32] = make_ulonglong2(acc[i][2], acc[i][3]);
      }
    }
    __syncthreads();
    if (kg > 0) return;
#pragma unroll
    for (int o = 1; o < KG; ++o) {
      const ulonglong2* theirs = all + ((o - 1) * WM + wm) * 16 * 32 + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const ulonglong2 lo = theirs[(2 * i) * 32], hi = theirs[(2 * i + 1) * 32];
        acc[i][0] = add2(acc[i][0], lo.x);
        acc[i][1] = add2(acc[i][1], lo.y);
        acc[i][2] = add2(acc[i][2], hi.x);
        acc[i][3] = add2(acc[i][3], hi.y);
      }
    }
  }

  // Divisions in 32 bits (rows fit: at most 65535 tiles), and those of the columns ahead of the rows: 64-bit ones at every
  // stored element made the attention layer of B2 S33 H6 D6 take 41 us instead of 29.
  float* c = static_cast<float*>(mat == 0 ? g.c[0] : (mat == 1 ? g.c[1] : g.c[2]));
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int col = (int)col0 + half * 32 + tx * 4;
    if (col >= g.n) continue;   // n is a multiple of 4: the group of four columns is inside or outside as a whole
    int64_t at[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e > 0 && vec_out) break;   // head_dim % 4 == 0: the four columns belong to one head
      const int h = (col + e) / g.head_dim;
      at[e] = (int64_t)h * g.cs[1] + (col + e - h * g.head_dim);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (int)row0 + wm * 32 + ty + 4 * i;
      if (row >= g.rows) continue;
      const int b = row / g.seq, s = row - b * g.seq;
      const float2 lo = unpack2(acc[i][2 * half]), hi = unpack2(acc[i][2 * half + 1]);
      float* dst = c + b * g.cs[0] + s * g.cs[2];
      if (vec_out) {
        *reinterpret_cast<float4*>(dst + at[0]) = make_float4(lo.x, lo.y, hi.x, hi.y);
      } else {
        dst[at[0]] = lo.x;
        dst[at[1]] = lo.y;
        dst[at[2]] = hi.x;
        dst[at[3]] = hi.y;
      }
    }
  }
}

template <int WM, int KG>
cudaError_t launch_f32_cfg(const GenericGemmParams& g, int mats, int vec_out, cudaStream_t stream) {
  using C = GCfg<WM, KG>;
  static_assert((KG - 1) * WM * 16 * 32 * 16 <= (int)C::kSmem, "the merge reuses the stages");
  static_assert(2 * (C::kSmem + 1024) <= 228 * 1024, "two CTAs per SM");
  auto kern = proj_gemm_f32_kernel<WM, KG>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((g.n + C::kBN - 1) / C::kBN), (unsigned)((g.rows + C::kBM - 1) / C::kBM), (unsigned)mats);
  kern<<<grid, C::kThreads, C::kSmem, stream>>>(g, vec_out);
  return cudaGetLastError();
}

cudaError_t launch_f32(const GenericGemmParams& g, int mats, cudaStream_t stream) {
  bool vec = g.head_dim % 4 == 0;
  for (int i = 0; i < 3; ++i) vec = vec && g.cs[i] % 4 == 0 && reinterpret_cast<uintptr_t>(g.c[i]) % 16 == 0;
  // Tile height: an SM's time is the rows of the tiles that the busiest SM gets, each tile with a fixed cost on top
  // (prologue, merge, the W tile).  64-row tiles split k over four warps, 128-row tiles over two, so that an SM holds
  // sixteen warps either way (128 registers, 20 and 68 bytes spilled).  1576 rows x 512: 167 us per attention layer with 64 rows,
  // 183 with 128 or with 32.  Of 14 layers of 64 to 2560 rows and widths of 256 to 1536 the pick was at most 4 % behind the other
  // height (B4 S197 H12 D64 191 us, 184 with 64 rows), which is up to 1.6 times slower where it is not picked.
  auto cost = [&](int bm) {
    const int64_t ctas = (g.rows + bm - 1) / bm * ((g.n + 63) / 64) * mats;
    return (ctas + 147) / 148 * (bm + 16);
  };
  if (cost(128) < cost(64)) return launch_f32_cfg<4, 2>(g, mats, vec, stream);
  return launch_f32_cfg<2, 4>(g, mats, vec, stream);
}

template <typename T>
cudaError_t launch_t(const ProjGemm& p, cudaStream_t stream) {
  GenericGemmParams g;
  g.a = p.a;
  for (int i = 0; i < 3; ++i) {
    g.w[i] = p.w[i < p.num_mats ? i : 0];
    g.c[i] = p.c[i < p.num_mats ? i : 0];
    g.cs[i] = p.c_stride[i];
  }
  g.rows = p.batch * p.seq;
  g.seq = (int)p.seq;
  g.k = (int)p.k;
  g.n = (int)p.n;
  g.head_dim = p.head_dim;
  g.out_f32 = p.out_f32 ? 1 : 0;
  if constexpr (sizeof(T) == 4) {
    bool vec = g.k % 4 == 0 && g.n % 4 == 0 && reinterpret_cast<uintptr_t>(g.a) % 16 == 0;
    for (int i = 0; i < p.num_mats; ++i) vec = vec && reinterpret_cast<uintptr_t>(g.w[i]) % 16 == 0;
    if (vec) return launch_f32(g, p.num_mats, stream);
  }
  const int64_t row_tiles = (g.rows + kTile - 1) / kTile;
  if (row_tiles > 65535) return cudaErrorInvalidValue;
  dim3 grid((unsigned)((p.n + kTile - 1) / kTile), (unsigned)row_tiles, (unsigned)p.num_mats);
  proj_gemm_generic_kernel<T><<<grid, 256, 0, stream>>>(g);
  return cudaGetLastError();
}

}  // namespace

bool proj_gemm_generic_supported(const ProjGemm& g, const char** why) {
  if (g.num_mats < 1 || g.num_mats > 3) { *why = "projection GEMM takes 1 to 3 weight matrices"; return false; }
  if (g.batch <= 0 || g.seq <= 0 || g.k <= 0 || g.n <= 0 || g.head_dim <= 0 || g.n % g.head_dim != 0) {
    *why = "projection GEMM: dimensions must be positive and heads * head_dim == n";
    return false;
  }
  if (g.seq > 0x7fffffffll || g.k > 0x7fffffffll || g.n > 0x7fffffffll || (g.batch * g.seq + kTile - 1) / kTile > 65535) {
    *why = "projection GEMM: more than 65535 * 64 rows or a dimension above 2^31";
    return false;
  }
  return true;
}

cudaError_t launch_proj_gemm_generic(const ProjGemm& g, int dtype, cudaStream_t stream) {
  if (dtype == AIDN_F32) return launch_t<float>(g, stream);
  if (dtype == AIDN_BF16) return launch_t<__nv_bfloat16>(g, stream);
  return launch_t<__half>(g, stream);
}

}  // namespace aidn
