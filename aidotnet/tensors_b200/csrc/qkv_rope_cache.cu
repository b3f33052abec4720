// Decode-step front end: y = W x + b for the packed Q/K/V projection of resident tokens, interleaved RoPE on the Q and K
// heads, Q written out and the K / V rows written straight into the KV cache the decode kernel reads.  fp32 weights, and one
// token with bf16 weights; several tokens with bf16 weights run on the tensor cores (csrc/qkv_rope_sm100.cu).
//
// Replaces CudaBackend.QkvProjectionRoPECacheD64 of the reference
// (src/AiDotNet.Tensors/Engines/DirectGpu/CUDA/CudaBackend.cs:8389-8439: one fp32 token, head_dim 64, cache
// [capacity, heads, 64]; its general path is cuBLAS GEMV + BiasAdd + rope_interleaved + three device copies through
// three scratch allocations) and rope_interleaved (CUDA/Kernels/CudaAttentionKernels.cs:1023-1050).
//
// The step is a GEMV: every weight is used once per token, so it is bound by streaming W from HBM
// ((heads + 2 kv_heads) * head_dim * model * sizeof(weight) bytes).  A warp owns
// one rotation pair of output rows (2r, 2r+1) - the two rows RoPE mixes - streams both with 16-byte no-allocate loads,
// reads the tokens' activations from shared memory or through L1, and finishes the pair in registers: bias, rotation by the token's
// (cos, sin), store in the destination dtype.  Up to 8 tokens share one pass over W.
#include "common.cuh"

namespace aidn {

namespace {


template <typename WT>
struct WVec;
template <>
struct WVec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(const uint4& u, float* f) {
    f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y); f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
  }
};
template <>
struct WVec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(const uint4& u, float* f) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};

__device__ __forceinline__ void store_as(void* base, int64_t idx, float x, int dtype) {
  if (dtype == AIDN_F32) static_cast<float*>(base)[idx] = x;
  else if (dtype == AIDN_F16) static_cast<__half*>(base)[idx] = __float2half_rn(x);
  else static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(x);
}

// T tokens starting at token t_base share this pass over W.  The activations of all T tokens sit in shared memory once
// per CTA, so the CTA is made wide (WARPS) when they are large: occupancy is then bounded by warps, not by CTAs.
// XS: the activations are staged in shared memory (measured faster with fp32 weights); otherwise they are read
// through L1 (measured faster with bf16 weights, and free of any size limit).
template <typename WT, int T, int WARPS, bool XS>
__global__ void __launch_bounds__(WARPS * 32) qkv_rope_cache_kernel(const QkvRopeParams p, const int t_base) {
  constexpr int kQkvWarps = WARPS;
  constexpr int N = WVec<WT>::N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int model = p.model;
  const int D = p.head_dim;
  const int ntok = min(T, p.tokens - t_base);

  pdl_wait();      // nothing above touches memory that an earlier kernel writes
  pdl_trigger();   // the attention that follows may be set up while this kernel runs
  extern __shared__ __align__(16) float xs[];   // [T][model] when XS
  if constexpr (XS) {
    constexpr int kStageUnroll = 4;   // independent loads in flight per thread
    const int tid = threadIdx.x;
    for (int base = tid * 4; base < T * model; base += kQkvWarps * 32 * 4 * kStageUnroll) {
      float4 v[kStageUnroll];
#pragma unroll
      for (int u = 0; u < kStageUnroll; ++u) {
        const int idx = base + u * kQkvWarps * 32 * 4;
        const int t = idx / model;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (idx < T * model && t < ntok)
          v[u] = *reinterpret_cast<const float4*>(p.input + (int64_t)(t_base + t) * model + (idx - t * model));
      }
#pragma unroll
      for (int u = 0; u < kStageUnroll; ++u) {
        const int idx = base + u * kQkvWarps * 32 * 4;
        if (idx < T * model) *reinterpret_cast<float4*>(xs + idx) = v[u];
      }
    }
    __syncthreads();
  }
  const int q_rows = p.heads * D, kv_rows = p.kv_heads * D;
  const int pairs = (q_rows + 2 * kv_rows) / 2;
  const WT* W = static_cast<const WT*>(p.weights);

  for (int pair = blockIdx.x * kQkvWarps + warp; pair < pairs; pair += gridDim.x * kQkvWarps) {
    const int r0 = 2 * pair;
    const WT* w0 = W + (int64_t)r0 * model;
    const WT* w1 = w0 + model;
    // what lane t needs to finish token t, requested ahead of the weights: after them it was a chain of three loads
    // (position -> cos, sin) at the end of every pair
    const bool is_q = r0 < q_rows;
    const bool is_k = !is_q && r0 < q_rows + kv_rows;
    const int tok = t_base + lane;
    int64_t crow = -1;
    float bias0 = 0.f, bias1 = 0.f, rc = 1.f, rs = 0.f;
    if (lane < ntok) {
      const int64_t pos = p.positions ? p.positions[tok] : (int64_t)p.position + tok;
      crow = p.cache_rows ? p.cache_rows[tok] : pos;
      if (p.bias) { bias0 = p.bias[r0]; bias1 = p.bias[r0 + 1]; }
      if ((is_q || is_k) && pos >= 0 && pos < p.max_position) {
        const int i = ((is_q ? r0 : r0 - q_rows) % D) >> 1;
        rc = p.cosine[pos * (D / 2) + i];
        rs = p.sine[pos * (D / 2) + i];
      }
    }
    float a0[T], a1[T];
#pragma unroll
    for (int t = 0; t < T; ++t) a0[t] = a1[t] = 0.f;

    constexpr int kUnroll = 4;
    for (int k0 = lane * N; k0 < model; k0 += 32 * N * kUnroll) {
      uint4 u0[kUnroll], u1[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = k0 + u * 32 * N;
        const bool ok = k < model;
        u0[u] = ok ? ld_stream16(w0 + k) : make_uint4(0, 0, 0, 0);
        u1[u] = ok ? ld_stream16(w1 + k) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = k0 + u * 32 * N;
        if (k >= model) continue;
        float f0[N], f1[N];
        WVec<WT>::unpack(u0[u], f0);
        WVec<WT>::unpack(u1[u], f1);
#pragma unroll
        for (int t = 0; t < T; ++t) {
          if (!XS && t >= ntok) continue;
          const float* x = XS ? xs + t * model + k : p.input + (int64_t)(t_base + t) * model + k;
#pragma unroll
          for (int e = 0; e < N; e += 4) {
            const float4 xv = *reinterpret_cast<const float4*>(x + e);
            a0[t] = fmaf(f0[e], xv.x, a0[t]); a0[t] = fmaf(f0[e + 1], xv.y, a0[t]);
            a0[t] = fmaf(f0[e + 2], xv.z, a0[t]); a0[t] = fmaf(f0[e + 3], xv.w, a0[t]);
            a1[t] = fmaf(f1[e], xv.x, a1[t]); a1[t] = fmaf(f1[e + 1], xv.y, a1[t]);
            a1[t] = fmaf(f1[e + 2], xv.z, a1[t]); a1[t] = fmaf(f1[e + 3], xv.w, a1[t]);
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a0[t] += __shfl_xor_sync(0xffffffffu, a0[t], o);
        a1[t] += __shfl_xor_sync(0xffffffffu, a1[t], o);
      }

    // lane t finishes token t: bias, rotation, store
    if (lane < ntok) {
      float y0 = 0.f, y1 = 0.f;
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (lane == t) { y0 = a0[t]; y1 = a1[t]; }
      y0 += bias0;
      y1 += bias1;
      if (is_q || is_k) {   // interleaved RoPE: (x_even, x_odd) -> (x_even c - x_odd s, x_even s + x_odd c)
        const float e = y0 * rc - y1 * rs, o = y0 * rs + y1 * rc;
        y0 = e;
        y1 = o;
      }
      if (is_q) {
        const int64_t at = (int64_t)tok * q_rows + r0;
        store_as(p.query, at, y0, p.query_dtype);
        store_as(p.query, at + 1, y1, p.query_dtype);
      } else if (crow >= 0 && crow < p.cache_capacity) {   // a row outside the cache is not written
        const int within = is_k ? r0 - q_rows : r0 - q_rows - kv_rows;
        const int64_t at = crow * kv_rows + within;
        void* dst = is_k ? p.key_cache : p.value_cache;
        store_as(dst, at, y0, p.cache_dtype);
        store_as(dst, at + 1, y1, p.cache_dtype);
      }
    }
  }
}

__global__ void rope_interleaved_kernel(const float* __restrict__ in, const float* __restrict__ cosc,
                                        const float* __restrict__ sinc, float* __restrict__ out, int64_t rows,
                                        int head_dim, int seq_len, int start_position) {
  const int half = head_dim / 2;
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= rows * half) return;
  const int i = (int)(g % half);
  const int64_t row = g / half;
  const int64_t pos = start_position + row % seq_len;
  const float c = cosc[pos * half + i], s = sinc[pos * half + i];
  const float2 x = *reinterpret_cast<const float2*>(in + row * head_dim + 2 * i);
  *reinterpret_cast<float2*>(out + row * head_dim + 2 * i) = make_float2(x.x * c - x.y * s, x.x * s + x.y * c);
}

// CTAs for `pairs` row pairs, one pair per warp and round: at most eight CTAs per SM are resident, and when the pairs
// need more than one round every warp gets the same number of rounds (a grid-stride split that leaves a few warps with
// one pair more than the rest ends the launch with those warps alone).
inline int balanced_grid(int pairs, int warps_per_cta, int num_sms) {
  const int warp_cap = num_sms * 8 * warps_per_cta;
  const int rounds = (pairs + warp_cap - 1) / warp_cap;
  const int warps = (pairs + rounds - 1) / rounds;
  return (warps + warps_per_cta - 1) / warps_per_cta;
}

template <typename WT, int T>
cudaError_t launch_qkv_t(const QkvRopeParams& p, int t_base, int num_sms, cudaStream_t stream) {
  const int pairs = (p.heads + 2 * p.kv_heads) * p.head_dim / 2;
  const size_t xbytes = (size_t)T * p.model * sizeof(float);
  if (sizeof(WT) == 4 && xbytes <= 200 * 1024) {
    constexpr int kQkvWarps = T >= 4 ? 16 : (T == 2 ? 8 : 4);   // wide CTAs when the staged activations are large
    auto kern = qkv_rope_cache_kernel<WT, T, kQkvWarps, true>;
    if (xbytes > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)xbytes);
      if (e != cudaSuccess) return e;
    }
    const int grid = balanced_grid(pairs, kQkvWarps, num_sms);
    return launch_dependent(kern, grid, kQkvWarps * 32, xbytes, stream, p, t_base);
  } else {
    constexpr int kQkvWarps = 4;
    const int grid = balanced_grid(pairs, kQkvWarps, num_sms);
    return launch_dependent(qkv_rope_cache_kernel<WT, T, kQkvWarps, false>, grid, kQkvWarps * 32, 0, stream, p, t_base);
  }
}

template <typename WT>
cudaError_t launch_qkv_w(const QkvRopeParams& p, int num_sms, cudaStream_t stream, int* launches) {
  *launches = 0;
  for (int t_base = 0; t_base < p.tokens;) {
    const int left = p.tokens - t_base;
    cudaError_t e;
    int took = 1;
    if constexpr (sizeof(WT) == 2) {   // one token: more go to qkv_rope_sm100.cu
      e = launch_qkv_t<WT, 1>(p, t_base, num_sms, stream);
    } else {
      // the kernel instantiated for T tokens stages T rows of activations whatever it is given: T must fit
      const int tmpl = left >= 5 ? 8 : (left >= 3 ? 4 : left);
      took = left < tmpl ? left : tmpl;
      if (tmpl == 8) e = launch_qkv_t<WT, 8>(p, t_base, num_sms, stream);
      else if (tmpl == 4) e = launch_qkv_t<WT, 4>(p, t_base, num_sms, stream);
      else if (tmpl == 2) e = launch_qkv_t<WT, 2>(p, t_base, num_sms, stream);
      else e = launch_qkv_t<WT, 1>(p, t_base, num_sms, stream);
    }
    if (e != cudaSuccess) return e;
    ++*launches;
    t_base += took;
  }
  return cudaSuccess;
}

}  // namespace

// Largest model dimension served (index arithmetic is 32-bit within a weight row).
int64_t qkv_rope_max_model() { return 1 << 20; }

cudaError_t launch_qkv_rope_cache(const QkvRopeParams& p, int weight_dtype, int num_sms, cudaStream_t stream,
                                  int* launches, bool expire) {
  if (qkv_rope_sm100_supported(p, weight_dtype)) return launch_qkv_rope_sm100(p, num_sms, stream, launches, expire);
  if (weight_dtype == AIDN_F32) return launch_qkv_w<float>(p, num_sms, stream, launches);
  return launch_qkv_w<__nv_bfloat16>(p, num_sms, stream, launches);
}

cudaError_t launch_rope_interleaved(const float* in, const float* cosc, const float* sinc, float* out, int64_t rows,
                                    int head_dim, int seq_len, int start_position, cudaStream_t stream) {
  const int64_t n = rows * (head_dim / 2);
  if (n == 0) return cudaSuccess;
  rope_interleaved_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(in, cosc, sinc, out, rows, head_dim, seq_len,
                                                                          start_position);
  return cudaGetLastError();
}

}  // namespace aidn
