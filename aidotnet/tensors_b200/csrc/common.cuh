// Shared definitions of the attention kernels: the flattened launch parameters, dtype helpers and the
// mask evaluation that every kernel uses so that mask semantics are defined once.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../../include/aidn_sdpa.h"

namespace aidn {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// Device status word values (bit flags) written by kernels that give up a bounded wait.
constexpr int kStatusTimeout = 1;
constexpr int kStatusBadBlock = 2;  // a block-table entry outside [0, num_blocks) was met (the key is skipped)

struct SdpaParams {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  float* lse;
  float* weights;   // [B, Hq, Sq, Sk] fp32 probabilities, or null (generic kernel only)
  void* peer_out[8];   // other devices' `out` tensors, mapped here (tcgen05 prefill only)
  int32_t peer_count;
  const void* mask;
  const int32_t* kv_len;
  int64_t mask_stride[4];
  int64_t qs[3], ks[3], vs[3], os[3];  // element strides for (B, H, S)
  int64_t seq_q, seq_kv;
  int64_t causal_offset;
  int32_t batch;
  int32_t num_q_heads, num_kv_heads, group;  // group = Hq / Hkv
  int32_t head_begin, head_count;            // q-head shard computed by this launch
  int32_t head_dim;
  int32_t mask_kind;
  int32_t causal;
  int32_t out_f32;  // 1: output is fp32, 0: output has the input dtype
  float scale;
  float softcap;
  int32_t* status;  // device word, or null
  // Paged K/V (null block_table = contiguous): key t of batch entry b lives in row
  // block_table[b * bt_stride + t / block_size] * block_size + t % block_size of the pool, and that row index
  // takes the place of the key index in the K/V address (ks[2] / vs[2] = token stride, ks[0] / vs[0] unused).
  const int32_t* block_table;
  int64_t bt_stride;
  int32_t block_size;
  int32_t block_shift;  // log2(block_size) when it is a power of two, else -1
  int32_t num_blocks;   // > 0: entries are range-checked against it
  int32_t no_tcgen05;   // 1: stay on the FP32 units (desc.path == AIDN_PATH_GENERIC); fp32 attention only
  int32_t expire;       // test hook of the fp32 tcgen05 kernel: nothing is loaded and every bounded wait gives up after 20 ms
};

template <typename T>
__device__ __forceinline__ float to_float(T x);
template <>
__device__ __forceinline__ float to_float<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_float<__half>(__half x) { return __half2float(x); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T>
__device__ __forceinline__ T from_float(float x);
template <>
__device__ __forceinline__ float from_float<float>(float x) { return x; }
template <>
__device__ __forceinline__ __half from_float<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Stores one output element either as fp32 or in the input dtype.
template <typename T>
__device__ __forceinline__ void store_out(void* base, int64_t idx, float x, int out_f32) {
  if (out_f32) static_cast<float*>(base)[idx] = x;
  else static_cast<T*>(base)[idx] = from_float<T>(x);
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The largest of three (a NaN counts only where all are), one instruction.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// exp used by the softmax: exact expf for fp32 inputs (1e-5 relative contract), ex2.approx otherwise.
template <typename T>
__device__ __forceinline__ float softmax_exp(float x) {
  if constexpr (sizeof(T) == 4) return expf(x);
  else return ex2_approx(x * kLog2e);
}

// Applies softcap, additive bias and every mask to a scaled logit.
// Order: scale (done by the caller) -> softcap -> bias -> keep masks / causal / padding,
// as CpuEngine.cs:27807-27816 (SDPA) and :29218-29239 (FlashAttention) of the reference.
// Returns -inf for a masked position.
__device__ __forceinline__ float finish_logit(const SdpaParams& p, float s, int b, int h, int64_t qi, int64_t kj,
                                              int64_t kv_limit) {
  if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
  if (kj >= kv_limit) return -INFINITY;
  if (p.causal && kj > qi + p.causal_offset) return -INFINITY;
  if (p.mask_kind != AIDN_MASK_NONE) {
    const int64_t idx = b * p.mask_stride[0] + h * p.mask_stride[1] + qi * p.mask_stride[2] + kj * p.mask_stride[3];
    if (p.mask_kind == AIDN_MASK_KEEP_U8) {
      if (static_cast<const uint8_t*>(p.mask)[idx] == 0) return -INFINITY;
    } else if (p.mask_kind == AIDN_MASK_KEEP_F32) {
      if (static_cast<const float*>(p.mask)[idx] == 0.0f) return -INFINITY;
    } else {
      s += static_cast<const float*>(p.mask)[idx];
    }
  }
  return s;
}

// Number of keys a batch entry can see before causal masking: min(seq_kv, kv_len[b]).
// (With a block table the host has already capped seq_kv at the keys the table's rows can address.)
__device__ __forceinline__ int64_t kv_limit_of(const SdpaParams& p, int b) {
  int64_t lim = p.seq_kv;
  if (p.kv_len) {
    int64_t l = p.kv_len[b];
    if (l < 0) l = 0;
    if (l < lim) lim = l;
  }
  return lim;
}

// Paged K/V addressing in two halves, so that a kernel can issue the block-table read a step ahead and touch its
// result only when the row is needed (anything computed from the entry right after the read would make the warp
// wait for it there).
//   kv_block_read: the raw entry of key's block (volatile: issued where the caller placed it).
//   kv_row_from:   pool row of the key from that entry; -1, and `bad` set, for an entry outside the pool.  No
//                  branch on the entry; the caller reports `bad` once, at its end, with report_bad_block().
__device__ __forceinline__ int32_t kv_block_read(const SdpaParams& p, int b, int64_t key) {
  const uint32_t k32 = (uint32_t)key;
  const uint32_t blk = p.block_shift >= 0 ? (k32 >> p.block_shift) : (k32 / (uint32_t)p.block_size);
  int32_t phys;
  asm volatile("ld.global.s32 %0, [%1];" : "=r"(phys) : "l"(p.block_table + (int64_t)b * p.bt_stride + blk));
  return phys;
}

__device__ __forceinline__ int64_t kv_row_from(const SdpaParams& p, int64_t key, int32_t phys, bool& bad) {
  const uint32_t k32 = (uint32_t)key;
  const uint32_t blk = p.block_shift >= 0 ? (k32 >> p.block_shift) : (k32 / (uint32_t)p.block_size);
  const bool out = phys < 0 || (p.num_blocks > 0 && phys >= p.num_blocks);
  bad = bad || out;
  const int64_t row = (int64_t)phys * p.block_size + (k32 - blk * (uint32_t)p.block_size);
  return out ? -1 : row;
}

// Pool row of key `key` of batch entry b (the key itself without a block table): read and use in one place.
__device__ __forceinline__ int64_t kv_row_of(const SdpaParams& p, int b, int64_t key, bool& bad) {
  if (!p.block_table) return key;
  return kv_row_from(p, key, kv_block_read(p, b, key), bad);
}

__device__ __forceinline__ void report_bad_block(const SdpaParams& p, bool bad) {
  if (bad && p.status) atomicOr(p.status, kStatusBadBlock);
}

// Programmatic dependent launch: a kernel started with launch_dependent may begin while its predecessor on the stream is
// still running - its launch latency and prologue then cost nothing - and must call pdl_wait before it touches memory that
// any earlier kernel reads or writes.  What an earlier kernel may write is not read-only for the whole of its life, so it
// must not go through the non-coherent path (ld.global.nc, __ldg, const __restrict__) either.  pdl_trigger in the
// predecessor says from when on; a kernel that never calls it is waited for as a whole, which is what the stream order
// alone would do.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The one exception: what launches before its predecessor have written, a kernel may read ahead of its own wait if every CTA of
// the predecessor triggers behind the predecessor's wait.  Those launches have then ended, and their writes are in the L2 cache; the wait
// made them visible to the predecessor alone, though, so an older copy might still be in an L1.  Either the kernel reads past that (ld_l2),
// or the predecessor triggers by pdl_hand_over and every thread of the kernel begins with pdl_take_over, whose fences carry on what the wait has
// given.  What the predecessor writes, and writes that it might read, stay behind the wait, and the kernel must not end without one: the next launch
// relies on both.
__device__ __forceinline__ void pdl_hand_over() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  pdl_trigger();
}
__device__ __forceinline__ void pdl_take_over() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");   // TMA loads too
}
__device__ __forceinline__ int32_t ld_l2(const int32_t* ptr) {
  int32_t r;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(r) : "l"(ptr) : "memory");
  return r;
}

// 16 bytes that are read once.
__device__ __forceinline__ uint4 ld_stream16(const void* ptr) {
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(ptr));
  return r;
}

// Launched as thread-block clusters of `cluster` CTAs (1 x 1 x 1: none), behind the whole of the launch before or as a dependent of it.
template <typename... P, typename... A>
inline cudaError_t launch_cluster(bool dependent, void (*kern)(P...), dim3 grid, unsigned threads, dim3 cluster, size_t smem,
                                  cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = dependent ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster.x;
  attr[1].val.clusterDim.y = cluster.y;
  attr[1].val.clusterDim.z = cluster.z;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // reported here: the next launch must not find it as its own
  return e;
}

template <typename... P, typename... A>
inline cudaError_t launch_dependent_cluster(void (*kern)(P...), dim3 grid, unsigned threads, dim3 cluster, size_t smem,
                                            cudaStream_t stream, A... args) {
  return launch_cluster(true, kern, grid, threads, cluster, smem, stream, args...);
}

template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, A... args) {
  return launch_dependent_cluster(kern, grid, threads, dim3(1), smem, stream, args...);
}

// Thread-block clusters: the barrier of all their threads (release / acquire), and reads of another CTA's shared memory.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// Host-side launchers (one per kernel family); each returns the CUDA error of its launch.
cudaError_t launch_generic(const SdpaParams& p, int dtype, cudaStream_t stream);
// The register-tiled fp32 kernel (csrc/sdpa_f32.cu); launch_generic hands it what it takes.
bool f32_supported(const SdpaParams& p, int dtype);
cudaError_t launch_f32(const SdpaParams& p, int dtype, cudaStream_t stream);
// fp32 tensors as three bf16 terms on tcgen05 (csrc/sdpa_f32_sm100.cu), of the calls that f32_supported accepts.
bool f32_sm100_supported(const SdpaParams& p, int dtype);
cudaError_t launch_f32_sm100(const SdpaParams& p, cudaStream_t stream);
// How the keys of a decode are cut: `nchunks` parts, of `chunk` keys each where cluster is 1; else `nchunks` clusters of
// `cluster` CTAs per (sequence, KV head), which share the sequence's keys evenly.  nchunks > 1 takes the workspace.
struct DecodePlan {
  int chunk, nchunks, cluster;
  int stream_ctas;   // > 0: that many CTAs, whose warps share all keys evenly (decode_stream_bytes of workspace)
};
// The workspace of such a launch and its CTAs for sequences with lengths that would otherwise be cut into `chunks` (or clusters); 0
// where that is the better way.  Of p only the sizes are looked at.
int64_t decode_stream_bytes(const SdpaParams& p, int dtype, int num_sms, const DecodePlan& chunks, int* ctas);
// Turns a plan of several chunks into one with clusters where that is faster; never one that needs more workspace.
void decode_plan_clusters(const SdpaParams& p, int dtype, int num_sms, DecodePlan* plan);
cudaError_t launch_decode(const SdpaParams& p, int dtype, const DecodePlan& plan, float* workspace, cudaStream_t stream, int* launches);
bool decode_supported(int dtype, int head_dim);
int64_t decode_static_scratch_bytes();
cudaError_t launch_decode_static(const SdpaParams& p, int dtype, const DecodePlan& plan, cudaStream_t stream, int* launches);
cudaError_t launch_cast(int kind, const void* src, void* dst, int64_t n, cudaStream_t stream);
cudaError_t launch_paged_append(const void* src_k, const void* src_v, void* pool_k, void* pool_v,
                                const int32_t* block_table, int64_t start, int64_t tokens, int block_size, int num_blocks,
                                int64_t row_bytes, cudaStream_t stream);

// Attention backward (csrc/sdpa_backward.cu): the forward's parameter block (p.out = O, p.lse = log-sum-exp, both
// inputs here) plus dO, the gradient outputs and the delta scratch.
struct BwdParams {
  SdpaParams p;
  const void* dout;   // dtype of p.out
  int64_t dos[3];
  float* dq;          // [B, Hc, Sq, D] fp32, Hc = heads of the shard
  float* dk;          // [B, Hc / group, Sk, D] fp32
  float* dv;
  float* delta;       // [B, Hc, Sq] scratch
  void* dout_t;       // scratch: dO in the input dtype, dense [B, Hc, Sq, D] (16-bit inputs with an fp32 dO), or null
  int32_t no_tcgen05; // 1: stay on the mma.sync / FFMA kernels (desc.path == AIDN_PATH_GENERIC)
  int32_t expire;     // test hook of the tcgen05 kernels: loads are withheld and every bounded wait gives up after 20 ms
  int32_t round_dout; // set by the launcher: delta is summed from dO as rounded into dout_t (what the tensor-core
                      // kernels multiply with), so that every row of dS sums to zero as it does in exact arithmetic
};
// *used_tcgen05 tells which family ran the dQ and dK / dV launches.
cudaError_t launch_backward(const BwdParams& bp, int dtype, cudaStream_t stream, int* launches, int* used_tcgen05);
// tcgen05 dQ and dK / dV launches (csrc/sdpa_backward_sm100.cu); delta (and dout_t) must already be on the stream.
bool backward_sm100_supported(const BwdParams& bp, int dtype);
cudaError_t launch_backward_sm100(const BwdParams& bp, int dtype, cudaStream_t stream, int* launches, const char** why);
// fp32 dQ and dK / dV launches on packed multiply-adds (csrc/sdpa_backward_f32.cu); delta must already be on the stream.
bool backward_f32_supported(const BwdParams& bp, int dtype);
cudaError_t launch_backward_f32(const BwdParams& bp, cudaStream_t stream);
// The same as three bf16 terms on tcgen05 (csrc/sdpa_backward_f32_sm100.cu), of the calls that backward_f32_supported accepts.
bool backward_f32_sm100_supported(const BwdParams& bp);
inline bool backward_f32_sm100_fits(const SdpaParams& p) { return p.head_dim <= 64 && p.seq_q >= 320 && p.seq_kv >= 320; }
cudaError_t launch_backward_f32_sm100(const BwdParams& bp, cudaStream_t stream);

// Packed Q/K/V projection + RoPE + KV-cache write (csrc/qkv_rope_cache.cu).
struct QkvRopeParams {
  const float* input;
  const void* weights;
  const float* bias;
  const float* cosine;
  const float* sine;
  void* query;
  void* key_cache;
  void* value_cache;
  const int32_t* positions;
  const int32_t* cache_rows;
  int32_t tokens, heads, kv_heads, head_dim;
  int32_t position;
  int32_t query_dtype, cache_dtype;
  int64_t cache_capacity, max_position;
  int32_t model;
};

int64_t qkv_rope_max_model();
// expire: test hook - the tcgen05 kernel withholds its loads and its bounded waits give up after 20 ms.
cudaError_t launch_qkv_rope_cache(const QkvRopeParams& p, int weight_dtype, int num_sms, cudaStream_t stream,
                                  int* launches, bool expire = false);
// Several tokens with bf16 weights on tcgen05 (csrc/qkv_rope_sm100.cu); launch_qkv_rope_cache hands it what it takes.
bool qkv_rope_sm100_supported(const QkvRopeParams& p, int weight_dtype);
cudaError_t launch_qkv_rope_sm100(const QkvRopeParams& p, int num_sms, cudaStream_t stream, int* launches, bool expire);
int32_t* qkv_rope_sm100_status();   // address of its status word in the current context, or null
cudaError_t launch_rope_interleaved(const float* in, const float* cosc, const float* sinc, float* out, int64_t rows,
                                    int head_dim, int seq_len, int start_position, cudaStream_t stream);

// Per-handle memory of the tcgen05 prefill launcher: the four TMA tensor maps of the last launch, with the tensors
// they were encoded for, and which kernel instantiations already had their shared-memory limit raised in the
// handle's context.  A launch whose pointers, extents and strides match re-uses the maps; encoding happens on the host
// only and is capture-safe either way.
struct alignas(64) PrefillMapCache {
  unsigned char maps[4][128];   // CUtensorMap images: q, k, v, out
  struct Key {
    const void* q; const void* k; const void* v; const void* out;
    int64_t qs[3], ks[3], vs[3], os[3];
    int64_t seq_q, kv_rows;
    int32_t batch, kv_batch, num_q_heads, num_kv_heads, head_dim, kv_box, out_f32, splits, dtype;
  } key;
  bool valid;
  bool attr_set[40];            // by instantiation: 8 * (PrefillMode) + (epilogue warpgroup ? 4 : 0) + (fp16 ? 2 : 0) + (head_dim 128 ? 1 : 0)
};
bool prefill_sm100_supported(const SdpaParams& p, int dtype, const char** why);
// How many parts the keys of every work item should be cut into (1: none), and the workspace (16-byte aligned) that this
// takes.
int prefill_splits(const SdpaParams& p, int num_sms);
int64_t prefill_split_bytes(const SdpaParams& p, int splits);
// cache may be null (maps are then encoded on every call); workspace is read for splits > 1 only.
cudaError_t launch_prefill_sm100(const SdpaParams& p, int dtype, cudaStream_t stream, int32_t* sched, int num_sms,
                                 float* debug, int debug_mode, PrefillMapCache* cache, int splits, float* workspace,
                                 const char** why);

// How proj_gemm_f32_sm100 does one GEMM: columns of a tile, CTAs of a cluster that share its K, and whether they cut W into its terms
// themselves or copy them in from an image.
struct ProjPlanF32 {
  int32_t width, splits;
  bool cut_w;
};

// Projection GEMM of the fused multi-head-attention forward (csrc/proj_gemm_sm100.cu):
// c[i][b, s, n] = sum_k a[b, s, k] * w[i][k, n] for up to three weight matrices that share a; column n lands at
// c[i] + b*c_stride[0] + (n / head_dim)*c_stride[1] + s*c_stride[2] + n % head_dim.
struct ProjGemm {
  const void* a;        // [batch, seq, k] dense; 16-bit for the tcgen05 kernel
  const void* w[3];     // [k, n] row-major, same type as a
  void* c[3];
  int64_t c_stride[3];  // elements for (batch, head, sequence position)
  int64_t batch, seq, k, n;
  int32_t num_mats;
  int32_t head_dim;
  bool out_f32;         // fp32 output, else the input dtype
  bool bf16;            // bf16 inputs, else fp16
  void* image;          // the terms of w, in tiles of f32_plan (proj_gemm_f32_sm100 only)
  ProjPlanF32 f32_plan; // the same for the launch that writes the image and the one that reads it
};
bool proj_gemm_sm100_supported(const ProjGemm& g, const char** why);
// expire: test hook - the producer withholds its loads and every bounded wait gives up after 20 ms.
cudaError_t launch_proj_gemm_sm100(const ProjGemm& g, cudaStream_t stream, int num_sms, int32_t* status,
                                   const char** why, bool expire = false);
// fp32 operands with 16-byte rows, every one as three bf16 terms on tcgen05 (csrc/proj_gemm_f32_sm100.cu).  launch_proj_split_f32
// writes the terms of the weights of one or two GEMMs to their `image`, of proj_gemm_f32_sm100_bytes bytes each, for the GEMMs
// behind it on the stream; where that is 0 (few rows, or a plan made without `images`) a GEMM cuts its weights itself.
bool proj_gemm_f32_sm100_fits(int64_t k, int64_t n);
bool proj_gemm_f32_sm100_supported(const ProjGemm& g);
ProjPlanF32 proj_gemm_f32_sm100_plan(int64_t rows, int64_t k, int64_t n, int mats, int num_sms, bool images, bool launched);
int64_t proj_gemm_f32_sm100_bytes(const ProjPlanF32& plan, int64_t k, int64_t n, int mats);
cudaError_t launch_proj_split_f32(const ProjGemm* gemms, int count, cudaStream_t stream);
cudaError_t launch_proj_gemm_f32_sm100(const ProjGemm& g, cudaStream_t stream, int32_t* status, bool expire = false);
// The same contract in fp32 FFMA arithmetic for any sizes and for a / w of `dtype` (csrc/proj_gemm_generic.cu).
bool proj_gemm_generic_supported(const ProjGemm& g, const char** why);
cudaError_t launch_proj_gemm_generic(const ProjGemm& g, int dtype, cudaStream_t stream);

}  // namespace aidn
