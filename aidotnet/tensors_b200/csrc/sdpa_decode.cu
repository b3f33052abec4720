// Split-KV decode (seq_q == 1): the HBM-bound half of the attention path.
//
// One CTA streams one chunk of one (batch, kv head)'s keys and values exactly once, serves all query heads of that
// kv head, and forms an un-normalised partial (max, sum, acc[D]).  The partials of a (batch, head) are merged by
// log-sum-exp: among the CTAs of a cluster through distributed shared memory where few enough CTAs run at once, by a
// second kernel through a workspace otherwise (decode_plan_clusters).  Only keys below kv_len[b] (and the causal limit) are touched, so padding costs no
// bandwidth.  Three partial kernels:
//   * sdpa_decode_gqa_ring_kernel - fp16 / bf16, head_dim 64 or 128, up to 16 query heads per kv head (plain
//     multi-head attention included): K/V go through a per-warp cp.async shared-memory ring and both products run
//     on mma.sync with the heads as the M / N dimension.  This is the kernel the benchmark's decode step uses.
//   * sdpa_decode_stream_kernel   - the same ring over equal shares of the keys of all sequences together, for launches with
//     lengths (decode_stream_bytes): the shares follow from the lengths on the device.
//   * sdpa_decode_partial_kernel  - everything else (fp32 inputs, head_dim 256, more than 16 heads per kv head):
//     16-byte streaming loads straight into registers and FFMA arithmetic.
//
// Supersedes flash_decode_partial / flash_decode_reduce of the reference
// (src/AiDotNet.Tensors/Engines/DirectGpu/CUDA/Kernels/CudaFlashDecodeKernels.cs:19-81), which run one
// thread per (head, split) with a serial, uncoalesced walk over the cache and take a single sequence.
// The PAGED instantiation reads K/V through a block table and supersedes paged_attention_decode{,_gqa}
// (src/AiDotNet.Tensors/Engines/DirectGpu/CUDA/Kernels/CudaPagedAttentionKernels.cs:23-55, :97-124), which run
// one thread per head over the whole sequence.
//
// Scratch layout (fp32): acc[B][Hc][nchunks][D] followed by ml[B][Hc][nchunks][2], Hc = heads of the shard.
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "mma_sync.cuh"

namespace aidn {
namespace {

constexpr int kDecWarps = 4;
constexpr int kUnroll = 4;

template <typename T>
struct Vec16 {
  static constexpr int EPL = 16 / sizeof(T);
};

template <typename T>
__device__ __forceinline__ void unpack16(const uint4& u, float* f);
template <>
__device__ __forceinline__ void unpack16<float>(const uint4& u, float* f) {
  f[0] = __uint_as_float(u.x);
  f[1] = __uint_as_float(u.y);
  f[2] = __uint_as_float(u.z);
  f[3] = __uint_as_float(u.w);
}
template <>
__device__ __forceinline__ void unpack16<__nv_bfloat16>(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void unpack16<__half>(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// Visible key count of a decode query of batch entry b: padding limit, then the causal limit of query 0.
__device__ __forceinline__ int64_t causal_len(const SdpaParams& p, int64_t L) {
  if (p.causal) {
    int64_t c = p.causal_offset + 1;
    if (c < 0) c = 0;
    if (c < L) L = c;
  }
  return L;
}
__device__ __forceinline__ int64_t decode_len(const SdpaParams& p, int b) { return causal_len(p, kv_limit_of(p, b)); }

// What a CTA does with the merged partial of its keys.
enum DecodeMerge : int {
  kMergeWorkspace = 0,   // write it to the workspace; sdpa_decode_combine_kernel merges the splits
  kMergeDirect = 1,      // there is one split: it is the result
  kMergeCluster = 2,     // the splits are the CTAs of one cluster, which merge through distributed shared memory
  kMergeBoth = 3,        // `nchunks` clusters per item: each merges its CTAs' partials and writes the result to the workspace
};

// Keys [start, end) of CTA c of `parts`.  With clusters every sequence is cut evenly by its own length (in steps of 16 keys),
// so that the CTAs that wait for one another end together; otherwise by `chunk`.
__device__ __forceinline__ void split_range(int64_t L, int chunk, int parts, int c, int merge, int64_t& start, int64_t& end) {
  const int64_t step = merge >= kMergeCluster ? ((L + parts - 1) / parts + 15) / 16 * 16 : chunk;
  start = c * step;
  end = start + step < L ? start + step : L;
}

// Merge of a cluster's partials: each CTA holds ROWS heads as acc[ROWS][D], m[ROWS], l[ROWS] from shared address `part` on
// (m = -inf: it saw no key), and forms one share of the (head, column) pairs, the splits in rank order.
template <typename T, int D, int ROWS>
__device__ __forceinline__ void merge_cluster(const SdpaParams& p, int b, int h0, int nheads, int rank, int splits, uint32_t part,
                                              float* ws, int slot, int nslots) {
  constexpr int kMaxSplits = 8;
  cluster_sync_all();   // every CTA's partial is written
  const int stride = splits * (int)blockDim.x;
  for (int idx = rank * (int)blockDim.x + (int)threadIdx.x; idx < nheads * D; idx += stride) {
    const int hh = idx / D, d = idx - hh * D, h = h0 + hh;
    float m[kMaxSplits], l[kMaxSplits], a[kMaxSplits];
#pragma unroll
    for (int r = 0; r < kMaxSplits; ++r) {
      m[r] = -INFINITY;
      l[r] = a[r] = 0.f;
      if (r < splits) {
        m[r] = ld_cluster_f32(part + (uint32_t)((ROWS * D + hh) * 4), r);
        l[r] = ld_cluster_f32(part + (uint32_t)((ROWS * (D + 1) + hh) * 4), r);
        a[r] = ld_cluster_f32(part + (uint32_t)((hh * D + d) * 4), r);
      }
    }
    float M = -INFINITY;
#pragma unroll
    for (int r = 0; r < kMaxSplits; ++r) M = fmaxf(M, m[r]);
    float acc = 0.f, lsum = 0.f;
#pragma unroll
    for (int r = 0; r < kMaxSplits; ++r) {
      if (m[r] == -INFINITY) continue;   // a weight that underflows to 0 still carries the split's NaN and Inf
      const float w = softmax_exp<T>(m[r] - M);
      acc = fmaf(w, a[r], acc);
      lsum = fmaf(w, l[r], lsum);
    }
    if (nslots > 1) {
      const int64_t at = ((int64_t)b * p.head_count + (h - p.head_begin)) * nslots + slot;
      ws[at * D + d] = acc;
      if (d == 0) {
        float* ml = ws + (int64_t)p.batch * p.head_count * nslots * D;
        ml[at * 2] = M;
        ml[at * 2 + 1] = lsum;
      }
      continue;
    }
    store_out<T>(p.out, b * p.os[0] + (int64_t)h * p.os[1] + d, acc * (lsum > 0.f ? 1.f / lsum : 0.f), p.out_f32);
    if (p.lse && d == 0) p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q] = lsum > 0.f ? M + logf(lsum) : -INFINITY;
  }
  __syncwarp();
  cluster_sync_all();   // nobody reads this CTA's shared memory any more
}

template <typename T, int D, int GT, bool PAGED, bool HEAD_FAST>
__global__ void __launch_bounds__(kDecWarps * 32)
    sdpa_decode_partial_kernel(const SdpaParams p, const int chunk, const int nchunks, float* __restrict__ ws,
                               const int merge, const int cluster) {
  constexpr int EPL = Vec16<T>::EPL;
  constexpr int LPK = D / EPL;    // lanes per key row
  constexpr int KPI = 32 / LPK;   // keys per warp-wide load
  constexpr int NG = kDecWarps * KPI;
  static_assert(LPK >= 1 && LPK <= 32 && (LPK & (LPK - 1)) == 0, "head_dim not coverable by one warp load");

  __shared__ float sm_m[NG][GT];
  __shared__ float sm_l[NG][GT];
  __shared__ __align__(16) float sm_acc[NG][GT][D];
  // for the cluster: acc[GT][D], m[GT], l[GT].  Only fp32 calls get one here (decode_plan_clusters); 16-bit ones would carry the memory
  // and the merge for nothing (B8, 8 heads of 256, 4096 keys 59.6 -> 59.2 us without them; 4 x 96/4 heads of 128, 2000 keys 66.0 -> 65.1).
  constexpr bool kClusters = sizeof(T) == 4;
  __shared__ float sm_part[kClusters ? GT * (D + 2) : 1];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = lane / LPK, gl = lane % LPK, d0 = gl * EPL;
  const int gchunks = (p.group + GT - 1) / GT;
  const int b = blockIdx.z;
  // Token-major caches ([S, Hkv, D] and the paged pool) interleave the heads of one token: there the grid's fast
  // axis is the head, so that CTAs running together read neighbouring 256-byte pieces of the same DRAM pages.
  const int by = HEAD_FAST ? blockIdx.x : blockIdx.y;
  const int kvh = p.head_begin / p.group + by / gchunks;
  const int gc = by % gchunks;
  const int h0 = kvh * p.group + gc * GT;
  const int nheads = min(GT, p.group - gc * GT);
  const int c = HEAD_FAST ? blockIdx.y : blockIdx.x;

  pdl_wait();      // nothing above touches memory that an earlier kernel writes
  pdl_trigger();   // the merge may be set up while this kernel runs
  const int64_t L = decode_len(p, b);
  int64_t start, end;
  split_range(L, chunk, nchunks * cluster, c, merge, start, end);
  const int Hc = p.head_count;

  if (start >= L && merge < kMergeCluster) {
    if (merge == kMergeDirect && c == 0) {  // nothing visible: zero output, -inf LSE
      for (int idx = tid; idx < nheads * D; idx += kDecWarps * 32) {
        const int g = idx / D, d = idx - g * D;
        store_out<T>(p.out, b * p.os[0] + (int64_t)(h0 + g) * p.os[1] + d, 0.f, p.out_f32);
        if (p.lse && d == 0) p.lse[((int64_t)b * p.num_q_heads + h0 + g) * p.seq_q] = -INFINITY;
      }
    }
    return;
  }

  float qf[GT][EPL];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    const int h = h0 + (g < nheads ? g : 0);
    const T* qp = static_cast<const T*>(p.q) + b * p.qs[0] + (int64_t)h * p.qs[1] + d0;
    const uint4 u = *reinterpret_cast<const uint4*>(qp);
    unpack16<T>(u, qf[g]);
  }
  const T* kbase = static_cast<const T*>(p.k) + (PAGED ? 0 : b * p.ks[0]) + (int64_t)kvh * p.ks[1] + d0;
  const T* vbase = static_cast<const T*>(p.v) + (PAGED ? 0 : b * p.vs[0]) + (int64_t)kvh * p.vs[1] + d0;

  float m[GT], l[GT], acc[GT][EPL];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < EPL; ++e) acc[g][e] = 0.f;
  }

  bool bad_block = false;
  constexpr int KPW = KPI * kUnroll;
  // Paged: one block-table read per key, issued an iteration ahead of the row loads that need it; the entry stays
  // raw in its register until then.
  int32_t blk_next[kUnroll];
  if constexpr (PAGED) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int64_t key = start + warp * KPW + u * KPI + grp;
      blk_next[u] = key < end ? kv_block_read(p, b, key) : 0;
    }
  }
  for (int64_t kb = start + warp * KPW; kb < end; kb += kDecWarps * KPW) {
    uint4 kv[kUnroll], vv[kUnroll];
    bool ok[kUnroll];
    int64_t row[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int64_t key = kb + u * KPI + grp;
      ok[u] = key < end;
      row[u] = key;
      if constexpr (PAGED) {
        row[u] = ok[u] ? kv_row_from(p, key, blk_next[u], bad_block) : -1;
        ok[u] = row[u] >= 0;
        const int64_t key_next = key + kDecWarps * KPW;
        blk_next[u] = key_next < end ? kv_block_read(p, b, key_next) : 0;
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) kv[u] = ok[u] ? ld_stream16(kbase + row[u] * p.ks[2]) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) vv[u] = ok[u] ? ld_stream16(vbase + row[u] * p.vs[2]) : make_uint4(0, 0, 0, 0);

    float s[GT][kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      float kf[EPL];
      unpack16<T>(kv[u], kf);
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        float dot = 0.f;
#pragma unroll
        for (int e = 0; e < EPL; ++e) dot = fmaf(qf[g][e], kf[e], dot);
        s[g][u] = dot;
      }
    }
#pragma unroll
    for (int g = 0; g < GT; ++g)
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) s[g][u] += __shfl_xor_sync(0xffffffffu, s[g][u], o);
      }

#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float mt = -INFINITY;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int64_t key = kb + u * KPI + grp;
        float val = -INFINITY;
        if (ok[u] && g < nheads) val = finish_logit(p, s[g][u] * p.scale, b, h0 + g, 0, key, L);
        s[g][u] = val;
        mt = fmaxf(mt, val);
      }
      const float m_new = fmaxf(m[g], mt);
      if (m_new != -INFINITY) {
        const float corr = (m[g] == -INFINITY) ? 0.f : softmax_exp<T>(m[g] - m_new);
        float psum = 0.f;
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          s[g][u] = (s[g][u] == -INFINITY) ? 0.f : softmax_exp<T>(s[g][u] - m_new);
          psum += s[g][u];
        }
        l[g] = l[g] * corr + psum;
#pragma unroll
        for (int e = 0; e < EPL; ++e) acc[g][e] *= corr;
        m[g] = m_new;
      } else {
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) s[g][u] = 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      float vf[EPL];
      unpack16<T>(vv[u], vf);
#pragma unroll
      for (int g = 0; g < GT; ++g)
#pragma unroll
        for (int e = 0; e < EPL; ++e) acc[g][e] = fmaf(s[g][u], vf[e], acc[g][e]);
    }
  }

  report_bad_block(p, bad_block);
  // merge the NG lane groups of the CTA
  const int ng = warp * KPI + grp;
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    if (gl == 0) {
      sm_m[ng][g] = m[g];
      sm_l[ng][g] = l[g];
    }
    if constexpr (EPL == 8) {
      *reinterpret_cast<float4*>(&sm_acc[ng][g][d0]) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
      *reinterpret_cast<float4*>(&sm_acc[ng][g][d0 + 4]) = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
    } else {
      *reinterpret_cast<float4*>(&sm_acc[ng][g][d0]) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
    }
  }
  __syncthreads();

  for (int idx = tid; idx < nheads * D; idx += kDecWarps * 32) {
    const int g = idx / D, d = idx - g * D;
    float M = -INFINITY;
#pragma unroll
    for (int n = 0; n < NG; ++n) M = fmaxf(M, sm_m[n][g]);
    float a = 0.f, lsum = 0.f;
    if (M != -INFINITY) {
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        const float mn = sm_m[n][g];
        const float w = (mn == -INFINITY) ? 0.f : softmax_exp<T>(mn - M);
        a = fmaf(w, sm_acc[n][g][d], a);
        lsum = fmaf(w, sm_l[n][g], lsum);
      }
    }
    const int h = h0 + g;
    if (kClusters && merge >= kMergeCluster) {
      sm_part[g * D + d] = a;
      if (d == 0) {
        sm_part[GT * D + g] = M;
        sm_part[GT * (D + 1) + g] = lsum;
      }
    } else if (merge == kMergeDirect) {
      store_out<T>(p.out, b * p.os[0] + (int64_t)h * p.os[1] + d, lsum > 0.f ? a / lsum : 0.f, p.out_f32);
      if (p.lse && d == 0)
        p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q] = lsum > 0.f ? M + logf(lsum) : -INFINITY;
    } else {
      const int64_t slot = ((int64_t)b * Hc + (h - p.head_begin)) * nchunks + c;
      ws[slot * D + d] = a;
      if (d == 0) {
        float* ml = ws + (int64_t)p.batch * Hc * nchunks * D;
        ml[slot * 2] = M;
        ml[slot * 2 + 1] = lsum;
      }
    }
  }
  __syncwarp();
  if constexpr (kClusters)
    if (merge >= kMergeCluster) merge_cluster<T, D, GT>(p, b, h0, nheads, c % cluster, cluster, ptx::smem_u32(sm_part), ws, c / cluster, nchunks);
}

// ---- grouped-query decode on the warp-level tensor-core path ---------------------------------------------------
// With several query heads per KV head the FFMA kernel above is bound by its shuffle reductions (one per head and
// key), not by HBM.  Here the heads of one KV head are the M dimension of mma.sync.m16n8k16 (up to 16, zero padded):
// a warp takes 16 keys per step, S[16 heads x 16 keys] = Q K^T and O[16 heads x D] += P V run on the tensor
// cores, and K and V still stream from global memory exactly once with 16-byte loads straight into the fragment
// registers.  That works without shared memory or ldmatrix because a dot product does not care about the order of
// its terms: the d index is assigned to the MMA's k slots (for Q K^T) and to its n columns (for P V) in whatever
// order the coalesced 16-byte loads deliver it, Q is loaded once in the matching order, and the output columns are
// un-permuted when the accumulators are written out.  The one re-arrangement needed, pairing two keys of the same
// d in one 32-bit B register for P V, is a byte permute of two loaded registers.
//
// Fragment geometry (g = lane / 4, c = lane % 4), per 16-key step starting at key kb:
//   K: thread loads rows kb + g and kb + 8 + g, 16-byte chunks i*4 + c (i < D/32); chunk register pair h supplies
//      k-step 2i + h: slots (2c, 2c+1) <- d = (i*4+c)*8 + 4h + {0,1}, slots (2c+8, 2c+9) <- d = ... + 2 + {0,1}.
//   V: P V runs transposed, O^T[d x heads] += V^T[d x keys] P^T[keys x heads], so that the 8 (or 16) live heads
//      are the N dimension and no accumulator register is spent on padding.  The thread loads rows
//      kb + {2c, 2c+1, 2c+8, 2c+9}; for D = 128 chunks g and g + 8, for D = 64 chunk g.  M-tile m has its row r at
//      d = r*8 + m (D = 128) or d = (r % 8)*8 + 4*(r / 8) + m (D = 64); the S accumulators of Q K^T are, as they
//      stand, the B fragments of P^T.

// Feeding: each warp owns a ring of kRingStages shared-memory stages (16 keys of K and 16 of V each) filled with
// 16-byte cp.async copies - a warp-wide copy moves two whole rows, so requests are fully coalesced - and retired in
// order with cp.async.wait_group: up to kRingStages steps per warp are in flight whatever the register budget (a
// variant that prefetched into registers held one step in flight and reached 0.71 of the HBM peak where this one
// reaches 0.85), there is no flag to spin on, and rows past the chunk's end or outside the pool are zero-filled by
// the copy itself (source size 0).  Rows are stored un-padded with their 16-byte chunks XOR-swizzled
// (K: chunk ^ 4*(row & 1); V: chunk ^ 2*((row / 2) & 3)) so that the fragment reads of both products are
// bank-conflict free.  After the loop a warp reuses its own ring for the partials it hands to the merge.
// NH16: more than 8 query heads per KV head (rows 8..15 of the tile are live).
constexpr int kRingStages = 3;
// CTAs of the ring kernels that an SM holds: by shared memory, and the compiler is held to it in registers.  (Left at two, heads of 64 took 168 to 186
// of them for more than eight query heads, so that a third of the equal shares were a second wave: 245 items of up to 3521 keys and nine
// heads 73 us, with three 46.)
template <int D>
constexpr int kRingCtas = D == 128 ? 2 : 3;

template <int D>
struct RingCfg {
  static constexpr int kRowBytes = D * 2;
  static constexpr int kKBytes = 16 * kRowBytes;
  static constexpr int kStageBytes = 2 * kKBytes;
  static constexpr int kWarpBytes = kRingStages * kStageBytes;
  static constexpr int kSmemBytes = kDecWarps * kWarpBytes;
  static_assert(kWarpBytes >= 16 * (D + 2) * 4, "a warp's partials must fit in its ring");
};


// What the 16-bit weights pb leave of pr.
template <typename T>
__device__ __forceinline__ uint32_t pack_rest(float a, float b, uint32_t packed) {
  float hi[2];
  if constexpr (std::is_same_v<T, __half>) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&packed));
    hi[0] = f.x; hi[1] = f.y;
  } else {
    hi[0] = __uint_as_float(packed << 16);
    hi[1] = __uint_as_float(packed & 0xffff0000u);
  }
  return pack_pair<T>(a - hi[0], b - hi[1]);
}

// A warp's query heads of one KV head and what it has summed up for them.
template <typename T, int D, bool NH16>
struct RingWarp {
  static constexpr int KI = D / 32, VX = D / 64, MT = D / 16, HN = NH16 ? 2 : 1;
  using R = RingCfg<D>;
  uint32_t qa[KI][4], qb[KI][4];   // Q in fragment order
  float acc[MT][HN][4];
  float m0, m1, l0, l1;

  __device__ __forceinline__ void begin(const SdpaParams& p, int b, int h0, int nheads, int g, int c) {
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      uint4 u = make_uint4(0, 0, 0, 0), w = make_uint4(0, 0, 0, 0);
      if (g < nheads)
        u = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.q) + b * p.qs[0] + (int64_t)(h0 + g) * p.qs[1] + (i * 4 + c) * 8);
      if (NH16 && g + 8 < nheads)
        w = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.q) + b * p.qs[0] + (int64_t)(h0 + g + 8) * p.qs[1] + (i * 4 + c) * 8);
      qa[i][0] = u.x; qa[i][1] = u.y; qa[i][2] = u.z; qa[i][3] = u.w;
      qb[i][0] = w.x; qb[i][1] = w.y; qb[i][2] = w.z; qb[i][3] = w.w;
    }
#pragma unroll
    for (int j = 0; j < MT; ++j)
#pragma unroll
      for (int hn = 0; hn < HN; ++hn) acc[j][hn][0] = acc[j][hn][1] = acc[j][hn][2] = acc[j][hn][3] = 0.f;
    m0 = m1 = -INFINITY;
    l0 = l1 = 0.f;
  }

  // The 16 keys from kb on, in the stage at `base`; bit i of rows_ok: key kb + i counts.  `refill` is called when the stage has been read.
  // two_terms: the weights go into their product as two 16-bit terms (sdpa_decode_stream_kernel).
  template <typename Refill>
  __device__ __forceinline__ void step(const SdpaParams& p, uint32_t base, uint32_t rows_ok, int b, int h0, int nheads, int64_t kb, int64_t L, int g,
                                       int c, bool two_terms, Refill refill) {
    // ---- S = Q K^T ------------------------------------------------------------------------------------
    float sacc[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      sacc[t][0] = sacc[t][1] = sacc[t][2] = sacc[t][3] = 0.f;
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        uint32_t kw[4];
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(kw[0]), "=r"(kw[1]), "=r"(kw[2]), "=r"(kw[3])
                     : "r"(base + (t * 8 + g) * R::kRowBytes + (((i * 4 + c) ^ ((g & 1) << 2)) << 4)));
#pragma unroll
        for (int h = 0; h < 2; ++h)
          mma16816<T>(sacc[t], qa[i][2 * h], qb[i][2 * h], qa[i][2 * h + 1], qb[i][2 * h + 1], kw[2 * h], kw[2 * h + 1]);
      }
    }
    // ---- V fragments to registers, then the stage is free for the copies two steps ahead ---------------
    uint32_t vw[4][VX][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int x = 0; x < VX; ++x) {
        const int vr = 2 * c + (e & 1) + (e >> 1) * 8;   // (vr / 2) & 3 == c
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(vw[e][x][0]), "=r"(vw[e][x][1]), "=r"(vw[e][x][2]), "=r"(vw[e][x][3])
                     : "r"(base + R::kKBytes + vr * R::kRowBytes + (((g + 8 * x) ^ (c << 1)) << 4)));
      }
    __syncwarp();   // every lane has read the stage: refill it with the step kRingStages ahead
    refill();

    // ---- online softmax over the step's 16 keys ---------------------------------------------------------
    float pr[2][4];
    {
      float mt0 = -INFINITY, mt1 = -INFINITY;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int idx = t * 8 + 2 * c + e;
          const int64_t key = kb + idx;
          const bool ok = (rows_ok >> idx) & 1u;
          float v0 = -INFINITY, v1 = -INFINITY;
          if (ok && g < nheads) v0 = finish_logit(p, sacc[t][e] * p.scale, b, h0 + g, 0, key, L);
          if (NH16 && ok && g + 8 < nheads) v1 = finish_logit(p, sacc[t][2 + e] * p.scale, b, h0 + g + 8, 0, key, L);
          sacc[t][e] = v0;
          sacc[t][2 + e] = v1;
          mt0 = fmaxf(mt0, v0);
          mt1 = fmaxf(mt1, v1);
        }
      mt0 = fmaxf(mt0, __shfl_xor_sync(0xffffffffu, mt0, 1));
      mt0 = fmaxf(mt0, __shfl_xor_sync(0xffffffffu, mt0, 2));
      if (NH16) {
        mt1 = fmaxf(mt1, __shfl_xor_sync(0xffffffffu, mt1, 1));
        mt1 = fmaxf(mt1, __shfl_xor_sync(0xffffffffu, mt1, 2));
      }
      const float n0 = fmaxf(m0, mt0), n1 = fmaxf(m1, mt1);
      const float c0 = (m0 == -INFINITY) ? 0.f : softmax_exp<T>(m0 - n0);
      const float c1 = (m1 == -INFINITY) ? 0.f : softmax_exp<T>(m1 - n1);
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          pr[t][e] = (sacc[t][e] == -INFINITY) ? 0.f : softmax_exp<T>(sacc[t][e] - n0);
          pr[t][2 + e] = (!NH16 || sacc[t][2 + e] == -INFINITY) ? 0.f : softmax_exp<T>(sacc[t][2 + e] - n1);
          s0 += pr[t][e];
          s1 += pr[t][2 + e];
        }
      l0 = l0 * c0 + s0;
      l1 = l1 * c1 + s1;
      m0 = n0;
      m1 = n1;
      const float ca = __shfl_sync(0xffffffffu, c0, 8 * c), cb = __shfl_sync(0xffffffffu, c0, 8 * c + 4);
#pragma unroll
      for (int j = 0; j < MT; ++j) {
        acc[j][0][0] *= ca;
        acc[j][0][1] *= cb;
        acc[j][0][2] *= ca;
        acc[j][0][3] *= cb;
      }
      if (NH16) {
        const float cc = __shfl_sync(0xffffffffu, c1, 8 * c), cd = __shfl_sync(0xffffffffu, c1, 8 * c + 4);
#pragma unroll
        for (int j = 0; j < MT; ++j) {
          acc[j][HN - 1][0] *= cc;
          acc[j][HN - 1][1] *= cd;
          acc[j][HN - 1][2] *= cc;
          acc[j][HN - 1][3] *= cd;
        }
      }
    }
    const uint32_t pb0 = pack_pair<T>(pr[0][0], pr[0][1]), pb1 = pack_pair<T>(pr[1][0], pr[1][1]);
    const uint32_t pc0 = pack_pair<T>(pr[0][2], pr[0][3]), pc1 = pack_pair<T>(pr[1][2], pr[1][3]);
    uint32_t rb0 = 0, rb1 = 0, rc0 = 0, rc1 = 0;
    if (two_terms) {
      rb0 = pack_rest<T>(pr[0][0], pr[0][1], pb0);
      rb1 = pack_rest<T>(pr[1][0], pr[1][1], pb1);
      rc0 = pack_rest<T>(pr[0][2], pr[0][3], pc0);
      rc1 = pack_rest<T>(pr[1][2], pr[1][3], pc1);
    }

    // ---- O^T += V^T P^T ------------------------------------------------------------------------------------
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint32_t sel = (m & 1) ? 0x7632u : 0x5410u;
      constexpr int xh = VX - 1;
      const int wl = m >> 1, wh = (D == 128) ? (m >> 1) : 2 + (m >> 1);
      const uint32_t a0 = __byte_perm(vw[0][0][wl], vw[1][0][wl], sel);
      const uint32_t a1 = __byte_perm(vw[0][xh][wh], vw[1][xh][wh], sel);
      const uint32_t a2 = __byte_perm(vw[2][0][wl], vw[3][0][wl], sel);
      const uint32_t a3 = __byte_perm(vw[2][xh][wh], vw[3][xh][wh], sel);
      mma16816<T>(acc[m][0], a0, a1, a2, a3, pb0, pb1);
      if (NH16) mma16816<T>(acc[m][HN - 1], a0, a1, a2, a3, pc0, pc1);
      if (two_terms) {
        mma16816<T>(acc[m][0], a0, a1, a2, a3, rb0, rb1);
        if (NH16) mma16816<T>(acc[m][HN - 1], a0, a1, a2, a3, rc0, rc1);
      }
    }
  }

  // The row sums, which are in four lanes' parts.
  __device__ __forceinline__ void gather_sums() {
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  }
};

// CTAS: that the compiler leaves registers for.
template <typename T, int D, bool NH16, bool PAGED, bool HEAD_FAST, int CTAS>
__global__ void __launch_bounds__(kDecWarps * 32, CTAS)
    sdpa_decode_gqa_ring_kernel(const SdpaParams p, const int chunk, const int nchunks, float* __restrict__ ws,
                                const int merge, const int cluster) {
  static_assert(sizeof(T) == 2 && (D == 64 || D == 128), "16-bit inputs, head_dim 64 or 128");
  using R = RingCfg<D>;
  constexpr int MT = D / 16, HN = NH16 ? 2 : 1;
  constexpr int ROWS = NH16 ? 16 : 8;
  constexpr int NG = kDecWarps;
  constexpr int kStep = 16;

  extern __shared__ __align__(128) uint8_t ring_smem[];
  const uint32_t smem0 = ptx::smem_u32(ring_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, c = lane & 3;
  const int b = blockIdx.z;
  const int kvh = p.head_begin / p.group + (HEAD_FAST ? (int)blockIdx.x : (int)blockIdx.y);
  const int h0 = kvh * p.group;
  const int nheads = p.group;
  const int cidx = HEAD_FAST ? blockIdx.y : blockIdx.x;

  pdl_wait();      // nothing above touches memory that an earlier kernel writes
  pdl_trigger();   // the merge may be set up while this kernel runs
  const int64_t L = decode_len(p, b);
  int64_t start, end;
  split_range(L, chunk, nchunks * cluster, cidx, merge, start, end);
  const int Hc = p.head_count;

  if (start >= L && merge < kMergeCluster) {
    if (merge == kMergeDirect && cidx == 0) {
      for (int idx = tid; idx < nheads * D; idx += kDecWarps * 32) {
        const int hh = idx / D, d = idx - hh * D;
        store_out<T>(p.out, b * p.os[0] + (int64_t)(h0 + hh) * p.os[1] + d, 0.f, p.out_f32);
        if (p.lse && d == 0) p.lse[((int64_t)b * p.num_q_heads + h0 + hh) * p.seq_q] = -INFINITY;
      }
    }
    return;
  }

  const uint32_t my_ring = smem0 + warp * R::kWarpBytes;
  const T* kbase = static_cast<const T*>(p.k) + (PAGED ? 0 : b * p.ks[0]) + (int64_t)kvh * p.ks[1];
  const T* vbase = static_cast<const T*>(p.v) + (PAGED ? 0 : b * p.vs[0]) + (int64_t)kvh * p.vs[1];
  bool bad_block = false;

  constexpr int CH = D / 8;          // 16-byte chunks per row
  constexpr int RPL = 16 * CH / 32;  // rows each lane copies per step (of K, and of V)
  const int my_ch = lane % CH, my_r0 = lane / CH;
  // Raw block-table entry of key kb + lane % 16 (paged), read a step before the copies that need it are issued.
  auto entry_of = [&](int64_t kb) -> int32_t {
    if constexpr (PAGED) {
      const int64_t key = kb + (lane & 15);
      return key < end ? kv_block_read(p, b, key) : 0;
    } else {
      return 0;
    }
  };
  // Issues the copies of the step at kb into `stage` and commits them as one group.  Returns the step's row mask
  // (bit i: key kb + i is inside the chunk and its row inside the pool); the other rows are zero-filled.
  auto issue = [&](int stage, int64_t kb, int32_t entry) -> uint32_t {
    const int64_t key = kb + (lane & 15);
    int64_t row = -1;
    if (key < end) {
      if constexpr (PAGED) row = kv_row_from(p, key, entry, bad_block);
      else row = key;
    }
    const uint32_t base = my_ring + stage * R::kStageBytes;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int ri = my_r0 + (32 / CH) * r;
      const int64_t rr = __shfl_sync(0xffffffffu, row, ri);
      const bool valid = rr >= 0;
      const int64_t ro = valid ? rr : 0;
      cp_async16(base + ri * R::kRowBytes + ((my_ch ^ ((ri & 1) << 2)) << 4), kbase + ro * p.ks[2] + my_ch * 8, valid);
      cp_async16(base + R::kKBytes + ri * R::kRowBytes + ((my_ch ^ (((ri >> 1) & 3) << 1)) << 4),
                 vbase + ro * p.vs[2] + my_ch * 8, valid);
    }
    cp_async_commit();
    return __ballot_sync(0xffffffffu, row >= 0) & 0xffffu;
  };

  RingWarp<T, D, NH16> rw;
  rw.begin(p, b, h0, nheads, g, c);

  // prologue: fill the ring (a group is committed per stage even when it is empty, so that wait_group counts steps)
  const int64_t kb0 = start + warp * kStep;
  constexpr int64_t kStride = NG * kStep;
  uint32_t row_mask[kRingStages];
  // The first entries are read together, in one latency; not by the instantiation that has no registers to spare (217 items of 229 keys, nine
  // heads of 128 25.8 -> 26.8 us).
  constexpr bool kTogether = !(NH16 && D == 128);
  int32_t first_entries[kRingStages];
  if (kTogether) {
#pragma unroll
    for (int s = 0; s < kRingStages; ++s) first_entries[s] = entry_of(kb0 + s * kStride);
  }
#pragma unroll
  for (int s = 0; s < kRingStages; ++s) {
    const int64_t kbs = kb0 + s * kStride;
    row_mask[s] = 0;
    if (kbs < end) row_mask[s] = issue(s, kbs, kTogether ? first_entries[s] : entry_of(kbs));
    else cp_async_commit();
  }
  int32_t ent_next = entry_of(kb0 + kRingStages * kStride);

  int step = 0;
  for (int64_t kb = kb0; kb < end; kb += kStride, ++step) {
    const int stage = step % kRingStages;
    cp_async_wait<kRingStages - 1>();   // this step's group has landed (later steps may still be in flight)
    __syncwarp();                       // ... for every lane's copies
    const uint32_t base = my_ring + stage * R::kStageBytes;
    uint32_t rows_ok = 0;
#pragma unroll
    for (int s = 0; s < kRingStages; ++s)
      if (s == stage) rows_ok = row_mask[s];

    rw.step(p, base, rows_ok, b, h0, nheads, kb, L, g, c, false, [&] {
        const int64_t kb_new = kb + kRingStages * kStride;
        const int32_t ent_new = ent_next;
        ent_next = entry_of(kb_new + kStride);
        uint32_t mask_new = 0;
        if (kb_new < end) mask_new = issue(stage, kb_new, ent_new);
        else cp_async_commit();
#pragma unroll
        for (int s = 0; s < kRingStages; ++s)
          if (s == stage) row_mask[s] = mask_new;
    });
  }

  report_bad_block(p, bad_block);
  cp_async_wait<0>();
  __syncwarp();
  // The warp's ring is free now: its partials go there.
  float* sm_acc = reinterpret_cast<float*>(ring_smem + warp * R::kWarpBytes);   // [ROWS][D], then m[ROWS], l[ROWS]
  float* sm_m = sm_acc + ROWS * D;
  float* sm_l = sm_m + ROWS;
  constexpr int kWarpFloats = R::kWarpBytes / 4;
  // ---- merge the warps of the CTA ---------------------------------------------------------------------------
  rw.gather_sums();
  if (c == 0) {
    sm_m[g] = rw.m0;
    sm_l[g] = rw.l0;
    if (NH16) {
      sm_m[g + 8] = rw.m1;
      sm_l[g + 8] = rw.l1;
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const int d_lo = g * 8 + m, d_hi = (D == 128) ? (g + 8) * 8 + m : g * 8 + 4 + m;
#pragma unroll
    for (int hn = 0; hn < HN; ++hn)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sm_acc[(8 * hn + 2 * c + e) * D + d_lo] = rw.acc[m][hn][e];
        sm_acc[(8 * hn + 2 * c + e) * D + d_hi] = rw.acc[m][hn][2 + e];
      }
  }
  __syncthreads();

  const float* all = reinterpret_cast<const float*>(ring_smem);   // warp n's partials start at n * kWarpFloats
  float* part = reinterpret_cast<float*>(ring_smem) + ROWS * (D + 2);   // for the cluster: acc[ROWS][D], m[ROWS], l[ROWS], behind warp 0's
  static_assert(2 * ROWS * (D + 2) <= kWarpFloats, "the CTA's partials must fit behind warp 0's");
  for (int idx = tid; idx < nheads * D; idx += kDecWarps * 32) {
    const int hh = idx / D, d = idx - hh * D;
    float M = -INFINITY;
#pragma unroll
    for (int n = 0; n < NG; ++n) M = fmaxf(M, all[n * kWarpFloats + ROWS * D + hh]);
    float a = 0.f, lsum = 0.f;
    if (M != -INFINITY) {
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        const float mn = all[n * kWarpFloats + ROWS * D + hh];
        const float wgt = (mn == -INFINITY) ? 0.f : softmax_exp<T>(mn - M);
        a = fmaf(wgt, all[n * kWarpFloats + hh * D + d], a);
        lsum = fmaf(wgt, all[n * kWarpFloats + ROWS * D + ROWS + hh], lsum);
      }
    }
    const int h = h0 + hh;
    if (merge >= kMergeCluster) {
      part[hh * D + d] = a;
      if (d == 0) {
        part[ROWS * D + hh] = M;
        part[ROWS * (D + 1) + hh] = lsum;
      }
    } else if (merge == kMergeDirect) {
      store_out<T>(p.out, b * p.os[0] + (int64_t)h * p.os[1] + d, lsum > 0.f ? a / lsum : 0.f, p.out_f32);
      if (p.lse && d == 0)
        p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q] = lsum > 0.f ? M + logf(lsum) : -INFINITY;
    } else {
      const int64_t slot = ((int64_t)b * Hc + (h - p.head_begin)) * nchunks + cidx;
      ws[slot * D + d] = a;
      if (d == 0) {
        float* ml = ws + (int64_t)p.batch * Hc * nchunks * D;
        ml[slot * 2] = M;
        ml[slot * 2 + 1] = lsum;
      }
    }
  }
  __syncwarp();
  if (merge >= kMergeCluster) merge_cluster<T, D, ROWS>(p, b, h0, nheads, cidx % cluster, cluster, ptx::smem_u32(part), ws, cidx / cluster, nchunks);
}

// ---- sequences of unequal lengths: equal shares of all keys --------------------------------------------------------
// The keys of a launch are one row of 16-key steps, sequence after sequence, which is cut into equal shares; neighbouring warps take the
// KV heads of one share, so that what lies together in a pool is read together, and all of them are resident at once.  A warp streams
// its share through its ring without a pause at the ends of sequences, of which it writes a partial each: share j's partial of
// sequence b is slot j + b (both only ever grow by one along the row), so that a sequence's slots are neighbours and the merge finds
// them from the lengths alone.
// Cut by sequence and head, the CTA of the longest sequence ran on alone, and every CTA spent 5 us on its way to its first keys
// and on its merge (16 sequences of 128 to 2048 keys, Hq32 / Hkv8 D128, 71 MB: 26.9 us in clusters of two, 27.3 in chunks of 256).
struct StreamPlan {
  int total, per;   // steps of a KV head, and of a share
};
constexpr int kStreamLeast = 4;   // steps of a share at least
__device__ __forceinline__ int stream_steps(const SdpaParams& p, int b) { return (int)((decode_len(p, b) + 15) / 16); }
// The same for the merge, which reads the lengths ahead of its wait (sdpa_decode_stream_kernel triggers behind its own); there are lengths.
__device__ __forceinline__ int stream_steps_early(const SdpaParams& p, int b) {
  const int64_t n = ld_l2(p.kv_len + b);
  return (int)((causal_len(p, n < 0 ? 0 : (n < p.seq_kv ? n : p.seq_kv)) + 15) / 16);
}
__device__ __forceinline__ StreamPlan stream_plan(int total, int shares) {
  StreamPlan s;
  s.total = total;
  s.per = (total + shares - 1) / shares;
  if (s.per < kStreamLeast) s.per = kStreamLeast;
  return s;
}

template <typename T, int D, bool NH16, bool PAGED>
__global__ void __launch_bounds__(kDecWarps * 32, kRingCtas<D>) sdpa_decode_stream_kernel(const SdpaParams p, float* __restrict__ ws, const int kv_heads, const int shares) {
  using R = RingCfg<D>;
  constexpr int MT = D / 16, HN = NH16 ? 2 : 1;
  extern __shared__ __align__(128) uint8_t ring_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int w = (int)blockIdx.x * kDecWarps + warp, share = w / kv_heads, kvh = w - share * kv_heads;
  const int nheads = p.group, h0 = p.head_begin + kvh * p.group;
  const uint32_t my_ring = ptx::smem_u32(ring_smem) + warp * R::kWarpBytes;
  pdl_wait();
  pdl_trigger();   // the merge finds its slots while this kernel runs

  int all = 0;
  for (int b0 = 0; b0 < p.batch; b0 += 32) all += __reduce_add_sync(0xffffffffu, b0 + lane < p.batch ? stream_steps(p, b0 + lane) : 0);
  const StreamPlan plan = stream_plan(all, shares);
  const int x0 = share * plan.per, x1 = x0 + plan.per < plan.total ? x0 + plan.per : plan.total;
  if (share >= shares || x0 >= x1) return;

  // A place on the row of steps.
  struct Cursor {
    int b, s, steps;   // sequence, step, steps of the sequence
    int64_t L;
  };
  auto at_sequence = [&](Cursor& k, int b) {
    k.b = b;
    k.L = decode_len(p, b);
    k.steps = (int)((k.L + 15) / 16);
  };
  auto advance = [&](Cursor& k) {   // (only where there is a next step)
    if (++k.s < k.steps) return;
    k.s = 0;
    do at_sequence(k, k.b + 1);
    while (k.steps == 0);
  };
  Cursor cur;
  {
    int before = 0, found = -1, found_before = 0;
    for (int b0 = 0; b0 < p.batch && found < 0; b0 += 32) {
      const int mine = b0 + lane < p.batch ? stream_steps(p, b0 + lane) : 0;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += y;
      }
      const uint32_t past = __ballot_sync(0xffffffffu, x0 < before + upto);
      if (past) {
        const int at = __ffs(past) - 1;
        found = b0 + at;
        found_before = before + __shfl_sync(0xffffffffu, upto - mine, at);
      }
      before += __shfl_sync(0xffffffffu, upto, 31);
    }
    at_sequence(cur, found);
    cur.s = x0 - found_before;
  }

  bool bad_block = false;
  constexpr int CH = D / 8, RPL = 16 * CH / 32;   // 16-byte chunks per row; rows that a lane copies per step
  const int my_ch = lane % CH, my_r0 = lane / CH;
  const T* head_k = static_cast<const T*>(p.k) + (int64_t)(h0 / p.group) * p.ks[1];
  const T* head_v = static_cast<const T*>(p.v) + (int64_t)(h0 / p.group) * p.vs[1];
  auto entry_of = [&](const Cursor& k) -> int32_t {
    if constexpr (PAGED) {
      const int64_t key = (int64_t)k.s * 16 + (lane & 15);
      return key < k.L ? kv_block_read(p, k.b, key) : 0;
    } else {
      return 0;
    }
  };
  auto issue = [&](int stage, const Cursor& k, int32_t entry) -> uint32_t {
    const int64_t key = (int64_t)k.s * 16 + (lane & 15);
    int64_t row = -1;
    if (key < k.L) {
      if constexpr (PAGED) row = kv_row_from(p, key, entry, bad_block);
      else row = key;
    }
    const T* kbase = head_k + (PAGED ? 0 : k.b * p.ks[0]);
    const T* vbase = head_v + (PAGED ? 0 : k.b * p.vs[0]);
    const uint32_t base = my_ring + stage * R::kStageBytes;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int ri = my_r0 + (32 / CH) * r;
      const int64_t rr = __shfl_sync(0xffffffffu, row, ri);
      const bool valid = rr >= 0;
      const int64_t ro = valid ? rr : 0;
      cp_async16(base + ri * R::kRowBytes + ((my_ch ^ ((ri & 1) << 2)) << 4), kbase + ro * p.ks[2] + my_ch * 8, valid);
      cp_async16(base + R::kKBytes + ri * R::kRowBytes + ((my_ch ^ (((ri >> 1) & 3) << 1)) << 4), vbase + ro * p.vs[2] + my_ch * 8, valid);
    }
    return __ballot_sync(0xffffffffu, row >= 0) & 0xffffu;
  };

  // The ring runs ahead of the products by its stages, across the ends of sequences.  A group is committed even where there is no
  // step, so that wait_group counts steps; the entries of the first steps are read together, later ones a step before they are needed.
  uint32_t row_mask[kRingStages];
  Cursor ahead = cur;
  int x_ahead = x0 + kRingStages;
  int32_t entry = 0;
  {
    Cursor k[kRingStages];
    int32_t e[kRingStages];
#pragma unroll
    for (int s = 0; s < kRingStages; ++s) {
      k[s] = ahead;
      e[s] = x0 + s < x1 ? entry_of(ahead) : 0;
      if (x0 + s + 1 < x1) advance(ahead);
    }
    if (x_ahead < x1) entry = entry_of(ahead);
#pragma unroll
    for (int s = 0; s < kRingStages; ++s) {
      row_mask[s] = x0 + s < x1 ? issue(s, k[s], e[s]) : 0;
      cp_async_commit();
    }
  }
  auto feed = [&](int stage) -> uint32_t {
    uint32_t mask = 0;
    if (x_ahead < x1) {
      const Cursor now = ahead;
      const int32_t e = entry;
      if (++x_ahead < x1) {
        advance(ahead);
        entry = entry_of(ahead);
      }
      mask = issue(stage, now, e);
    }
    cp_async_commit();
    return mask;
  };

  // A weight is 1 without rounding where its key is the largest of a partial, and shares have fewer partials than chunks: with weights of one term, outputs
  // are 0.7 to 4 % further from 64 bits than by chunks.  16-bit outputs therefore get two (16 sequences of up to 2048 keys with their projection
  // 2.44e-3 -> 1.94e-3, by chunks 2.42e-3; the time is the same).  fp32 outputs, which would move by what the rounding is, 1.5e-3, keep the values they have.
  const bool two_terms = !p.out_f32;
  RingWarp<T, D, NH16> rw;
  rw.begin(p, cur.b, h0, nheads, g, c);
  for (int x = x0; x < x1; ++x) {
    const int stage = (x - x0) % kRingStages;
    cp_async_wait<kRingStages - 1>();
    __syncwarp();
    uint32_t rows_ok = 0;
#pragma unroll
    for (int s = 0; s < kRingStages; ++s)
      if (s == stage) rows_ok = row_mask[s];
    rw.step(p, my_ring + stage * R::kStageBytes, rows_ok, cur.b, h0, nheads, (int64_t)cur.s * 16, cur.L, g, c, two_terms, [&] {
      const uint32_t mask = feed(stage);
#pragma unroll
      for (int s = 0; s < kRingStages; ++s)
        if (s == stage) row_mask[s] = mask;
    });
    const bool last = x + 1 == x1;
    if (last || cur.s + 1 == cur.steps) {   // the end of the sequence, or of the share
      rw.gather_sums();
      const int64_t slot = ((int64_t)(share + cur.b) * kv_heads + kvh) * nheads;
      float* ml = ws + (int64_t)(shares + p.batch) * kv_heads * nheads * D;
      if (c == 0) {
        if (g < nheads) *reinterpret_cast<float2*>(ml + (slot + g) * 2) = make_float2(rw.m0, rw.l0);
        if (NH16 && g + 8 < nheads) *reinterpret_cast<float2*>(ml + (slot + g + 8) * 2) = make_float2(rw.m1, rw.l1);
      }
      // a thread's columns of a head are neighbours: d = 8 g + m and, from the second half of the fragments, 64 + 8 g + m (D 128) or 8 g + 4 + m
#pragma unroll
      for (int hn = 0; hn < HN; ++hn)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int hh = 8 * hn + 2 * c + e;
          if (hh >= nheads) continue;
          float* dst = ws + (slot + hh) * D + g * 8;
#pragma unroll
          for (int m = 0; m < MT; m += 4) {
            *reinterpret_cast<float4*>(dst + m) = make_float4(rw.acc[m][hn][e], rw.acc[m + 1][hn][e], rw.acc[m + 2][hn][e], rw.acc[m + 3][hn][e]);
            *reinterpret_cast<float4*>(dst + (D == 128 ? 64 : 4) + m) =
                make_float4(rw.acc[m][hn][2 + e], rw.acc[m + 1][hn][2 + e], rw.acc[m + 2][hn][2 + e], rw.acc[m + 3][hn][2 + e]);
          }
        }
      if (!last) {
        advance(cur);
        rw.begin(p, cur.b, h0, nheads, g, c);
      }
    } else {
      advance(cur);
    }
  }
  report_bad_block(p, bad_block);
}

// Merges the splits of one (sequence, head): the weight of every split is formed once, in parallel, and the columns are
// summed by 16-byte vectors over groups of splits.  Bound by latency - a few KB per CTA - so nothing in it is a serial
// chain over the splits except the last sum of 128 / (D / 4) partial columns.
constexpr int kMaxCombine = 1024;   // split weights held in shared memory; more splits are taken in rounds

template <typename T>
__global__ void __launch_bounds__(128)
    sdpa_decode_combine_kernel(const SdpaParams p, const int chunk, const int nchunks, const float* ws) {
  __shared__ float weight[kMaxCombine];
  __shared__ float red[8];
  __shared__ float4 cols[128];
  pdl_wait();   // the partial results of the kernel before this one
  const int b = blockIdx.y;
  const int hl = blockIdx.x;
  const int h = p.head_begin + hl;
  const int D = p.head_dim;
  const int Hc = p.head_count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t L = decode_len(p, b);
  int nvalid = (int)((L + chunk - 1) / chunk);
  if (nvalid > nchunks) nvalid = nchunks;
  const int64_t slot0 = ((int64_t)b * Hc + hl) * nchunks;
  const float2* ml = reinterpret_cast<const float2*>(ws + (int64_t)p.batch * Hc * nchunks * D) + slot0;

  float M = -INFINITY;
  for (int c = tid; c < nvalid; c += 128) M = fmaxf(M, ml[c].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  if (lane == 0) red[warp] = M;
  __syncthreads();
  M = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));

  const int vecs = D / 4, groups = 128 / vecs;      // D = 64, 128, 256: 8, 4, 2 groups of splits
  const int grp = tid / vecs, d4 = tid - grp * vecs;
  const float4* rows = reinterpret_cast<const float4*>(ws + slot0 * D) + d4;
  float lsum = 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int c0 = 0; c0 < nvalid; c0 += kMaxCombine) {
    const int n = min(kMaxCombine, nvalid - c0);
    if (c0 > 0) __syncthreads();
    for (int c = tid; c < n; c += 128) {
      const float2 v = ml[c0 + c];
      const float w = v.x == -INFINITY ? -1.f : softmax_exp<T>(v.x - M);   // -1: a split that saw no key
      weight[c] = w;
      if (v.x != -INFINITY) lsum = fmaf(w, v.y, lsum);
    }
    __syncthreads();
#pragma unroll 4
    for (int c = grp; c < n; c += groups) {
      const float w = weight[c];
      if (w < 0.f) continue;   // its columns are undefined; a weight that underflows to 0 still carries their NaN and Inf
      const float4 x = rows[(int64_t)(c0 + c) * vecs];
      a.x = fmaf(w, x.x, a.x); a.y = fmaf(w, x.y, a.y); a.z = fmaf(w, x.z, a.z); a.w = fmaf(w, x.w, a.w);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if (lane == 0) red[4 + warp] = lsum;
  cols[tid] = a;
  __syncthreads();
  lsum = (red[4] + red[5]) + (red[6] + red[7]);
  if (grp == 0) {
    for (int g = 1; g < groups; ++g) {
      const float4 x = cols[g * vecs + d4];
      a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
    }
    const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
    const int64_t at = b * p.os[0] + (int64_t)h * p.os[1] + d4 * 4;
    store_out<T>(p.out, at, a.x * inv, p.out_f32);
    store_out<T>(p.out, at + 1, a.y * inv, p.out_f32);
    store_out<T>(p.out, at + 2, a.z * inv, p.out_f32);
    store_out<T>(p.out, at + 3, a.w * inv, p.out_f32);
  }
  if (p.lse && tid == 0)
    p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q] = lsum > 0.f ? M + logf(lsum) : -INFINITY;
}

// The same for the slots of sdpa_decode_stream_kernel, which are found from the lengths alone, before the launch in front has ended.  W warps per
// (sequence, head), each with every W-th row (heads of 64: two rows at a time) and eight passes in flight, a lane with four columns.  With
// CTAs of a head each, whose threads met three times, it took 3 to 9 us behind its launch, and sequences of equal lengths were faster by
// chunks; us, equal lengths / from 1 / 16 of the keys, chunks or clusters -> that -> this:
//   D 128: 128 items, 2048 keys 27.9 -> 29.6 -> 28.4 / 22.1 -> 20.0 -> 18.9, in a pool 28.5 -> 30.8 -> 29.8 / 26.5 -> 20.9 -> 20.2; 65 items, 3729 keys
//          24.9 -> 27.2 -> 25.2 / 20.1 -> 20.4 -> 18.3; 512 items, 500 keys 35.6 -> 29.3 -> 28.2 / 25.1 -> 20.5 -> 19.6
//   D 64:  406 items, 885 keys 23.2 -> 24.8 -> 23.7 / 17.5 -> 17.7 -> 16.6; 368 items, 336 keys 14.4 -> 17.3 -> 13.8 / 11.8 -> 14.1 -> 11.0;
//          402 items of eight heads, 1712 keys 42.8 -> 44.2 -> 37.9 / 29.1 -> 31.1 -> 24.5
template <typename T, int D, int W>
__global__ void __launch_bounds__(128) sdpa_decode_stream_merge_kernel(const SdpaParams p, const int shares, const float* ws) {
  constexpr int kLanes = D / 4, kRows = 32 / kLanes, kHop = W * kRows, kFlight = 8;   // lanes of a row, rows of a warp's pass, rows to its next
  __shared__ float4 cols[W][W > 1 ? kLanes : 1];
  __shared__ float sums[W];
  static_assert(W == 1 || W == 4, "a head per warp, or per CTA");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.y, Hc = p.head_count;
  const int hl = W == 1 ? (int)blockIdx.x * 4 + warp : (int)blockIdx.x;
  __shared__ int all_of[4], before_of[4], steps_of_b;
  int before = 0, all = 0;
  for (int i = threadIdx.x; i < p.batch; i += 128) {   // (every thread of all CTAs reads the same few lines of L2: once each)
    const int n = stream_steps_early(p, i);
    all += n;
    if (i < b) before += n;
    if (i == b) steps_of_b = n;
  }
  all = __reduce_add_sync(0xffffffffu, all);
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) {
    all_of[warp] = all;
    before_of[warp] = before;
  }
  __syncthreads();
  before = before_of[0] + before_of[1] + before_of[2] + before_of[3];
  const StreamPlan plan = stream_plan(all_of[0] + all_of[1] + all_of[2] + all_of[3], shares);
  const int steps = steps_of_b, first = before / plan.per;
  const int n = steps > 0 && hl < Hc ? (before + steps - 1) / plan.per - first + 1 : 0;
  const int64_t slot0 = (int64_t)(first + b) * Hc + hl;
  const float2* ml = reinterpret_cast<const float2*>(ws + (int64_t)(shares + p.batch) * Hc * D) + slot0;
  const float4* rows = reinterpret_cast<const float4*>(ws + slot0 * D) + lane % kLanes;
  const int c0 = (W == 1 ? 0 : warp * kRows) + lane / kLanes;
  // The partial results.  No trigger: what follows in a decode step is the projection of the next tokens, whose CTAs would be put where these leave room
  // first, two to an SM while others stay idle (36 sequences of up to 838 keys, Hq60 / Hkv15, with the projection 106 -> 126 us).
  pdl_wait();

  float4 x[kFlight];
  float2 v[kFlight];
  auto request = [&](int c) {
#pragma unroll
    for (int i = 0; i < kFlight; ++i) {
      const int at = c + i * kHop;
      x[i] = at < n ? rows[(int64_t)at * Hc * kLanes] : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i] = at < n ? ml[(int64_t)at * Hc] : make_float2(-INFINITY, 0.f);
    }
  };
  request(c0);
  float M = -INFINITY;
  for (int c = lane; c < n; c += 32) M = fmaxf(M, ml[(int64_t)c * Hc].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  float l = 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int c = c0; c < n; c += kFlight * kHop) {
    if (c > c0) request(c);
#pragma unroll
    for (int i = 0; i < kFlight; ++i) {
      if (v[i].x == -INFINITY) continue;   // saw no key: its columns are undefined; a weight that underflows to 0 still carries NaN and Inf
      const float w = softmax_exp<T>(v[i].x - M);
      l = fmaf(w, v[i].y, l);
      a.x = fmaf(w, x[i].x, a.x); a.y = fmaf(w, x[i].y, a.y); a.z = fmaf(w, x[i].z, a.z); a.w = fmaf(w, x[i].w, a.w);
    }
  }
  if constexpr (kRows == 2) {
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    a.x += __shfl_xor_sync(0xffffffffu, a.x, 16);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, 16);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, 16);
    a.w += __shfl_xor_sync(0xffffffffu, a.w, 16);
  }
  if constexpr (W > 1) {
    if (lane < kLanes) cols[warp][lane] = a;
    if (lane == 0) sums[warp] = l;
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int i = 1; i < W; ++i) {
      const float4 y = cols[i][lane % kLanes];
      a.x += y.x; a.y += y.y; a.z += y.z; a.w += y.w;
      l += sums[i];
    }
  }
  if (hl >= Hc || lane >= kLanes) return;
  const int h = p.head_begin + hl;
  const float inv = l > 0.f ? 1.f / l : 0.f;
  const int64_t at = b * p.os[0] + (int64_t)h * p.os[1] + lane * 4;
  store_out<T>(p.out, at, a.x * inv, p.out_f32);
  store_out<T>(p.out, at + 1, a.y * inv, p.out_f32);
  store_out<T>(p.out, at + 2, a.z * inv, p.out_f32);
  store_out<T>(p.out, at + 3, a.w * inv, p.out_f32);
  if (p.lse && lane == 0) p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q] = l > 0.f ? M + logf(l) : -INFINITY;
}

template <typename T, int D, int GT>
cudaError_t launch_partial(const SdpaParams& p, const DecodePlan& plan, float* ws, int merge, cudaStream_t stream) {
  const unsigned heads_y = (unsigned)((p.head_count / p.group) * ((p.group + GT - 1) / GT)), parts = (unsigned)(plan.nchunks * plan.cluster);
  const bool head_fast = p.ks[1] < p.ks[2] && parts <= 65535;
  const dim3 grid = head_fast ? dim3(heads_y, parts, (unsigned)p.batch) : dim3(parts, heads_y, (unsigned)p.batch);
  const dim3 shape = head_fast ? dim3(1, (unsigned)plan.cluster) : dim3((unsigned)plan.cluster);
  auto kern = head_fast ? (p.block_table ? sdpa_decode_partial_kernel<T, D, GT, true, true> : sdpa_decode_partial_kernel<T, D, GT, false, true>)
                        : (p.block_table ? sdpa_decode_partial_kernel<T, D, GT, true, false> : sdpa_decode_partial_kernel<T, D, GT, false, false>);
  return launch_dependent_cluster(kern, grid, kDecWarps * 32, shape, 0, stream, p, plan.chunk, plan.nchunks, ws, merge, plan.cluster);
}

template <typename T, int D, bool NH16, int CTAS>
cudaError_t launch_gqa_ctas(const SdpaParams& p, const DecodePlan& plan, float* ws, int merge, cudaStream_t stream) {
  const unsigned kvheads = (unsigned)(p.head_count / p.group), parts = (unsigned)(plan.nchunks * plan.cluster);
  const bool head_fast = p.ks[1] < p.ks[2] && parts <= 65535;
  const dim3 grid = head_fast ? dim3(kvheads, parts, (unsigned)p.batch) : dim3(parts, kvheads, (unsigned)p.batch);
  const dim3 shape = head_fast ? dim3(1, (unsigned)plan.cluster) : dim3((unsigned)plan.cluster);
  auto kern = head_fast ? (p.block_table ? sdpa_decode_gqa_ring_kernel<T, D, NH16, true, true, CTAS> : sdpa_decode_gqa_ring_kernel<T, D, NH16, false, true, CTAS>)
                        : (p.block_table ? sdpa_decode_gqa_ring_kernel<T, D, NH16, true, false, CTAS> : sdpa_decode_gqa_ring_kernel<T, D, NH16, false, false, CTAS>);
  constexpr int smem = RingCfg<D>::kSmemBytes;
  if (smem > 48 * 1024) {   // (below, a launch needs no leave for it)
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return launch_dependent_cluster(kern, grid, kDecWarps * 32, shape, smem, stream, p, plan.chunk, plan.nchunks, ws, merge, plan.cluster);
}

// Heads of 64 with more than eight query heads in a pool: three CTAs an SM take nine registers from each, 0.6 to 1.2 us where two an SM are all
// there is (113 items of 508 keys, 16 heads 13.1 -> 14.3), and save a second wave where there are more (100 items of 500 keys, 9 heads 16.1 -> 9.4).
template <typename T, int D, bool NH16>
cudaError_t launch_gqa(const SdpaParams& p, const DecodePlan& plan, float* ws, int merge, cudaStream_t stream) {
  if constexpr (NH16 && D == 64) {
    const int64_t ctas = (int64_t)(p.head_count / p.group) * p.batch * plan.nchunks * plan.cluster;
    if (ctas <= 2 * 148) return launch_gqa_ctas<T, D, NH16, 2>(p, plan, ws, merge, stream);
  }
  return launch_gqa_ctas<T, D, NH16, kRingCtas<D>>(p, plan, ws, merge, stream);
}

// 16-bit inputs with up to 16 query heads per KV head (plain multi-head attention included: the padding rows of the MMA
// tile cost nothing on an HBM-bound kernel): the tensor-core kernel with the cp.async ring.
bool takes_ring(const SdpaParams& p, int dtype) {
  return dtype != AIDN_F32 && (p.head_dim == 64 || p.head_dim == 128) && p.group <= 16;
}

template <typename T, int D>
cudaError_t launch_partial_g(const SdpaParams& p, const DecodePlan& plan, float* ws, int merge, cudaStream_t stream) {
  if constexpr (sizeof(T) == 2 && (D == 64 || D == 128)) {
    if (p.group <= 8) return launch_gqa<T, D, false>(p, plan, ws, merge, stream);
    if (p.group <= 16) return launch_gqa<T, D, true>(p, plan, ws, merge, stream);
  }
  if (p.group == 1) return launch_partial<T, D, 1>(p, plan, ws, merge, stream);
  if (p.group == 2) return launch_partial<T, D, 2>(p, plan, ws, merge, stream);
  if (p.group <= 4) return launch_partial<T, D, 4>(p, plan, ws, merge, stream);
  return launch_partial<T, D, 8>(p, plan, ws, merge, stream);
}

constexpr int stream_ctas(int head_dim, int num_sms) { return (head_dim == 128 ? kRingCtas<128> : kRingCtas<64>) * num_sms; }   // resident at once

template <typename T, int D, bool NH16>
cudaError_t launch_stream(const SdpaParams& p, const DecodePlan& plan, float* ws, cudaStream_t stream) {
  auto kern = p.block_table ? sdpa_decode_stream_kernel<T, D, NH16, true> : sdpa_decode_stream_kernel<T, D, NH16, false>;
  constexpr int smem = RingCfg<D>::kSmemBytes;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int kv_heads = p.head_count / p.group, shares = plan.stream_ctas * kDecWarps / kv_heads;
  e = launch_dependent(kern, dim3((unsigned)plan.stream_ctas), kDecWarps * 32, smem, stream, p, ws, kv_heads, shares);
  if (e != cudaSuccess) return e;
  // A CTA per output row while these are few (us at 128 / 65 items above with a warp each: 29.0 / 25.2 for 28.4 / 25.2; D 64, 406 rows 23.7 for 23.9).
  const unsigned heads = (unsigned)p.head_count, batch = (unsigned)p.batch;
  if ((int64_t)heads * batch <= (D == 128 ? 1024 : 256))
    return launch_dependent(sdpa_decode_stream_merge_kernel<T, D, 4>, dim3(heads, batch), 128, 0, stream, p, shares, static_cast<const float*>(ws));
  return launch_dependent(sdpa_decode_stream_merge_kernel<T, D, 1>, dim3((heads + 3) / 4, batch), 128, 0, stream, p, shares, static_cast<const float*>(ws));
}

template <typename T>
cudaError_t launch_decode_t(const SdpaParams& p, const DecodePlan& plan, float* ws, cudaStream_t stream, int* launches) {
  const int nchunks = plan.nchunks;
  const int merge = plan.cluster > 1 ? (nchunks == 1 ? kMergeCluster : kMergeBoth) : (nchunks == 1 ? kMergeDirect : kMergeWorkspace);
  cudaError_t e;
  if constexpr (sizeof(T) == 2) {
    if (plan.stream_ctas > 0) {
      *launches = 2;
      if (p.head_dim == 64) return p.group <= 8 ? launch_stream<T, 64, false>(p, plan, ws, stream) : launch_stream<T, 64, true>(p, plan, ws, stream);
      return p.group <= 8 ? launch_stream<T, 128, false>(p, plan, ws, stream) : launch_stream<T, 128, true>(p, plan, ws, stream);
    }
  }
  switch (p.head_dim) {
    case 64: e = launch_partial_g<T, 64>(p, plan, ws, merge, stream); break;
    case 128: e = launch_partial_g<T, 128>(p, plan, ws, merge, stream); break;
    case 256:
      if constexpr (sizeof(T) == 2) {
        e = launch_partial_g<T, 256>(p, plan, ws, merge, stream);
        break;
      }
      return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
  *launches = 1;
  if (e != cudaSuccess || nchunks == 1) return e;
  dim3 grid((unsigned)p.head_count, (unsigned)p.batch);
  *launches = 2;
  // chunk 1: with clusters every slot is written (m = -inf where there was no key)
  return launch_dependent(sdpa_decode_combine_kernel<T>, grid, 128, 0, stream, p, plan.cluster > 1 ? 1 : plan.chunk, nchunks, static_cast<const float*>(ws));
}


// ---- decode with library-owned static scratch ---------------------------------------------------------------
// Some callers may not allocate device memory at the point where they decode: code running inside a CUDA-graph
// capture or a real-time serving loop where cudaMalloc (which can synchronise the device) is forbidden, or a
// host whose memory budget was handed out up front.  For them the split-KV partials live in this fixed array
// instead of a caller or handle allocation.  Every GPU that loads the library holds the array until exit.
constexpr int64_t kStaticScratchFloats = 4ll * 1024 * 1024;  // 16 MiB
static __device__ __align__(256) float g_decode_static_scratch[kStaticScratchFloats];

// The array has one address per CUDA context, not per device ordinal: a process may hold the primary context and a
// context of its own making (the reference's backend creates one with cuCtxCreate) on the same GPU, and each has its
// own copy of the library's device image.  The address is therefore looked up once per context and remembered under
// the context's id (cuCtxGetId: unique for the life of the process, unlike the handle, which a later context may reuse).
constexpr int kMaxContexts = 64;
struct ScratchSlot {
  unsigned long long ctx_id;
  float* ptr;
};
ScratchSlot g_static_scratch[kMaxContexts] = {};
int g_static_scratch_used = 0;
std::mutex g_static_scratch_mutex;

typedef int (*CtxGetIdFn)(void*, unsigned long long*);   // CUresult cuCtxGetId(CUcontext, unsigned long long*)
CtxGetIdFn ctx_get_id_fn() {
  static CtxGetIdFn fn = nullptr;   // written under g_static_scratch_mutex
  if (!fn) {
    void* raw = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &raw, cudaEnableDefault, &qres) == cudaSuccess && raw &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetIdFn>(raw);
  }
  return fn;
}

// In host code the array's name is only a stand-in; the device address has to be asked for with the context that
// will run the kernel current.
cudaError_t static_scratch_address(float** out) {
  // binds the runtime to the caller's current context (or to the primary one when the thread has none)
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  unsigned long long id = 0;
  CtxGetIdFn get = ctx_get_id_fn();
  const bool have_id = get && get(nullptr, &id) == 0;   // a null context means the current one
  if (have_id)
    for (int i = 0; i < g_static_scratch_used; ++i)
      if (g_static_scratch[i].ctx_id == id) {
        *out = g_static_scratch[i].ptr;
        return cudaSuccess;
      }
  float* ptr = nullptr;
  e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_decode_static_scratch);
  if (e != cudaSuccess) return e;
  // without a context id (or with the table full) the address is simply looked up again on every call
  if (have_id && g_static_scratch_used < kMaxContexts) g_static_scratch[g_static_scratch_used++] = {id, ptr};
  *out = ptr;
  return cudaSuccess;
}

}  // namespace

bool decode_supported(int dtype, int head_dim) {
  if (head_dim == 64 || head_dim == 128) return true;
  return head_dim == 256 && dtype != AIDN_F32;
}

// Clusters save the merge kernel and its trip through L2, and cut each sequence by its own length; but CTAs that wait for one
// another hold their place, so they pay only while all of a launch's CTAs are resident at once, and while a CTA's keys do not last
// longer than chunks would that keep every SM busy to the end.  Measured with 200 to 16384 keys, and with lengths from 1 / 16 of the keys
// to all of them; us, chunks with a merge kernel / clusters of (n), bf16 heads of 128 unless stated:
//   * Clusters of 8 are all resident up to 0.89 of the places (heads of 64, three CTAs an SM: 0.86, not at 0.88), of 4 up to 0.93, of 2 up
//     to all; then the largest that is.  500 keys: 33 items 7.9 / 7.4 (8), 34 items 8.2 / 10.4 (8) / 7.3 (4); 69 items 14.3 / 8.8 (4),
//     74 items 14.4 / 13.5 (4) / 9.6 (2); heads of 64, 49 items, 305 keys 6.6 / 8.5 (8).
//   * Keys of a CTA: 28 items, 16384 keys 55 / 42 (8); 50 items, 8192 keys 48 / 41 (4), with lengths 32 / 36; heads of 64, 56 items,
//     4096 keys 16.2 / 15.5 (4) at 1024 a CTA, 8192 keys 31 / 34, 3000 keys with lengths 12.4 / 13.2; 103 items, 7254 keys 41 / 33 (4);
//     48 items, 7733 keys 29 / 21 (8).
//   * Several clusters of 8 and the merge kernel where one would have more than 400 keys a CTA: 4 items of heads of 64, 4096 keys
//     8.3 / 8.5 (2 x 8) / 7.9 (8 x 8); 2 items, 16384 keys 30 / 12.7 (8 x 8).
//   * Two CTAs each, at most one wave: 128 items, 2048 keys 37 / 29, with lengths 23.3 / 22.9; 80 items, 2048 keys 27.6 / 23.8, with
//     lengths 19.2 / 21.5.  Two waves pay where the second is nearly full: 256 items, 2048 keys 55 / 51, with lengths 36.2 / 37.5;
//     180 items 44.6 / 49.2, 500 keys 20.4 / 20.4; 149 items, 500 keys 23.2 / 17.6.
//   * fp32 on the FP32 units is bound by them, not by bytes, and chunks spread better (heads of 64): 4 items, 700 keys 6.9 / 6.6 (8),
//     2000 keys 8.1 / 11.7 (8) / 7.9 (8 x 8), 8000 keys 13.6 / 12.3 (8 x 8); 32 items, 2000 keys 16.6 / 15.0 (8), 4000 keys 22.5 / 25.4 (8) /
//     20.2 (2 x 8); 64 items, 8000 keys 53 / 53 (8), 4000 keys 33.6 / 29.2; 74 items are not all resident: 8000 keys 59 / 94 (8); 22 items,
//     4786 keys 21 / 19 (3 x 8); of four heads: 43 items, 3402 keys 39 / 50 (8), 2 items, 695 keys 10.2 / 11.3, 10 items, 464 keys 10.4 / 9.6.
//     Few items with 1000 to 1280 keys lose 0.1 to 1.4 us of 7 to 8 on the GPU; the second launch would cost the host of a token more.
// 1100 shapes drawn from 1 to 300 items and 150 to 16384 keys: 0.83 of the chunks' time for 16-bit tensors, 0.91 for fp32, and more than
// 8 % above it in 12 of them (clusters without these limits: 0.86, 0.95 and 111, the longest 1.6 times the chunks' time).
void decode_plan_clusters(const SdpaParams& p, int dtype, int num_sms, DecodePlan* plan) {
  const bool ring = takes_ring(p, dtype), lengths = p.kv_len != nullptr, wide = p.head_dim == 128;
  if (!ring && (dtype != AIDN_F32 || p.group > 8)) return;
  const int64_t items = (int64_t)p.batch * (p.head_count / p.group), keys = p.seq_kv;
  const int64_t room = (ring ? (wide ? kRingCtas<128> : kRingCtas<64>) : 4) * (int64_t)num_sms;   // CTAs that are resident at once
  int64_t cluster = 1, clusters = 1;
  if (!ring) {
    const int64_t eights = (wide ? room : room * 94 / 100) / (8 * items);   // clusters of 8 per item
    const int64_t little = p.group == 1 ? (lengths ? 768 : 1280) : 480, some = (lengths ? 28 : 80) * items / p.group;
    if (eights < 1) return;
    if (wide ? keys <= 512 : (keys <= little || keys <= some || (items >= 60 * p.group && !lengths))) cluster = 8;
    else if (wide) return;
    else if (eights >= 8) { if (keys >= 3200) cluster = clusters = 8; }
    else if (!lengths && eights >= 2 && keys >= 1600 && (eights >= 4 || keys <= 8192)) cluster = 8, clusters = eights;
  } else {
    const int64_t eights = room * (wide ? 90 : 87) / 100 / (8 * items), fours = room * 95 / 100 / (4 * items);
    int64_t most = lengths ? (wide ? 1024 : 700) : (wide || 40 * items >= 3 * room ? 2048 : 1300);   // keys of a CTA
    if (eights >= 1) {
      if ((eights >= 8 && keys > 3072) || (eights >= 4 && keys > 3500) || keys > (lengths ? 5600 : 5000)) clusters = eights >= 8 ? 8 : (eights > 4 ? 4 : eights);
      if (clusters > plan->nchunks) clusters = plan->nchunks;
      if (clusters > 1 && lengths) most = wide ? 768 : 384;
      if (keys <= 8 * clusters * most) cluster = 8;
    } else if (fours >= 1) {
      if (!lengths) most = 20 * items >= 3 * room ? 4096 : (wide ? 2048 : 1024);   // (three places in five are taken)
      if (keys <= 4 * most) cluster = 4;
    } else if (2 * items <= room) {
      if (keys <= (lengths && 8 * items < 3 * room ? 1024 : 2048)) cluster = 2;
    } else if (items <= room) {
      if (4 * items >= 3 * room) { if (keys <= (lengths ? 1024 : 2048)) cluster = 2; }
      else if (keys <= 512 && (!lengths || 5 * items < 3 * room)) cluster = 2;
    }
  }
  if (cluster == 1) return;
  if (clusters > plan->nchunks) clusters = plan->nchunks;   // never more workspace
  plan->cluster = (int)cluster;
  plan->nchunks = (int)clusters;
}

// Equal shares of all keys pay where the plan without them has no clusters, two waves of them, or CTAs with so many keys that the longest
// sequence's run on alone.  Below 48 items, and with less than that to a CTA, the second launch and the way to the first keys (10 us)
// weigh more.  Lengths from 1 / 8 or 1 / 16 of the keys to all of them, us before -> after; items are (sequence, KV head) pairs:
//   pays       128 items, 2048 keys, D 128 26.9 -> 21.5; 72 items, 1584 keys 16.3 -> 14.5; 182 items, 750 keys 19.6 -> 16.8; 228 items, 1117
//              keys 28.6 -> 24.9; 266 items, 353 keys 16.9 -> 13.8; 222 items, 4234 keys 59 -> 51; 512 items, 4096 keys 115 -> 106;
//              heads of 64: 60 items, 3549 keys 15.6 -> 14.6; 405 items, 483 keys 13.7 -> 12.5; 128 items, 2048 keys 18.5 -> 15.9
//   does not   96 items, 618 keys 10.2 -> 11.2; 110 items, 241 keys 7.2 -> 11.0; 54 items, 1395 keys 16.1 -> 17.9; 24 items, 5170 keys 15.3 ->
//              16.9; 20 items, 8626 keys 21.5 -> 23.1; heads of 64: 190 items, 814 keys 11.0 -> 15.4; 84 items, 2711 keys 15.9 -> 19.4
// (these with a merge that took 1 to 7 us longer, sdpa_decode_stream_merge_kernel).  The host does not see the lengths: sequences that are all as
// long as the tensor take 0.82 of the time before in pools and 0.94 otherwise (137 shapes), and up to 1.06 where one wave of clusters of two had
// been (144 items of 1795 keys 27.3 -> 28.9, 128 of 2048 in a pool 28.5 -> 29.9).
int64_t decode_stream_bytes(const SdpaParams& p, int dtype, int num_sms, const DecodePlan& chunks, int* ctas) {
  *ctas = 0;
  if (!takes_ring(p, dtype) || chunks.nchunks <= 1) return 0;
  const int kv_heads = p.head_count / p.group, n = stream_ctas(p.head_dim, num_sms);
  const int64_t items = (int64_t)p.batch * kv_heads, steps = (p.seq_kv + 15) / 16;
  if (items < 48 || items * steps > 0x3fffffff || p.batch > 256 || kv_heads > n * kDecWarps) return 0;
  // Less than 2.5 steps to a warp, 3.3 with heads of 64: 174 items of up to 128 keys, D 128, 9.6 -> 11.4 us, 255 of 134 in a pool, with its projection, 22.7 -> 25.4; heads of
  // 64: 418 items of 166 keys 10.6 -> 14.0, 402 of 218 10.4 -> 11.5, 225 of 143 22.8 -> 27.2.  Above that 216 items of 239 keys, D 128, 28.1 -> 26.7, 336 of 274, D 64, 34.9 -> 33.6.
  if (items * steps * 6 < (int64_t)n * kDecWarps * (p.head_dim == 64 ? 20 : 15)) return 0;
  // Long launches stream at the memory's rate either way, and chunks read larger pieces: of 400 MB, or with the heads of a token side by
  // side of 1.2 GB, on (2048 items of 4096 keys 382 -> 405 us; in a pool 512 items of 4096 keys, 1.07 GB, 115 -> 106).
  if (items * p.seq_kv * p.head_dim * 4 > (p.block_table || p.ks[1] < p.ks[2] ? 1200000000 : 400000000)) return 0;
  SdpaParams q = p;
  const int32_t some_lengths = 0;
  q.kv_len = &some_lengths;   // (only whether there are any)
  DecodePlan plan = chunks;
  decode_plan_clusters(q, dtype, num_sms, &plan);
  const int64_t parts = (int64_t)plan.cluster * plan.nchunks;
  if (plan.cluster > 1 && items * parts <= n && p.seq_kv / parts * p.head_dim < 100000) return 0;
  // A fifth more CTAs than are resident at once, in clusters of two, few keys and heads of 64: the rest finds places soon enough (224 to 264 items of up to 450 to 512 keys
  // 9.8 to 11.4 us, in shares 12.0; in a pool 12.2 and 15.2).
  if (plan.cluster == 2 && p.head_dim == 64 && p.seq_kv <= 512 && items * parts * 5 <= (int64_t)n * 6) return 0;
  *ctas = n;
  return ((int64_t)(n * kDecWarps / kv_heads) + p.batch) * kv_heads * p.group * (p.head_dim + 2) * (int64_t)sizeof(float);
}

cudaError_t launch_decode(const SdpaParams& p, int dtype, const DecodePlan& plan, float* workspace, cudaStream_t stream, int* launches) {
  switch (dtype) {
    case AIDN_F32: return launch_decode_t<float>(p, plan, workspace, stream, launches);
    case AIDN_F16: return launch_decode_t<__half>(p, plan, workspace, stream, launches);
    default: return launch_decode_t<__nv_bfloat16>(p, plan, workspace, stream, launches);
  }
}

}  // namespace aidn

namespace aidn {

int64_t decode_static_scratch_bytes() { return kStaticScratchFloats * (int64_t)sizeof(float); }

// Same two kernels as launch_decode, with the partials in the library's static array.  `need_bytes` is what the
// shape requires; the caller has already checked it against decode_static_scratch_bytes().
cudaError_t launch_decode_static(const SdpaParams& p, int dtype, const DecodePlan& plan, cudaStream_t stream, int* launches) {
  float* scratch = nullptr;
  cudaError_t e = static_scratch_address(&scratch);
  if (e != cudaSuccess) return e;
  return launch_decode(p, dtype, plan, scratch, stream, launches);
}

}  // namespace aidn
