// Attention forward in fp32 arithmetic on register-tiled packed multiply-adds: the path for the 16-bit head sizes that the tcgen05
// kernel does not take and for fp32 tensors whose calls are too small for the three-term products of csrc/sdpa_f32_sm100.cu
// (head_dim <= 128, contiguous K / V, 16-byte rows).
//
// Two things bound it: the FP32 pipe (128 multiply-adds per SM and cycle) and shared memory, which hands 128 bytes per
// cycle to the registers whether lanes read the same words or not.  Each warp owns 16 query rows and walks tiles of 32
// keys on its own; lane (ty, tx) of the 4 x 8 lanes holds a 4 x 4 block of logits and a 4 x (head_dim / 8) block of the
// output.  8-row blocks would halve the shared-memory reads, but take 255 registers and with them half of the warps:
// B1 H8 S512 D64 took 42 us that way against 27 (62 for the kernel of sdpa_generic.cu).  Sixteen warps leave 128 registers:
// at head_dim 64 the fp32 instantiations spill up to 56 bytes (mask values), the 16-bit ones, with a tile in registers, 172.
//   S = Q K^T   both operands have d contiguous, so the two halves of `fma.rn.f32x2` sum the even and the odd d of one
//               logit: no operand has to be duplicated
//   O += P V    the pair runs along d; P goes through shared memory transposed (rows contiguous) and is duplicated in
//               registers
// Row sums stay per lane until the end; a row's maximum needs three shuffles per tile.
//
// The CTA is WR row warps by WK key warps: the key warps take the key tiles in turn and merge their (max, sum, output)
// through shared memory at the end.  One K and one V buffer: K(s + 1) lands under P V of step s, V(s + 1) under the scores
// of step s + 1 (cp.async for fp32; through registers for 16-bit types, which are widened on the way).
#include "common.cuh"
#include "ffma2.cuh"

namespace aidn {
namespace {

constexpr int kRowsW = 16;     // query rows of a warp
constexpr int kR = 4;          // of a lane: ty + 4 i
constexpr int kKeysW = 32;     // keys of a warp's tile
constexpr int kTileSpan = 64;  // anything above both tile extents (clamp of the tile bounds)
constexpr int kPPitch = 20;    // floats per key of the stored probabilities: 16 rows, padded

template <int DP, int WR, int WK>
struct FCfg {
  static constexpr int kThreads = WR * WK * 32;
  static constexpr int kPitch = DP + 4;                       // floats per row: 16-byte reads of 8 rows are conflict-free
  static constexpr int kStageKeys = WK * kKeysW;
  static constexpr int kQFloats = WR * kRowsW * kPitch;
  static constexpr int kTileFloats = kStageKeys * kPitch;     // K, and as many again of V
  static constexpr int kPFloats = WR * WK * kKeysW * kPPitch;
  static constexpr size_t kSmem = sizeof(float) * (kQFloats + 2 * kTileFloats + kPFloats);
  static constexpr int kMinCtas = DP > 64 ? 1 : 512 / kThreads;   // 16 warps per SM within 128 registers
};

template <typename T, int DP, int WR, int WK, bool PLAIN>
__global__ void __launch_bounds__(WR* WK * 32, FCfg<DP, WR, WK>::kMinCtas) sdpa_f32_kernel(const SdpaParams p, const int vec_out) {
  using C = FCfg<DP, WR, WK>;
  constexpr int NV = DP / 32;                 // 16-byte groups of output columns per lane
  constexpr int N = Chunk16<T>::N;            // elements per 16-byte chunk
  constexpr int CH = DP / N;                  // chunks per row
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* Kbuf = Qs + C::kQFloats;             // [kStageKeys][kPitch]
  float* Vbuf = Kbuf + C::kTileFloats;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wr = warp % WR, wk = warp / WR;
  const int ty = lane >> 3, tx = lane & 7;
  float* Ps = Vbuf + C::kTileFloats + warp * kKeysW * kPPitch;

  const int b = blockIdx.z, h = p.head_begin + blockIdx.y, kvh = h / p.group;
  // under a causal mask the last rows see the most keys: start them first
  const int64_t tile = p.causal ? (int64_t)gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const int64_t cta_row0 = tile * (WR * kRowsW);
  const int64_t row0 = cta_row0 + wr * kRowsW;
  const int D = p.head_dim;
  const T* qb = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const T* kb = static_cast<const T*>(p.k) + b * p.ks[0] + kvh * p.ks[1];
  const T* vb = static_cast<const T*>(p.v) + b * p.vs[0] + kvh * p.vs[1];

  const int64_t kv_limit = kv_limit_of(p, b);
  auto visible_end = [&](int64_t last_row) {   // keys [0, end) can be visible to rows <= last_row
    int64_t end = kv_limit;
    if (p.causal) {
      if (last_row > p.seq_q - 1) last_row = p.seq_q - 1;
      const int64_t c = last_row + p.causal_offset + 1;
      if (c < end) end = c;
    }
    return end;
  };
  const int64_t kend = visible_end(cta_row0 + WR * kRowsW - 1);
  const int64_t warp_end = row0 < p.seq_q ? visible_end(row0 + kRowsW - 1) : 0;
  const int64_t first_end = visible_end(row0);   // keys below it are visible to every row of the warp

  // One K or V tile: keys past kend (padding beyond kv_len, the causal future) and columns past head_dim are zeros and
  // are not read - their probability is 0, and 0 * (NaN or Inf left in unused memory) would be NaN.  A thread copies one
  // column chunk of every RP-th row.
  constexpr bool kAsync = sizeof(T) == 4;
  constexpr int RP = C::kThreads / CH, kPer = (C::kStageKeys + RP - 1) / RP;
  const int cp_row = tid / CH, cp_col = (tid - cp_row * CH) * N;
  const bool cp_any = cp_row < RP && cp_col < D;
  uint4 reg[kAsync ? 1 : kPer];
  auto fetch = [&](const T* base, int64_t stride, float* buf, int64_t s) {
    const int64_t left = kend - s * C::kStageKeys;   // keys of the tile that are read
    const T* src = base + (s * C::kStageKeys + cp_row) * stride + cp_col;
    float* dst = buf + cp_row * C::kPitch + cp_col;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int j = cp_row + e * RP;
      const bool ok = cp_any && j < left;
      if constexpr (kAsync) {
        if (cp_row < RP && (C::kStageKeys % RP == 0 || j < C::kStageKeys)) cp_async16_f(dst, ok ? src : base, ok);
      } else {
        reg[e] = ok && j < C::kStageKeys ? *reinterpret_cast<const uint4*>(src) : make_uint4(0, 0, 0, 0);
      }
      src += RP * stride;
      dst += RP * C::kPitch;
    }
    if constexpr (kAsync) cp_async_commit_f();
  };
  auto land = [&](float* buf) {   // fp32: the copy has landed; 16-bit types: widen the fetched registers into the buffer
    if constexpr (kAsync) {
      cp_async_wait_f<0>();
    } else {
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const int j = cp_row + e * RP;
        if (cp_row < RP && (C::kStageKeys % RP == 0 || j < C::kStageKeys)) store_chunk<T>(buf + j * C::kPitch + cp_col, reg[e]);
      }
    }
  };

  const int64_t steps = kend > 0 ? (kend + C::kStageKeys - 1) / C::kStageKeys : 0;
  if (steps > 0) fetch(kb, p.ks[2], Kbuf, 0);
  for (int idx = tid; idx < WR * kRowsW * CH; idx += C::kThreads) {
    const int r = idx / CH, d = (idx - r * CH) * N;
    const int64_t row = cta_row0 + r;
    const bool ok = row < p.seq_q && d < D;
    store_chunk<T>(Qs + r * C::kPitch + d, ok ? *reinterpret_cast<const uint4*>(qb + row * p.qs[2] + d) : make_uint4(0, 0, 0, 0));
  }

  float m[kR], l[kR];
  uint64_t acc[kR][NV][2];
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n) acc[i][n][0] = acc[i][n][1] = 0;
  }
  const int64_t mask_bh = b * p.mask_stride[0] + h * p.mask_stride[1];
  const float* qrow = Qs + (wr * kRowsW + ty) * C::kPitch;
  auto row = [&](int i) { return ty + 4 * i; };   // the lane's rows and keys within the warp's tile
  auto key = [&](int k) { return tx + 8 * k; };

  if (steps > 0) land(Kbuf);
  __syncthreads();
  for (int64_t s = 0; s < steps; ++s) {
    fetch(vb, p.vs[2], Vbuf, s);
    const int64_t j0 = s * C::kStageKeys + wk * kKeysW;
    const bool live = j0 < warp_end;   // (warp-uniform) something of this tile is visible to the warp's rows
    if (live) {
      const float* krow = Kbuf + (wk * kKeysW + tx) * C::kPitch;
      const TileBounds tb(p, row0, j0, kv_limit, kTileSpan);
      auto seen = [&](int i, int k) { return tb.seen(row(i), key(k)); };
      MaskBlock<kR, 4> mask;
      if (!PLAIN && p.mask_kind != AIDN_MASK_NONE)
        fetch_mask(p, mask_bh + row0 * p.mask_stride[2] + j0 * p.mask_stride[3], row, key, seen, mask);

      float sc[kR][4];
      {
        uint64_t s2[kR][4];
#pragma unroll
        for (int i = 0; i < kR; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k) s2[i][k] = 0;
#pragma unroll 2
        for (int d = 0; d < DP; d += 4) {
          Pair2 k4[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) k4[k] = lds_pairs(krow + 8 * k * C::kPitch + d);
#pragma unroll
          for (int i = 0; i < kR; ++i) {
            const Pair2 q4 = lds_pairs(qrow + 4 * i * C::kPitch + d);
#pragma unroll
            for (int k = 0; k < 4; ++k) s2[i][k] = fma2(q4.a, k4[k].a, s2[i][k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) s2[i][k] = fma2(q4.b, k4[k].b, s2[i][k]);
          }
        }
#pragma unroll
        for (int i = 0; i < kR; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k) sc[i][k] = sum2(s2[i][k]) * p.scale;
      }
      if (!PLAIN) {
#pragma unroll
        for (int i = 0; i < kR; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k) sc[i][k] = finish_logit_with(p, sc[i][k], seen(i, k), mask.v[i][k]);
      } else if (j0 + kKeysW > first_end) {   // a tile on the diagonal or at the end of the keys
#pragma unroll
        for (int i = 0; i < kR; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (!seen(i, k)) sc[i][k] = -INFINITY;
      }

#pragma unroll
      for (int i = 0; i < kR; ++i) {
        float mt = fmaxf(fmaxf(sc[i][0], sc[i][1]), fmaxf(sc[i][2], sc[i][3]));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
        const float m_new = fmaxf(m[i], mt);
        const float corr = m[i] == -INFINITY ? 0.f : softmax_exp<T>(m[i] - m_new);
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sc[i][k] = sc[i][k] == -INFINITY ? 0.f : softmax_exp<T>(sc[i][k] - m_new);
          sum += sc[i][k];
        }
        l[i] = fmaf(l[i], corr, sum);
        m[i] = m_new;
        const uint64_t c2 = pack2(corr, corr);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          acc[i][n][0] = mul2(acc[i][n][0], c2);
          acc[i][n][1] = mul2(acc[i][n][1], c2);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)   // slot 4 ty + i holds row ty + 4 i
        *reinterpret_cast<float4*>(Ps + key(k) * kPPitch + ty * 4) = make_float4(sc[0][k], sc[1][k], sc[2][k], sc[3][k]);
    }
    land(Vbuf);
    __syncthreads();   // V(s) is complete, and every warp has left K(s)
    if (s + 1 < steps) fetch(kb, p.ks[2], Kbuf, s + 1);
    if (live) {
      const float* prow = Ps + ty * 4;
      const float* vcol = Vbuf + wk * kKeysW * C::kPitch + tx * 4;
#pragma unroll 4
      for (int j = 0; j < kKeysW; ++j) {
        const float4 pa = *reinterpret_cast<const float4*>(prow + j * kPPitch);
        const float pj[kR] = {pa.x, pa.y, pa.z, pa.w};
        Pair2 v4[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) v4[n] = lds_pairs(vcol + j * C::kPitch + 32 * n);
#pragma unroll
        for (int i = 0; i < kR; ++i) {
          const uint64_t p2 = pack2(pj[i], pj[i]);
#pragma unroll
          for (int n = 0; n < NV; ++n) {
            acc[i][n][0] = fma2(p2, v4[n].a, acc[i][n][0]);
            acc[i][n][1] = fma2(p2, v4[n].b, acc[i][n][1]);
          }
        }
      }
    }
    if (s + 1 < steps) land(Kbuf);
    __syncthreads();   // K(s + 1) is complete, and every warp has left V(s)
  }

#pragma unroll
  for (int i = 0; i < kR; ++i)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);

  if constexpr (WK > 1) {   // merge the key warps of each row warp: group 0 reads what the others left
    constexpr int MP = DP + 4;
    if (wk > 0) {
      float* mine = Kbuf + ((wk - 1) * WR + wr) * kRowsW * MP;
#pragma unroll
      for (int i = 0; i < kR; ++i) {
        float* at = mine + row(i) * MP;
#pragma unroll
        for (int n = 0; n < NV; ++n) *reinterpret_cast<ulonglong2*>(at + tx * 4 + 32 * n) = make_ulonglong2(acc[i][n][0], acc[i][n][1]);
        if (tx == 0) { at[DP] = m[i]; at[DP + 1] = l[i]; }
      }
    }
    __syncthreads();
    if (wk > 0) return;
#pragma unroll
    for (int g = 1; g < WK; ++g) {
      const float* theirs = Kbuf + ((g - 1) * WR + wr) * kRowsW * MP;
#pragma unroll
      for (int i = 0; i < kR; ++i) {
        const float* at = theirs + row(i) * MP;
        const float mg = at[DP], lg = at[DP + 1];
        const float m_new = fmaxf(m[i], mg);
        const float f0 = m[i] == -INFINITY ? 0.f : softmax_exp<T>(m[i] - m_new);
        const float f1 = mg == -INFINITY ? 0.f : softmax_exp<T>(mg - m_new);
        m[i] = m_new;
        l[i] = fmaf(lg, f1, l[i] * f0);
        const uint64_t a2 = pack2(f0, f0), b2 = pack2(f1, f1);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const Pair2 t = lds_pairs(at + tx * 4 + 32 * n);
          acc[i][n][0] = fma2(t.a, b2, mul2(acc[i][n][0], a2));
          acc[i][n][1] = fma2(t.b, b2, mul2(acc[i][n][1], a2));
        }
      }
    }
  }

#pragma unroll
  for (int i = 0; i < kR; ++i) {
    if (row0 + row(i) >= p.seq_q) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const int64_t obase = b * p.os[0] + h * p.os[1] + (row0 + row(i)) * p.os[2];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int d = tx * 4 + 32 * n;
      if (d >= D) continue;
      const float2 lo = unpack2(acc[i][n][0]), hi = unpack2(acc[i][n][1]);
      const float o4[4] = {lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv};
      if (vec_out && p.out_f32) {
        *reinterpret_cast<float4*>(static_cast<float*>(p.out) + obase + d) = make_float4(o4[0], o4[1], o4[2], o4[3]);
      } else if (vec_out && sizeof(T) == 2) {
        T t[4] = {from_float<T>(o4[0]), from_float<T>(o4[1]), from_float<T>(o4[2]), from_float<T>(o4[3])};
        *reinterpret_cast<uint2*>(static_cast<T*>(p.out) + obase + d) = *reinterpret_cast<const uint2*>(t);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) store_out<T>(p.out, obase + d + e, o4[e], p.out_f32);
      }
    }
    if (p.lse && tx == 0)
      p.lse[((int64_t)b * p.num_q_heads + h) * p.seq_q + row0 + row(i)] = l[i] > 0.f ? m[i] + logf(l[i]) : -INFINITY;
  }
}

template <typename T, int DP, int WR, int WK>
cudaError_t launch_cfg(const SdpaParams& p, int vec_out, cudaStream_t stream) {
  using C = FCfg<DP, WR, WK>;
  static_assert(C::kSmem <= 227 * 1024 && C::kMinCtas * (C::kSmem + 1024) <= 228 * 1024, "shared memory of the resident CTAs");
  static_assert((WK - 1) * WR * kRowsW * (DP + 4) <= 2 * C::kTileFloats + C::kPFloats, "the merge reuses the tiles");
  const bool plain = p.mask_kind == AIDN_MASK_NONE && !(p.softcap > 0.f);
  auto kern = plain ? sdpa_f32_kernel<T, DP, WR, WK, true> : sdpa_f32_kernel<T, DP, WR, WK, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((p.seq_q + WR * kRowsW - 1) / (WR * kRowsW)), (unsigned)p.head_count, (unsigned)p.batch);
  kern<<<grid, C::kThreads, C::kSmem, stream>>>(p, vec_out);
  return cudaGetLastError();
}

template <typename T, int DP>
cudaError_t launch_dp(const SdpaParams& p, cudaStream_t stream) {
  const int osz = p.out_f32 ? 4 : (int)sizeof(T);
  bool vec = reinterpret_cast<uintptr_t>(p.out) % (4 * osz) == 0;
  for (int i = 0; i < 3; ++i) vec = vec && p.os[i] % 4 == 0;
  // Row warps against key warps.  An SM's time is its share of the row tiles (the busiest SM counts) times the key tiles,
  // rounded up to what its key warps take at once; the most row warps of equal cost share each K / V tile best.
  // With lengths the CTAs are unequal, half of a full one on average for the host that cannot see them: what counts is the
  // average SM and the tail of one CTA, with the merge of its key warps on top, and smaller CTAs win.  34 shapes with lengths
  // spread from 1 / 8 of the keys: at most 15 % from the best of the three, the rule above up to 2.8 times (B2 H4 S2048 D64 337 us
  // with 8 x 1, 154 with 4 x 4, 176 with 2 x 8, causal 331, 150 and 118; B8 H16 S197 D32 35, 35 and 56).
  const int64_t heads = (int64_t)p.head_count * p.batch, key_tiles = (p.seq_kv + kKeysW - 1) / kKeysW;
  auto cost = [&](int wr, int wk) {
    const int64_t ctas = (p.seq_q + wr * kRowsW - 1) / (wr * kRowsW) * heads;
    const int64_t steps = (key_tiles + wk - 1) / wk * wk;
    if (p.kv_len) return (ctas * 10 + 4 * 148) * (wr * steps + wk);   // (ctas / 148 + 0.4) CTAs, in whole numbers
    return (ctas + 147) / 148 * wr * steps;
  };
  if constexpr (DP <= 64) {
    const int64_t c8 = cost(8, 1), c4 = cost(4, 4), c2 = cost(2, 8);
    if (c8 <= c4 && c8 <= c2) return launch_cfg<T, DP, 8, 1>(p, vec, stream);
    if (c4 <= c2) return launch_cfg<T, DP, 4, 4>(p, vec, stream);
    return launch_cfg<T, DP, 2, 8>(p, vec, stream);
  } else {
    // Above head_dim 64 one CTA fills an SM and 2 x 4 reads every K / V tile four times as often: with lengths it needs a margin
    // (B3 H16 S700 D80, costs 1.06 to 1: 177 us with 8 x 1, 221 with 2 x 4; B16 H8 100 x 1500 D128, 1.24 to 1: 387 and 257).
    if (cost(8, 1) * 20 <= cost(2, 4) * (p.kv_len ? 23 : 20)) return launch_cfg<T, DP, 8, 1>(p, vec, stream);
    return launch_cfg<T, DP, 2, 4>(p, vec, stream);
  }
}

template <typename T>
cudaError_t launch_type(const SdpaParams& p, cudaStream_t stream) {
  if (p.head_dim <= 32) return launch_dp<T, 32>(p, stream);
  if (p.head_dim <= 64) return launch_dp<T, 64>(p, stream);
  if (p.head_dim <= 96) return launch_dp<T, 96>(p, stream);
  return launch_dp<T, 128>(p, stream);
}

}  // namespace

// Everything that writes the attention weights, reads a block table, has rows that are not 16-byte aligned or a head
// size above 128 stays on sdpa_generic_kernel.
bool f32_supported(const SdpaParams& p, int dtype) {
  const int esz = dtype == AIDN_F32 ? 4 : 2;
  return !p.weights && !p.block_table && p.head_dim <= 128 && (p.head_dim * esz) % 16 == 0 && rows_aligned16(p.q, p.qs, esz) &&
         rows_aligned16(p.k, p.ks, esz) && rows_aligned16(p.v, p.vs, esz);
}

cudaError_t launch_f32(const SdpaParams& p, int dtype, cudaStream_t stream) {
  if (f32_sm100_supported(p, dtype)) return launch_f32_sm100(p, stream);
  switch (dtype) {
    case AIDN_F32: return launch_type<float>(p, stream);
    case AIDN_F16: return launch_type<__half>(p, stream);
    default: return launch_type<__nv_bfloat16>(p, stream);
  }
}

}  // namespace aidn
