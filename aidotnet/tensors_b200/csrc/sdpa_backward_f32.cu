// Attention backward of fp32 tensors on register-tiled packed multiply-adds: dQ and dK / dV as two launches of one kernel
// (head_dim <= 128, contiguous K / V, 16-byte rows; the formulas and the mask rules are those of sdpa_backward.cu).  Head sizes up
// to 64 go to the three-term products of csrc/sdpa_backward_f32_sm100.cu where the sequences are long enough for them.
//
// A warp keeps 16 rows of one sequence ("stationary") and walks 32-row tiles of the other past them:
//   KEYS = true  (dK, dV): X = its K rows, Y = its V rows; a tile is U = Q rows, W = dO rows of one query head of the group.
//   KEYS = false (dQ):     X = its Q rows, Y = its dO rows; a tile is U = K rows, W = V rows.
//   S = X U^T    dP = Y W^T    acc0 += dS U    KEYS: acc1 += P W      with P = exp(S scale - lse), dS = P (dP - delta)
// Lane tiling, the even / odd split of the score sums and the transposed probabilities in shared memory are those of the
// forward kernel (sdpa_f32.cu), and so are its bounds: the FP32 pipe and the shared-memory reads.  U and W are double
// buffered.  CTA = WR stationary groups x WK warps that take the streamed tiles in turn; the WK sums are added in warp
// order at the end, so every gradient is summed in a fixed order (deterministic, no atomics).
#include "common.cuh"
#include "ffma2.cuh"

namespace aidn {
namespace {

constexpr int kOwnW = 16;      // stationary rows of a warp
constexpr int kTileW = 32;     // streamed rows of a warp's tile
constexpr int kTileSpan = 64;  // anything above both tile extents (clamp of the tile bounds)
constexpr int kPPitch = 20;    // floats per streamed row of the stored probabilities: 16 own rows, padded

template <int DP, int WR, int WK>
struct BFCfg {
  static constexpr int kThreads = WR * WK * 32;
  static constexpr int kPitch = DP + 4;
  static constexpr int kStageRows = WK * kTileW;
  static constexpr int kXFloats = WR * kOwnW * kPitch;             // X, and as many again of Y
  static constexpr int kStageFloats = 2 * kStageRows * kPitch;     // U and W
  static constexpr int kPFloats = WR * WK * kTileW * kPPitch;
  static constexpr size_t kSmem = sizeof(float) * (2 * kXFloats + 2 * kStageFloats + kPFloats);
};

template <int DP, int WR, int WK, bool KEYS>
__global__ void __launch_bounds__(WR* WK * 32, 1) bwd_f32_kernel(const BwdParams bp) {
  using C = BFCfg<DP, WR, WK>;
  constexpr int NV = DP / 32, CH = DP / 4;
  const SdpaParams& p = bp.p;
  extern __shared__ __align__(16) float smem[];
  float* Xs = smem;
  float* Ys = Xs + C::kXFloats;
  float* ST = Ys + C::kXFloats;               // [2 stages][U rows, W rows][kPitch]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wr = warp % WR, wk = warp / WR;
  const int ty = lane >> 3, tx = lane & 7;
  float* Ps = ST + 2 * C::kStageFloats + warp * kTileW * kPPitch;

  const int b = blockIdx.z;
  const int kv_heads = p.head_count / p.group;
  const int hl0 = KEYS ? blockIdx.y * p.group : blockIdx.y;    // (first) query head within the shard
  const int h0 = p.head_begin + hl0, kvh = h0 / p.group;
  // under a causal mask the last query rows and the first keys have the most to do: start them first
  const int64_t tile = !KEYS && p.causal ? (int64_t)gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const int64_t cta0 = tile * (WR * kOwnW), own0 = cta0 + wr * kOwnW;
  const int D = p.head_dim;
  const int64_t kv_limit = kv_limit_of(p, b);
  const float* kb = static_cast<const float*>(p.k) + b * p.ks[0] + (int64_t)kvh * p.ks[1];
  const float* vb = static_cast<const float*>(p.v) + b * p.vs[0] + (int64_t)kvh * p.vs[1];
  const float* qb = static_cast<const float*>(p.q) + b * p.qs[0] + (int64_t)h0 * p.qs[1];
  const float* gb = static_cast<const float*>(bp.dout) + b * bp.dos[0] + (int64_t)h0 * bp.dos[1];

  // streamed rows [first, last) of one head that any of the CTA's own rows takes part with
  int64_t first = 0, last = KEYS ? p.seq_q : kv_limit;
  if (p.causal) {
    if constexpr (KEYS) {
      first = cta0 - p.causal_offset;              // query rows that see the CTA's first key
      first = first > 0 ? first / kTileW * kTileW : 0;
    } else {
      int64_t last_row = cta0 + WR * kOwnW - 1;
      if (last_row > p.seq_q - 1) last_row = p.seq_q - 1;
      if (last_row + p.causal_offset + 1 < last) last = last_row + p.causal_offset + 1;
    }
  }
  if (KEYS && cta0 >= kv_limit) last = 0;
  const int64_t own_end = KEYS ? kv_limit : p.seq_q;    // own rows past it take no part
  const int per_head = last > first ? (int)((last - first + C::kStageRows - 1) / C::kStageRows) : 0;
  const int steps = KEYS ? per_head * p.group : per_head;

  auto fetch = [&](int s) {
    float* stage = ST + (s & 1) * C::kStageFloats;
    const int g = KEYS ? s / per_head : 0;
    const int64_t base = first + (int64_t)(s - g * per_head) * C::kStageRows;
    const float* us = KEYS ? qb + (int64_t)g * p.qs[1] : kb;
    const float* ws = KEYS ? gb + (int64_t)g * bp.dos[1] : vb;
    const int64_t ustr = KEYS ? p.qs[2] : p.ks[2], wstr = KEYS ? bp.dos[2] : p.vs[2];
#pragma unroll
    for (int e = 0; e < C::kStageRows * CH / C::kThreads; ++e) {
      const int idx = tid + e * C::kThreads;
      const int j = idx / CH, d = (idx - j * CH) * 4;
      const bool ok = base + j < last && d < D;
      cp_async16_f(stage + j * C::kPitch + d, us + (ok ? (base + j) * ustr + d : 0), ok);
      cp_async16_f(stage + (C::kStageRows + j) * C::kPitch + d, ws + (ok ? (base + j) * wstr + d : 0), ok);
    }
    cp_async_commit_f();
  };

  {
    const float* xs = KEYS ? kb : qb;
    const float* ys = KEYS ? vb : gb;
    const int64_t xstr = KEYS ? p.ks[2] : p.qs[2], ystr = KEYS ? p.vs[2] : bp.dos[2];
    for (int idx = tid; idx < WR * kOwnW * CH; idx += C::kThreads) {
      const int r = idx / CH, d = (idx - r * CH) * 4;
      const bool ok = cta0 + r < own_end && d < D;
      cp_async16_f(Xs + r * C::kPitch + d, xs + (ok ? (cta0 + r) * xstr + d : 0), ok);
      cp_async16_f(Ys + r * C::kPitch + d, ys + (ok ? (cta0 + r) * ystr + d : 0), ok);
    }
    if (steps > 0) fetch(0);
  }

  auto own = [&](int i) { return ty + 4 * i; };   // the lane's own and streamed rows within the warp's tile
  auto str = [&](int k) { return tx + 8 * k; };
  float lse_own[4], delta_own[4];    // dQ: of the lane's own rows
  if constexpr (!KEYS) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool ok = own0 + own(i) < p.seq_q;
      lse_own[i] = ok ? p.lse[((int64_t)b * p.num_q_heads + h0) * p.seq_q + own0 + own(i)] : -INFINITY;
      delta_own[i] = ok ? bp.delta[((int64_t)b * p.head_count + hl0) * p.seq_q + own0 + own(i)] : 0.f;
    }
  }
  uint64_t acc0[4][NV][2], acc1[KEYS ? 4 : 1][NV][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      acc0[i][n][0] = acc0[i][n][1] = 0;
      if constexpr (KEYS) acc1[i][n][0] = acc1[i][n][1] = 0;
    }

  // 4 x 4 dot products of the lane's own rows with its streamed rows
  auto product = [&](const float* xrow, const float* urow, float (&out)[4][4]) {
    uint64_t s2[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) s2[i][k] = 0;
#pragma unroll 2
    for (int d = 0; d < DP; d += 4) {
      Pair2 u4[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) u4[k] = lds_pairs(urow + 8 * k * C::kPitch + d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const Pair2 x4 = lds_pairs(xrow + 4 * i * C::kPitch + d);
#pragma unroll
        for (int k = 0; k < 4; ++k) s2[i][k] = fma2(x4.a, u4[k].a, s2[i][k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) s2[i][k] = fma2(x4.b, u4[k].b, s2[i][k]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) out[i][k] = sum2(s2[i][k]);
  };
  // acc += w^T tile, w[i][k] = weight of streamed row k for own row i
  auto accumulate = [&](const float (&w)[4][4], const float* tile_rows, auto& acc) {
    __syncwarp();   // the buffer's previous contents have been read
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<float4*>(Ps + str(k) * kPPitch + ty * 4) = make_float4(w[0][k], w[1][k], w[2][k], w[3][k]);
    __syncwarp();
#pragma unroll 4
    for (int j = 0; j < kTileW; ++j) {
      const float4 a = *reinterpret_cast<const float4*>(Ps + j * kPPitch + ty * 4);
      const float pj[4] = {a.x, a.y, a.z, a.w};
      Pair2 v4[NV];
#pragma unroll
      for (int n = 0; n < NV; ++n) v4[n] = lds_pairs(tile_rows + j * C::kPitch + tx * 4 + 32 * n);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint64_t p2 = pack2(pj[i], pj[i]);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          acc[i][n][0] = fma2(p2, v4[n].a, acc[i][n][0]);
          acc[i][n][1] = fma2(p2, v4[n].b, acc[i][n][1]);
        }
      }
    }
  };

  for (int s = 0; s < steps; ++s) {
    cp_async_wait_f<0>();
    __syncthreads();   // the stage is complete, and every warp has left the other one
    if (s + 1 < steps) fetch(s + 1);
    const int g = KEYS ? s / per_head : 0;
    const int64_t j0 = first + (int64_t)(s - g * per_head) * C::kStageRows + wk * kTileW;
    // (warp-uniform) nothing of this tile takes part with the warp's own rows
    if (own0 >= own_end || j0 >= last) continue;
    if (p.causal) {
      if constexpr (KEYS) {
        if (j0 + kTileW - 1 + p.causal_offset < own0) continue;
      } else {
        if (own0 + kOwnW - 1 + p.causal_offset < j0) continue;
      }
    }
    const float* Us = ST + (s & 1) * C::kStageFloats + wk * kTileW * C::kPitch;
    const float* Ws = Us + C::kStageRows * C::kPitch;
    const int64_t row0 = KEYS ? j0 : own0, key0 = KEYS ? own0 : j0;
    const TileBounds tb(p, row0, key0, kv_limit, kTileSpan);
    auto rows = [&](int i) { return KEYS ? str(i) : own(i); };
    auto keys = [&](int k) { return KEYS ? own(k) : str(k); };
    MaskBlock<4, 4> mask;   // [row][key]
    if (p.mask_kind != AIDN_MASK_NONE)
      fetch_mask(p, b * p.mask_stride[0] + (h0 + g) * p.mask_stride[1] + row0 * p.mask_stride[2] + key0 * p.mask_stride[3], rows, keys,
                 [&](int i, int k) { return tb.seen(rows(i), keys(k)); }, mask);
    float lse_s[4], delta_s[4];
    if constexpr (KEYS) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = j0 + str(k) < p.seq_q;
        lse_s[k] = ok ? p.lse[((int64_t)b * p.num_q_heads + h0 + g) * p.seq_q + j0 + str(k)] : -INFINITY;
        delta_s[k] = ok ? bp.delta[((int64_t)b * p.head_count + hl0 + g) * p.seq_q + j0 + str(k)] : 0.f;
      }
    }
    float pr[4][4], ds[4][4];
    product(Xs + (wr * kOwnW + ty) * C::kPitch, Us + tx * C::kPitch, pr);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool seen = KEYS ? tb.seen(str(k), own(i)) : tb.seen(own(i), str(k));
        const float lse = KEYS ? lse_s[k] : lse_own[i];
        const float val = finish_logit_with(p, pr[i][k] * p.scale, seen, KEYS ? mask.v[k][i] : mask.v[i][k]);
        pr[i][k] = val == -INFINITY || lse == -INFINITY ? 0.f : expf(val - lse);
      }
    if constexpr (KEYS) accumulate(pr, Ws, acc1);
    product(Ys + (wr * kOwnW + ty) * C::kPitch, Ws + tx * C::kPitch, ds);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) ds[i][k] = pr[i][k] * (ds[i][k] - (KEYS ? delta_s[k] : delta_own[i]));
    accumulate(ds, Us, acc0);
  }

  if constexpr (WK > 1) {   // lane-major images of the other warps' sums: conflict-free both ways
    cp_async_wait_f<0>();
    __syncthreads();
    constexpr int kVecs = 4 * NV * (KEYS ? 2 : 1);
    ulonglong2* all = reinterpret_cast<ulonglong2*>(ST);
    if (wk > 0) {
      ulonglong2* mine = all + ((wk - 1) * WR + wr) * kVecs * 32 + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          mine[(i * NV + n) * 32] = make_ulonglong2(acc0[i][n][0], acc0[i][n][1]);
          if constexpr (KEYS) mine[(4 * NV + i * NV + n) * 32] = make_ulonglong2(acc1[i][n][0], acc1[i][n][1]);
        }
    }
    __syncthreads();
    if (wk > 0) return;
#pragma unroll
    for (int o = 1; o < WK; ++o) {
      const ulonglong2* theirs = all + ((o - 1) * WR + wr) * kVecs * 32 + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const ulonglong2 t = theirs[(i * NV + n) * 32];
          acc0[i][n][0] = add2(acc0[i][n][0], t.x);
          acc0[i][n][1] = add2(acc0[i][n][1], t.y);
          if constexpr (KEYS) {
            const ulonglong2 u = theirs[(4 * NV + i * NV + n) * 32];
            acc1[i][n][0] = add2(acc1[i][n][0], u.x);
            acc1[i][n][1] = add2(acc1[i][n][1], u.y);
          }
        }
    }
  }

  const uint64_t scale2 = pack2(p.scale, p.scale);
  const int64_t out_rows = KEYS ? p.seq_kv : p.seq_q;
  const int64_t base = KEYS ? ((int64_t)b * kv_heads + blockIdx.y) * out_rows : ((int64_t)b * p.head_count + hl0) * out_rows;
  float* out0 = KEYS ? bp.dk : bp.dq;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (own0 + own(i) >= out_rows) continue;
    const int64_t at = (base + own0 + own(i)) * D;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int d = tx * 4 + 32 * n;
      if (d >= D) continue;
      *reinterpret_cast<ulonglong2*>(out0 + at + d) = make_ulonglong2(mul2(acc0[i][n][0], scale2), mul2(acc0[i][n][1], scale2));
      if constexpr (KEYS) *reinterpret_cast<ulonglong2*>(bp.dv + at + d) = make_ulonglong2(acc1[i][n][0], acc1[i][n][1]);
    }
  }
}

template <int DP, int WR, int WK, bool KEYS>
cudaError_t launch_one(const BwdParams& bp, cudaStream_t stream) {
  using C = BFCfg<DP, WR, WK>;
  static_assert(C::kSmem <= 227 * 1024, "shared memory of one CTA");
  static_assert(C::kStageRows * DP / 4 % C::kThreads == 0, "whole chunks per thread");
  static_assert((WK - 1) * WR * 4 * (DP / 32) * 2 * 32 * 16 <= (int)sizeof(float) * 2 * C::kStageFloats, "the merge reuses the stages");
  const SdpaParams& p = bp.p;
  auto kern = bwd_f32_kernel<DP, WR, WK, KEYS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
  if (e != cudaSuccess) return e;
  const int64_t rows = KEYS ? p.seq_kv : p.seq_q;
  dim3 grid((unsigned)((rows + WR * kOwnW - 1) / (WR * kOwnW)), (unsigned)(KEYS ? p.head_count / p.group : p.head_count), (unsigned)p.batch);
  kern<<<grid, C::kThreads, C::kSmem, stream>>>(bp);
  return cudaGetLastError();
}

template <int DP, bool KEYS>
cudaError_t launch_dir(const BwdParams& bp, cudaStream_t stream) {
  // Four stationary groups, and as many warps that share them as registers (168 up to head_dim 64, with 4 to 24 bytes
  // spilled; 255 above) and shared memory allow - sixteen warps of 128 registers spill more and are 2 us slower for dQ on
  // B2 H8 S509 D64; half the stationary rows when four groups leave a good part of the SMs without a CTA.  Both sides
  // measured (whole backward, CTAs of 64 rows, four groups / two, us): D 64 S 512: 48 CTAs 141 / 84, 112 143 / 156, 128 144 / 156,
  // 144 145 / 156; D 128 104 CTAs 245 / 322, 128 246 / 323.  Above one wave two groups can be ahead again: D 64 160 CTAs 241 / 219.
  const int64_t rows = KEYS ? bp.p.seq_kv : bp.p.seq_q;
  const int64_t heads = (int64_t)(KEYS ? bp.p.head_count / bp.p.group : bp.p.head_count) * bp.p.batch;
  const bool wide = (rows + 4 * kOwnW - 1) / (4 * kOwnW) * heads >= 112;
  if constexpr (DP <= 64) {
    if (wide) return launch_one<DP, 4, 3, KEYS>(bp, stream);
    return launch_one<DP, 2, 4, KEYS>(bp, stream);
  } else {
    if (wide) return launch_one<DP, 4, 2, KEYS>(bp, stream);
    return launch_one<DP, 2, 2, KEYS>(bp, stream);
  }
}

template <int DP>
cudaError_t launch_dp(const BwdParams& bp, cudaStream_t stream) {
  const cudaError_t e = launch_dir<DP, false>(bp, stream);
  return e != cudaSuccess ? e : launch_dir<DP, true>(bp, stream);
}

}  // namespace

bool backward_f32_supported(const BwdParams& bp, int dtype) {
  const SdpaParams& p = bp.p;
  const uintptr_t outs = reinterpret_cast<uintptr_t>(bp.dq) | reinterpret_cast<uintptr_t>(bp.dk) | reinterpret_cast<uintptr_t>(bp.dv);
  return dtype == AIDN_F32 && !p.block_table && p.head_dim <= 128 && p.head_dim % 4 == 0 && rows_aligned16(p.q, p.qs, 4) &&
         rows_aligned16(p.k, p.ks, 4) && rows_aligned16(p.v, p.vs, 4) && rows_aligned16(bp.dout, bp.dos, 4) && outs % 16 == 0 &&
         (p.seq_q + kTileW) * p.group / kTileW < 0x7fffffffll && p.seq_kv / kTileW < 0x7fffffffll;
}

cudaError_t launch_backward_f32(const BwdParams& bp, cudaStream_t stream) {
  if (backward_f32_sm100_supported(bp)) return launch_backward_f32_sm100(bp, stream);
  if (bp.p.head_dim <= 32) return launch_dp<32>(bp, stream);
  if (bp.p.head_dim <= 64) return launch_dp<64>(bp, stream);
  if (bp.p.head_dim <= 96) return launch_dp<96>(bp, stream);
  return launch_dp<128>(bp, stream);
}

}  // namespace aidn
