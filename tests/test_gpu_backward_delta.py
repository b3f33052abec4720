"""The row sums of dO * O in front of the backward kernels: 16-byte vectors where the rows allow it, scalar elsewhere, fp32 and
16-bit O / dO, rows that end inside a warp's steps, and a dO that starts off a 16-byte boundary.  Seen through dQ, dK, dV of
the whole call against float64, at the bar of the other backward tests - of 1 at least, the size of the dP and delta whose
difference dQ and dK are made of (with one visible key it is 0: a dO rounded to 16 bits on one side only leaves 3e-3 there)."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200.backend import CudaBackend, GpuBuffer
from oracle import sdpa_oracle as O

from tests._harness import TORCH_DT, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,out", [("bf16", "f32"), ("bf16", "bf16"), ("f16", "f16"), ("f32", "f32")])
@pytest.mark.parametrize("D,S", [(64, 1), (64, 63), (64, 130), (128, 15), (128, 129), (96, 33)])
@pytest.mark.parametrize("shift", [0, 1])
def test_delta(dtype, out, D, S, shift):
    B, H = 2, 3
    n = B * H * S * D
    (q, qf), (k, kf), (v, vf) = (gen((B, H, S, D), dtype, i) for i in (1, 2, 3))
    g, gf = gen((B, H, S, D), out, 4, 1.0)
    flat = torch.zeros(n + 8, dtype=TORCH_DT[out], device="cuda")
    flat[shift:shift + n] = g.reshape(-1)
    backend = CudaBackend(0)
    buf = lambda t: GpuBuffer(t.reshape(-1))
    o, stats = backend.AllocateBuffer(n, TORCH_DT[out]), backend.AllocateBuffer(B * H * S)
    dq, dk, dv = (backend.AllocateBuffer(n) for _ in range(3))
    backend.FlashAttentionV2(buf(q), buf(k), buf(v), o, stats, B, H, S, S, D, D ** -0.5, True)
    backend.FlashAttentionBackward(GpuBuffer(flat[shift:shift + n]), buf(q), buf(k), buf(v), o, stats, dq, dk, dv, B, H, S, S, D,
                                   D ** -0.5, True)
    for got, want in zip((dq, dk, dv), O.sdpa_backward(qf, kf, vf, gf, causal=True, causal_offset=0)[:3]):
        x = got.tensor.cpu().numpy().reshape(want.shape)
        assert np.isfinite(x).all()
        assert np.abs(x - want).max() <= (2e-5 if dtype == "f32" else 2e-2) * max(np.abs(want).max(), 1.0)
    backend.Dispose()
