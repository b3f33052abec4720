"""The register-tiled fp32 kernels (csrc/sdpa_f32.cu, sdpa_backward_f32.cu, the fp32 GEMM of proj_gemm_generic.cu) at the
sizes where they can go wrong: one row or key more or less than a warp's tile, remainders of the key split, padded head
sizes, every CTA shape, every mask kind, strided K / V, and what they hand to the general kernels."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import compare, compare_lse, gen, run_gpu

pytestmark = pytest.mark.gpu


# (B, Hq, Hkv, Sq, Sk, D): the CTA shapes follow from rows x heads against the SMs (few: keys split over 8 or 4 warps)
SHAPES = [(1, 2, 1, 1, 31, 32), (1, 2, 2, 16, 32, 64), (1, 4, 2, 17, 33, 64), (2, 3, 3, 127, 257, 64), (1, 8, 8, 129, 255, 36),
          (2, 16, 4, 300, 300, 64), (8, 16, 16, 197, 197, 32), (4, 48, 48, 130, 65, 64), (1, 2, 2, 65, 129, 128), (2, 40, 40, 129, 97, 128),
          (1, 3, 3, 70, 64, 80), (3, 40, 20, 130, 70, 96)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("variant", ["plain", "causal", "lengths", "keep", "bias_softcap"])
def test_forward_f32(shape, variant):
    B, Hq, Hkv, Sq, Sk, D = shape
    q, qf = gen((B, Hq, Sq, D), "f32", 1, 1.0)
    k, kf = gen((B, Hkv, Sk, D), "f32", 2, 1.0)
    v, vf = gen((B, Hkv, Sk, D), "f32", 3, 1.0)
    kw, okw = {}, {}
    rng = np.random.default_rng(4)
    if variant == "causal":
        kw, okw = dict(causal=True, bottom_right=False, causal_offset=Sk - Sq - 3), dict(causal=True, causal_offset=Sk - Sq - 3)
    elif variant == "lengths":
        lens = rng.integers(0, Sk + 1, B).astype(np.int32)
        lens[0] = Sk
        for b in range(B):                                    # what lies beyond a sequence's keys must never matter
            k[b, :, lens[b]:], v[b, :, lens[b]:] = float("nan"), float("inf")
        kw, okw = dict(kv_len=torch.from_numpy(lens).cuda()), dict(kv_len=lens)
    elif variant == "keep":
        keep = (rng.random((1, Hq, Sq, Sk)) < 0.7).astype(np.uint8)
        keep[:, :, Sq // 2] = 0                               # a row that sees nothing
        kw, okw = dict(mask=torch.from_numpy(keep).cuda(), mask_kind=N.MASK_KEEP_U8), dict(mask=keep, mask_kind=O.MASK_KEEP_U8)
    elif variant == "bias_softcap":
        bias = rng.standard_normal((B, 1, Sq, Sk)).astype(np.float32)
        bias[..., ::7] = -np.inf
        bias[..., 1] = np.finfo(np.float32).min
        kw = dict(mask=torch.from_numpy(bias).cuda(), mask_kind=N.MASK_ADD_F32, softcap=20.0)
        okw = dict(mask=bias, mask_kind=O.MASK_ADD_F32, softcap=20.0)
    out, lse, _ = run_gpu(q, k, v, dtype="f32", want_lse=True, path=N.PATH_GENERIC, **kw)
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, **okw)
    compare(out, ref, "f32", f"{shape} {variant}")
    compare_lse(lse, ref_lse, "f32", f"{shape} {variant}")


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("out", ["f32", "same"])
def test_forward_16bit_head_size(dtype, out):
    """16-bit tensors of a head size that the tensor-core kernel does not take keep fp32 probabilities."""
    q, qf = gen((2, 6, 150, 96), dtype, 1)
    k, kf = gen((2, 3, 210, 96), dtype, 2)
    v, vf = gen((2, 3, 210, 96), dtype, 3)
    got, _, info = run_gpu(q, k, v, dtype=dtype, out_dtype="f32" if out == "f32" else dtype, causal=True)
    assert info["path"] == N.PATH_GENERIC
    ref = O.sdpa(qf, kf, vf, causal=True, causal_offset=60)
    if out == "f32":   # no rounding but the inputs', which the reference sees too; ex2.approx: 2^-22 relative per weight
        assert np.abs(got.cpu().numpy() - ref).max() <= 4e-6 * np.abs(ref).max()
    else:
        compare(got, ref, dtype, "head size 96")


def test_forward_strided_and_unaligned_rows():
    """K / V as [S, H, D] slices are read in place; rows that start off a 16-byte boundary take the general kernel.  Both
    give what dense tensors give."""
    B, H, S, D = 2, 4, 90, 64
    q, qf = gen((B, H, S, D), "f32", 1, 1.0)
    kv, kvf = gen((B, S, 2, H, D), "f32", 2, 1.0)
    ref = O.sdpa(qf, kvf[:, :, 0].transpose(0, 2, 1, 3), kvf[:, :, 1].transpose(0, 2, 1, 3))
    stride = (S * 2 * H * D, D, 2 * H * D)
    for shift in (0, 1):
        flat = torch.zeros(kv.numel() + 4, device="cuda")
        flat[shift:shift + kv.numel()] = kv.reshape(-1)
        base = flat[shift:]
        out, _, _ = run_gpu(q, base, base[H * D:], dtype="f32", k_stride=stride, v_stride=stride, seq_kv=S, num_kv_heads=H)
        compare(out, ref, "f32", f"shift {shift}")


@pytest.mark.parametrize("B,S,H,D", [(1, 5, 3, 4), (1, 63, 2, 10), (2, 64, 5, 36), (3, 43, 4, 32), (1, 2500, 16, 32), (9, 130, 33, 20)])
def test_projection_f32(B, S, H, D):
    """The fp32 projections around their 64 / 128-row tiles: one row more or less, widths that end inside a 64-column tile
    or a 32-deep slice, head sizes that a group of four columns straddles.  A dot product of n terms of unit variance
    scaled by 1 / sqrt(n) and rounded n times: 4 x 2^-24 x sqrt(n) / 2 on values of magnitude up to 5; two in a row."""
    from aidotnet.tensors_b200.backend import CudaBackend, GpuBuffer
    rng = np.random.default_rng(S)
    dm = H * D
    x = rng.standard_normal((B, S, dm), dtype=np.float32)
    ws = [(rng.standard_normal((dm, dm)) / np.sqrt(dm)).astype(np.float32) for _ in range(4)]
    backend = CudaBackend(0)
    buf = lambda a: GpuBuffer(torch.from_numpy(a).cuda().reshape(-1))
    out = backend.AllocateBuffer(B * S * dm)
    backend.MultiHeadAttentionForward(buf(x), *[buf(w) for w in ws], out, B, S, dm, H, exact=True)
    xd = torch.from_numpy(x).cuda().double()
    wd = [torch.from_numpy(w).cuda().double() for w in ws]
    q, k, v = ((xd @ w).view(B, S, H, D).transpose(1, 2) for w in wd[:3])
    p = torch.softmax(q @ k.transpose(2, 3) / np.sqrt(D), -1)
    ref = ((p @ v).transpose(1, 2).reshape(B, S, dm) @ wd[3]).cpu().numpy()
    err = np.abs(out.tensor.cpu().numpy().reshape(ref.shape) - ref).max()
    assert err <= 8 * 2.0 ** -24 * np.sqrt(dm) * max(1.0, np.abs(ref).max()), err


BWD_SHAPES = [(1, 2, 1, 1, 1, 64), (1, 2, 2, 31, 33, 32), (1, 4, 2, 64, 97, 64), (2, 12, 6, 127, 65, 36), (8, 16, 16, 65, 64, 64),
              (3, 20, 10, 130, 129, 32), (1, 3, 3, 70, 40, 128), (2, 30, 30, 129, 130, 128), (1, 6, 2, 95, 160, 96)]


@pytest.mark.parametrize("shape", BWD_SHAPES)
@pytest.mark.parametrize("variant", ["plain", "causal", "keep_lengths", "bias"])
def test_backward_f32(shape, variant):
    """dQ, dK, dV against float64.  Each is a sum of n <= 160 products of fp32 values, through a probability and a dS that
    are off by the rounding of two more such sums: 16 x 2^-24 x sqrt(n) of the largest value."""
    from tests.test_gpu_backward import _fwd_bwd
    B, Hq, Hkv, Sq, Sk, D = shape
    ts = [gen(s, "f32", i + 1, 1.0) for i, s in enumerate([(B, Hq, Sq, D), (B, Hkv, Sk, D), (B, Hkv, Sk, D), (B, Hq, Sq, D)])]
    (q, qf), (k, kf), (v, vf), (g, gf) = ts
    rng = np.random.default_rng(5)
    kw, okw = {}, {}
    if variant == "causal":
        kw = okw = dict(causal=True, causal_offset=Sk - Sq + 2)
    elif variant == "keep_lengths":
        keep = (rng.random((B, 1, Sq, Sk)) < 0.8).astype(np.uint8)
        lens = rng.integers(1, Sk + 1, B).astype(np.int32)
        kw, okw = dict(mask=torch.from_numpy(keep).cuda(), mask_kind=N.MASK_KEEP_U8, kv_len=lens), dict(keep=keep, kv_len=lens)
    elif variant == "bias":
        bias = rng.standard_normal((1, Hq, Sq, Sk)).astype(np.float32)
        kw, okw = dict(mask=torch.from_numpy(bias).cuda(), mask_kind=N.MASK_ADD_F32), dict(bias=bias)
    got = _fwd_bwd(q, k, v, g, dtype="f32", **kw)
    want = O.sdpa_backward(qf, kf, vf, gf, **okw)[:3]
    for x, y, name in zip(got, want, ("dQ", "dK", "dV")):
        x = x.cpu().numpy()
        assert np.isfinite(x).all(), name
        assert np.abs(x - y).max() <= 16 * 2.0 ** -24 * np.sqrt(max(Sq, Sk, D)) * max(1.0, np.abs(y).max()), (name, np.abs(x - y).max())
    again = _fwd_bwd(q, k, v, g, dtype="f32", **kw)
    assert all(torch.equal(x, y) for x, y in zip(got, again))
