"""Explicit masks of the 16-bit tcgen05 kernels (csrc/mask_tile.cuh) where their tiles can go wrong: rows off 16 bytes and off 4, fewer rows or
keys than a tile, masks that are broadcast or transposed, head pairs and single heads, poison around what the mask may be read from."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import AIDN_DT, compare, gen
from tests.test_gpu_backward import _check, _fwd_bwd

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Sq, Sk, D): keys in whole tiles of 64, in whole 16-byte rows, neither, and in whole 4-byte rows; rows up to one past a tile
SHAPES = [(2, 2, 2, 128, 192, 64), (1, 4, 2, 129, 208, 128), (2, 3, 1, 33, 97, 64), (1, 2, 1, 257, 450, 128), (3, 2, 2, 31, 523, 64), (2, 2, 2, 70, 100, 64),
          (1, 3, 3, 129, 120, 128)]
KINDS = ["bytes", "floats", "bias"]
LAYOUTS = ["dense", "offset", "one_row", "one_key", "transposed"]


def _mask(shape, kind, layout, seed):
    """The mask as the kernel gets it (a view between rows of poison) and as numpy broadcasts it."""
    B, Hq, _, Sq, Sk, _ = shape
    rng = np.random.default_rng(seed)
    rows, keys = (1 if layout == "one_row" else Sq), (1 if layout == "one_key" else Sk)
    if kind == "bias":
        m = rng.standard_normal((B, Hq, rows, keys)).astype(np.float32)
        if keys > 1:
            m[..., 5::11] = -np.inf
    else:
        m = (rng.random((B, Hq, rows, keys)) < 0.7).astype(np.uint8 if kind == "bytes" else np.float32)
        m[..., 0] = 1                                               # every row of the first key's causal triangle sees something
    at = m.swapaxes(2, 3) if layout == "transposed" else m
    pad = 3 if layout == "offset" else 0                            # elements: rows and base off every alignment
    flat = torch.full((at.size + 64 + pad * at.shape[2] * B * Hq,), float("nan") if kind != "bytes" else 1, dtype=torch.uint8 if kind == "bytes" else torch.float32,
                      device="cuda")
    view = flat[16 + pad: 16 + pad + B * Hq * at.shape[2] * (at.shape[3] + pad)].view(B, Hq, at.shape[2], at.shape[3] + pad)[..., : at.shape[3]]
    view.copy_(torch.from_numpy(np.ascontiguousarray(at)))
    return view.swapaxes(2, 3) if layout == "transposed" else view, m


def _strides(t, full):
    return tuple(0 if (t.shape[a] == 1 and full[a] != 1) else t.stride(a) for a in range(4))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("causal", [False, True])
def test_masks_forward_and_backward(shape, kind, layout, causal):
    B, Hq, Hkv, Sq, Sk, D = shape
    dtype = "bf16" if Sk % 2 else "f16"
    q, qf = gen((B, Hq, Sq, D), dtype, 1)
    k, kf = gen((B, Hkv, Sk, D), dtype, 2)
    v, vf = gen((B, Hkv, Sk, D), dtype, 3)
    dout, dof = gen((B, Hq, Sq, D), "f32", 4, scale=1.0)
    dev, m = _mask(shape, kind, layout, 5)
    mask_kind = {"bytes": N.MASK_KEEP_U8, "floats": N.MASK_KEEP_F32, "bias": N.MASK_ADD_F32}[kind]
    full = np.ascontiguousarray(np.broadcast_to(m, (B, Hq, Sq, Sk)))
    okw = dict(mask=full, mask_kind=mask_kind, causal=causal, causal_offset=Sk - Sq if causal else 0)
    out = torch.full((B, Hq, Sq, D), float("nan"), device="cuda")
    h = N.Handle(device=0, qkv_dtype=AIDN_DT[dtype], out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv, causal=causal,
                 causal_bottom_right=True, mask_kind=mask_kind)
    stream = torch.cuda.current_stream().cuda_stream
    h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk, stream=stream, mask=dev.data_ptr(),
             mask_stride=_strides(dev, (B, Hq, Sq, Sk)))
    h.poll(stream)
    h.close()
    ref = O.sdpa(qf, kf, vf, **okw)
    compare(out, ref[0] if isinstance(ref, tuple) else ref, dtype, f"{shape} {kind} {layout}")
    got = _fwd_bwd(q, k, v, dout, dtype=dtype, causal=causal, bottom_right=True, mask=dev, mask_kind=mask_kind)
    want = O.sdpa_backward(qf, kf, vf, dof, causal=causal, causal_offset=okw["causal_offset"], **({"bias": full} if kind == "bias" else {"keep": full}))
    for x, y, name in zip(got, want, ("dQ", "dK", "dV")):
        _check(x, y, dtype, f"{name} {shape} {kind} {layout}")


@pytest.mark.parametrize("shape", SHAPES[1:4])
@pytest.mark.parametrize("kind", KINDS)
def test_masks_with_softcap_and_lengths(shape, kind):
    """Behind a softcap, with sequences shorter than the mask, whose rows beyond them are NaN."""
    B, Hq, Hkv, Sq, Sk, D = shape
    q, qf = gen((B, Hq, Sq, D), "bf16", 1)
    k, kf = gen((B, Hkv, Sk, D), "bf16", 2)
    v, vf = gen((B, Hkv, Sk, D), "bf16", 3)
    lens = np.array([Sk - 1, Sk // 2, 1][:B], np.int32)
    dev, m = _mask(shape, kind, "offset", 6)
    if kind == "bias":
        for b in range(B):
            dev[b, ..., int(lens[b]):] = float("nan")
    mask_kind = {"bytes": N.MASK_KEEP_U8, "floats": N.MASK_KEEP_F32, "bias": N.MASK_ADD_F32}[kind]
    out = torch.full((B, Hq, Sq, D), float("nan"), device="cuda")
    h = N.Handle(device=0, qkv_dtype=N.BF16, out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv, mask_kind=mask_kind, softcap=20.0)
    stream = torch.cuda.current_stream().cuda_stream
    kl = torch.from_numpy(lens).cuda()
    h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk, stream=stream, mask=dev.data_ptr(),
             mask_stride=_strides(dev, (B, Hq, Sq, Sk)), kv_len=kl.data_ptr())
    h.poll(stream)
    h.close()
    ref = O.sdpa(qf, kf, vf, mask=m, mask_kind=mask_kind, softcap=20.0, kv_len=lens)
    compare(out, ref[0] if isinstance(ref, tuple) else ref, "bf16", f"{shape} {kind}")


@pytest.mark.parametrize("shape", [(1, 3, 3, 129, 120, 64), (2, 2, 1, 300, 333, 32), (2, 2, 2, 200, 450, 128)])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("softcap", [0.0, 20.0])
def test_masks_fp32(shape, kind, layout, softcap):
    """fp32 calls: floats through the row warps' tiles, one row of them and bytes as bits, whole tiles of rows and the last ones."""
    B, Hq, Hkv, Sq, Sk, D = shape
    (q, qf), (k, kf), (v, vf) = (gen((B, H, S, D), "f32", i, 1.0) for i, (H, S) in enumerate(((Hq, Sq), (Hkv, Sk), (Hkv, Sk))))
    dev, m = _mask(shape, kind, layout, 7)
    mask_kind = {"bytes": N.MASK_KEEP_U8, "floats": N.MASK_KEEP_F32, "bias": N.MASK_ADD_F32}[kind]
    out = torch.full((B, Hq, Sq, D), float("nan"), device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    with N.Handle(device=0, qkv_dtype=N.F32, out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv, mask_kind=mask_kind, softcap=softcap) as h:
        h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk, stream=stream, mask=dev.data_ptr(),
                 mask_stride=_strides(dev, (B, Hq, Sq, Sk)))
        h.poll(stream)
    ref = O.sdpa(qf, kf, vf, mask=m, mask_kind=mask_kind, softcap=softcap)
    compare(out, ref[0] if isinstance(ref, tuple) else ref, "f32", f"{shape} {kind} {layout} {softcap}")
