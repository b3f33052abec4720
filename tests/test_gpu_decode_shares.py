"""Decode launches whose warps share all keys evenly (csrc/sdpa_decode.cu, sdpa_decode_stream_kernel): shares that end inside, at and beyond
the ends of sequences, sequences without keys at either end of the batch and between, every instantiation, pools, head shards; and
the line of decode_stream_bytes, told by the workspace that a launch asks for."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import compare, compare_lse, gen, run_gpu
from tests.test_gpu_paged import _launch_paged, _pool, _tables

pytestmark = pytest.mark.gpu


def _lens(kind, B, Sk):
    rng = np.random.default_rng(3)
    if kind == "ragged":
        lens = rng.integers(0, Sk + 1, B)
        lens[0], lens[1], lens[2], lens[-1] = 0, 1, Sk, 0
    elif kind == "one":
        lens = np.zeros(B, np.int64)
        lens[B // 2] = Sk - 3
    elif kind == "none":
        lens = np.zeros(B, np.int64)
    else:
        lens = np.full(B, Sk)
    return lens.astype(np.int32)


# (B, Hq, Hkv, Sk, D, dtype): one and several query heads a KV head, above eight of them, KV heads that do not divide the warps; output rows for
# a merge of a CTA each and of a warp each (heads off the four of a CTA), with "one" more partials than are in flight at once
SHAPES = [(70, 4, 4, 353, 128, "bf16"), (40, 24, 3, 1500, 64, "f16"), (33, 20, 10, 700, 128, "f16"), (24, 48, 4, 3000, 64, "bf16"), (100, 24, 2, 800, 128, "bf16"),
          (229, 1, 1, 700, 64, "bf16"), (45, 30, 10, 600, 64, "f16"), (62, 18, 9, 512, 128, "bf16")]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["ragged", "one", "none", "full"])
def test_equal_shares(shape, kind):
    B, Hq, Hkv, Sk, D, dtype = shape
    q, qf = gen((B, Hq, 1, D), dtype, 1)
    k, kf = gen((B, Hkv, Sk, D), dtype, 2)
    v, vf = gen((B, Hkv, Sk, D), dtype, 3)
    lens = _lens(kind, B, Sk)
    for b in range(B):                                     # what lies beyond a sequence's keys must never matter
        k[b, :, lens[b]:], v[b, :, lens[b]:] = float("nan"), float("inf")
    kw = dict(dtype=dtype, want_lse=True, path=N.PATH_DECODE, kv_len=torch.from_numpy(lens).cuda())
    out, lse, info = run_gpu(q, k, v, **kw)
    assert info["launches"] == 2
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, kv_len=lens)
    compare(out, ref, dtype, f"{shape} {kind}")
    compare_lse(lse, ref_lse, dtype, f"{shape} {kind}")
    again, _, _ = run_gpu(q, k, v, **kw)
    assert torch.equal(out, again)
    whole, _, _ = run_gpu(q, k, v, decode_chunk=64, **kw)  # another way to cut the keys
    assert (whole - out).abs().max() <= 4e-3 * max(1.0, float(np.abs(ref).max()))   # 16-bit weights against other maxima


@pytest.mark.parametrize("shape", [(70, 8, 4, 600, 128, 16), (48, 24, 3, 2300, 64, 24)])
def test_equal_shares_of_a_pool(shape):
    B, heads, kv_heads, L, D, bs = shape
    rng = np.random.default_rng(11)
    lens = _lens("ragged", B, L)
    nblocks = int(sum((int(x) + bs - 1) // bs for x in lens)) + 4
    k, kf, v, vf = _pool(nblocks, bs, kv_heads, D, "bf16", 500)
    q, qf = gen((B, 1, heads, D), "bf16", 502)
    bt = _tables(rng, B, (L + bs - 1) // bs, nblocks, lens, bs)
    out, info = _launch_paged(q, k, v, bt, dtype="bf16", block_size=bs, seq_q=1, seq_kv=L, heads=heads, kv_heads=kv_heads, head_dim=D, kv_len=lens)
    assert info["launches"] == 2
    ref = O.paged_sdpa(qf.transpose(0, 2, 1, 3), kf, vf, np.where(bt == 0x3fffffff, 0, bt), block_size=bs, seq_kv=L, kv_len=lens)
    compare(out, ref.transpose(0, 2, 1, 3), "bf16", f"{shape}")


def test_equal_shares_with_a_mask_causal_and_a_head_shard():
    B, Hq, Hkv, Sk, D = 70, 8, 4, 353, 128
    q, qf = gen((B, Hq, 1, D), "bf16", 1)
    k, kf = gen((B, Hkv, Sk, D), "bf16", 2)
    v, vf = gen((B, Hkv, Sk, D), "bf16", 3)
    lens = _lens("ragged", B, Sk)
    keep = (np.random.default_rng(4).random((B, 1, 1, Sk)) < 0.7).astype(np.uint8)
    kw = dict(dtype="bf16", path=N.PATH_DECODE, kv_len=torch.from_numpy(lens).cuda(), mask=torch.from_numpy(keep).cuda(), mask_kind=N.MASK_KEEP_U8,
              causal=True, bottom_right=False, causal_offset=300)
    out, _, _ = run_gpu(q, k, v, **kw)
    ref = O.sdpa(qf, kf, vf, kv_len=lens, mask=keep, mask_kind=O.MASK_KEEP_U8, causal=True, causal_offset=300)
    compare(out, ref[0] if isinstance(ref, tuple) else ref, "bf16", "mask and causal limit")
    part, _, _ = run_gpu(q, k, v, head_begin=4, head_count=4, **kw)
    assert (part[:, 4:] - out[:, 4:]).abs().max() <= 4e-3


@pytest.mark.parametrize("batch,kv_heads,keys,dim,shares", [(48, 1, 8192, 128, True), (47, 1, 8192, 128, False), (128, 1, 2048, 128, True), (110, 1, 241, 128, False),
                                                            (148, 1, 1500, 128, False), (149, 1, 500, 128, True), (190, 1, 814, 64, False), (225, 1, 814, 64, True),
                                                            (64, 32, 4096, 128, False)])
def test_line_of_equal_shares(batch, kv_heads, keys, dim, shares):
    """A launch is given what it asks for; one that cuts its keys evenly asks for a partial per resident warp and sequence."""
    h = N.Handle(device=0, qkv_dtype=N.BF16, head_dim=dim, num_q_heads=kv_heads, num_kv_heads=kv_heads)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = (2 if dim == 128 else 3) * sms * 4
    even = -(-((warps // kv_heads + batch) * kv_heads * (dim + 2) * 4) // 256) * 256
    need = h.workspace_bytes(batch, 1, keys)
    h.close()
    items = batch * kv_heads
    splits = max(1, -(-1184 // items))
    chunk = min(1024, max(64, -(-(-(-keys // splits)) // 64) * 64))
    chunks = -(-keys // chunk)
    plain = -(-(items * chunks * (dim + 2) * 4) // 256) * 256 if chunks > 1 else 0
    assert need == (max(plain, even) if shares else plain)


@pytest.mark.parametrize("shape", SHAPES)
def test_weights_of_two_terms(shape):
    """16-bit outputs against 64 bits: their own rounding and next to nothing more.  Operands of 16 bits are exact, weights of two 16-bit terms are off by 2^-18 of
    themselves, so that the root mean square of the error is that of the rounded exact result (a tenth is left for the rounding of values that lie between); weights of
    one term, whose errors are as large as those of the outputs, make it 1.3 to 1.4 times as large."""
    B, Hq, Hkv, Sk, D, dtype = shape
    q, qf = gen((B, Hq, 1, D), dtype, 1)
    k, kf = gen((B, Hkv, Sk, D), dtype, 2)
    v, vf = gen((B, Hkv, Sk, D), dtype, 3)
    lens = np.maximum(_lens("ragged", B, Sk), 1)
    out, _, info = run_gpu(q, k, v, dtype=dtype, out_dtype=dtype, path=N.PATH_DECODE, kv_len=torch.from_numpy(lens).cuda())
    assert info["launches"] == 2
    got, own = 0.0, 0.0
    for b in range(B):
        n, g = lens[b], Hq // Hkv
        s = np.einsum("hgd,hkd->hgk", qf[b, :, 0].reshape(Hkv, g, D).astype(np.float64), kf[b, :, :n].astype(np.float64)) / np.sqrt(D)
        w = np.exp(s - s.max(-1, keepdims=True))
        want = torch.from_numpy(np.einsum("hgk,hkd->hgd", w / w.sum(-1, keepdims=True), vf[b, :, :n].astype(np.float64)).reshape(Hq, D))
        got += float((out[b, :, 0].cpu().double() - want).square().sum())
        own += float((want.to(out.dtype).double() - want).square().sum())
    assert got <= 1.1 ** 2 * own, (got / own) ** 0.5


@pytest.mark.parametrize("batch,kv_heads,keys,dim,shares", [(87, 2, 128, 128, False), (216, 1, 239, 128, True), (209, 2, 166, 64, False), (201, 2, 218, 64, False), (168, 2, 274, 64, True), (126, 2, 450, 64, False), (134, 2, 450, 64, True)])
def test_line_of_few_steps(batch, kv_heads, keys, dim, shares):
    test_line_of_equal_shares(batch, kv_heads, keys, dim, shares)
