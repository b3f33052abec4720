"""The work that users of this library have it do, as measurable cases over the library's public entry points.

A case is a dict of plain values; ``kind`` names the call sequence:

  ``sdpa``    ScaledDotProductAttention: inference attention over contiguous [B, H, S, D] tensors (prefill, encoder
              layers, and with one query row the batched decode over padded caches)
  ``chunk``   paged_kv_append of a prompt chunk's keys and values, then PagedAttentionPrefillGqa of the chunk
  ``step``    qkv_rope_cache of one token per sequence into a paged pool, then PagedAttentionDecodeBatched
  ``token``   QkvProjectionRoPECacheD64 and FlashDecode: one token of one sequence through a dense cache
  ``train``   FlashAttentionV2 and FlashAttentionBackward: forward with statistics, then dQ, dK and dV
  ``mha``     MultiHeadAttentionForward: projections, attention and output projection in one call

Values are normal, scaled 0.5 for 16-bit tensors and 1.0 for fp32 ones, as in the parity tests and ``bench.py``.
"""
import math

import torch

from aidotnet.tensors_b200 import native
from aidotnet.tensors_b200.backend import CudaBackend, GpuBuffer

TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
NATIVE = {"f32": native.F32, "f16": native.F16, "bf16": native.BF16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}

_backends = {}


def _backend():
    """The program's one backend object per device, kept across calls as a host program keeps it."""
    device = torch.cuda.current_device()
    if device not in _backends:
        _backends[device] = CudaBackend(device)
    return _backends[device]


# ---- the cases ------------------------------------------------------------------------------------------------------

def listed():
    return [
        # one token of one sequence, the smallest call sequence: bound by latency and launches
        dict(name="token_h32_d64_ctx1237", kind="token", weights="bf16", cache="bf16", heads=32, position=1236,
             capacity=2048),
        # the fp32 contract on a small problem (baseline configuration 1)
        dict(name="sdpa_f32_b1_h8_s512_d64", kind="sdpa", dtype="f32", out="f32", batch=1, heads=8, kv_heads=8,
             seq_q=512, seq_k=512, dim=64, causal=False, mask="none", softcap=0.0),
        # an fp32 transformer layer with small heads and a padding mask, ragged length
        dict(name="mha_f32_b8_s197_h16_d32", kind="mha", dtype="f32", out="f32", batch=8, seq=197, heads=16, dim=32,
             mask=True),
        # fp32 training step with a relative-position bias, ragged length
        dict(name="train_f32_b2_h8_s509_d64_bias", kind="train", dtype="f32", out="f32", batch=2, heads=8, seq=509,
             dim=64, causal=False, bias=True),
        # a serving decode step of sixteen sequences: grouped-query projections into a paged pool, then attention
        dict(name="step_b16_h32_kv8_d128_ctx2048", kind="step", dtype="bf16", batch=16, heads=32, kv_heads=8, dim=128,
             block=16, shortest=128, longest=2048),
        # encoder batch of unequal lengths, fp16 in and out, head size 64, no causal mask
        dict(name="sdpa_f16_b6_h16_s997_d64_padded", kind="sdpa", dtype="f16", out="f16", batch=6, heads=16,
             kv_heads=16, seq_q=997, seq_k=997, dim=64, causal=False, mask="lengths", softcap=0.0),
        # a chunk of a long prompt against the paged cache built so far (grouped-query)
        dict(name="chunk_512_at_7600_h32_kv8_d128", kind="chunk", dtype="bf16", tokens=512, start=7600, heads=32,
             kv_heads=8, dim=128, block=16),
        # batched decode over padded caches (baseline configuration 4)
        dict(name="decode_b64_h32_d128_ctx4096", kind="sdpa", dtype="bf16", out="f32", batch=64, heads=32, kv_heads=32,
             seq_q=1, seq_k=4096, dim=128, causal=False, mask="lengths", softcap=0.0),
        # prompt prefill (baseline configuration 2)
        dict(name="prefill_b4_h32_s2048_d128", kind="sdpa", dtype="bf16", out="f32", batch=4, heads=32, kv_heads=32,
             seq_q=2048, seq_k=2048, dim=128, causal=True, mask="none", softcap=0.0),
        # mixed-precision training step of the same layer, one sequence per GPU
        dict(name="train_bf16_b1_h32_s2048_d128", kind="train", dtype="bf16", out="f32", batch=1, heads=32, seq=2048,
             dim=128, causal=True, bias=False),
        # a whole attention layer with resident 16-bit weights
        dict(name="mha_bf16_b4_s2048_h32_d128", kind="mha", dtype="bf16", out="f32", batch=4, seq=2048, heads=32,
             dim=128, mask=False),
        # one GPU's heads of a long-context grouped-query prefill (baseline configuration 5): the largest
        dict(name="prefill_b1_h8_kv1_s32768_d128", kind="sdpa", dtype="bf16", out="f32", batch=1, heads=8, kv_heads=1,
             seq_q=32768, seq_k=32768, dim=128, causal=True, mask="none", softcap=0.0),
    ]


def _log(rng, low, high):
    """A whole number spread evenly over the logarithm of [low, high]."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _heads(rng, low, high, ratios=(1, 1, 2, 4, 8)):
    kv = _log(rng, low, high)
    ratio = rng.choice([r for r in ratios if kv * r <= high * 2])
    return kv * ratio, kv


def _draw_once(rng):
    kind = rng.choice(("prefill", "prefill", "decode", "chunk", "step", "token", "train", "train", "mha"))
    half = rng.choice(("bf16", "bf16", "f16"))
    if kind == "prefill":
        dtype = rng.choice((half, half, "f32"))
        heads, kv_heads = _heads(rng, 1, 32)
        seq_k = _log(rng, 64, 16384 if dtype != "f32" else 2048)
        causal = rng.random() < 0.6
        seq_q = seq_k if rng.random() < 0.7 else _log(rng, 16, seq_k)
        mask = rng.choice(("none", "none", "lengths", "keep"))
        dims = (64, 128, 64, 128, 96) if dtype != "f32" else (32, 64, 80, 128)
        return dict(kind="sdpa", dtype=dtype, out=rng.choice(("f32", dtype)), batch=_log(rng, 1, 16), heads=heads,
                    kv_heads=kv_heads, seq_q=seq_q, seq_k=seq_k, dim=rng.choice(dims), causal=causal, mask=mask,
                    softcap=rng.choice((0.0, 0.0, 0.0, 30.0)))
    if kind == "decode":
        heads, kv_heads = _heads(rng, 2, 32)
        return dict(kind="sdpa", dtype=rng.choice((half, half, half, "f32")), out="f32", batch=_log(rng, 1, 128),
                    heads=heads, kv_heads=kv_heads, seq_q=1, seq_k=_log(rng, 128, 16384), dim=rng.choice((64, 128)),
                    causal=False, mask="lengths", softcap=0.0)
    if kind == "chunk":
        heads, kv_heads = _heads(rng, 2, 32)
        return dict(kind="chunk", dtype=half, tokens=_log(rng, 32, 2048), start=_log(rng, 16, 16384), heads=heads,
                    kv_heads=kv_heads, dim=rng.choice((64, 128)), block=rng.choice((16, 32, 64)))
    if kind == "step":
        heads, kv_heads = _heads(rng, 2, 32, ratios=(1, 4, 8))
        longest = _log(rng, 128, 8192)
        return dict(kind="step", dtype=half, batch=_log(rng, 1, 64), heads=heads, kv_heads=kv_heads,
                    dim=rng.choice((64, 128)), block=rng.choice((16, 32, 64)), shortest=max(1, longest // 16),
                    longest=longest)
    if kind == "token":
        capacity = _log(rng, 256, 8192)
        weights = rng.choice(("bf16", "bf16", "f32"))
        return dict(kind="token", weights=weights, cache="f32" if weights == "f32" else "bf16",
                    heads=_log(rng, 4, 64), position=rng.randrange(capacity // 2, capacity), capacity=capacity)
    if kind == "train":
        dtype = rng.choice((half, half, "f32"))
        return dict(kind="train", dtype=dtype, out=rng.choice(("f32", dtype)), batch=_log(rng, 1, 16),
                    heads=_log(rng, 2, 48), seq=_log(rng, 64, 8192 if dtype != "f32" else 1024),
                    dim=rng.choice((64, 128)), causal=rng.random() < 0.6, bias=rng.random() < 0.3)
    dtype = rng.choice((half, half, "f32"))
    return dict(kind="mha", dtype=dtype, out=rng.choice(("f32", dtype)), batch=_log(rng, 1, 16),
                seq=_log(rng, 16, 4096 if dtype != "f32" else 512), heads=2 * _log(rng, 1, 24),
                dim=rng.choice((64, 128) if dtype != "f32" else (16, 32, 64)), mask=rng.random() < 0.3)


def _cost(case):
    """A rough common scale of what a case costs: fp32 and odd head sizes run on the FP32 units."""
    w = work(case)
    slow = "f32" in (case.get("dtype"), case.get("cache")) or case.get("dim") == 96
    return w["flops"] * (64 if slow else 1) + w["bytes"] * 200


def draw(rng):
    cap = max(_cost(c) for c in listed())
    while True:
        case = _draw_once(rng)
        if _cost(case) <= cap:
            return case


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def _lengths(count, low, high):
    """``count`` lengths spread evenly over [low, high]: every seed shuffles the same ones."""
    return [high - (high - low) * i // max(1, count - 1) for i in range(count)] if count > 1 else [high]


def _sdpa_lengths(case):
    if case["mask"] != "lengths":
        return [case["seq_k"]] * case["batch"]
    return _lengths(case["batch"], max(1, case["seq_k"] // 8), case["seq_k"])


def _pairs(seq_q, seq_k, causal, offset, limit):
    """Visible (query, key) pairs: key k < limit, and k <= q + offset under a causal mask."""
    if not causal:
        return seq_q * min(seq_k, limit)
    total = 0
    rows_full = max(0, min(seq_q, seq_q - max(0, limit - 1 - offset)))   # rows that see all of the `limit` keys
    rows = seq_q - rows_full
    first = max(0, -offset)                                              # rows before this one see no key
    if rows > first:
        total += (rows - first) * ((first + offset + 1) + (rows + offset)) // 2
    return total + rows_full * limit


def work(case):
    kind = case["kind"]
    if kind == "sdpa":
        b, hq, hkv, sq, sk, d = (case[k] for k in ("batch", "heads", "kv_heads", "seq_q", "seq_k", "dim"))
        e, o = BYTES[case["dtype"]], BYTES[case["out"]]
        lens = _sdpa_lengths(case)
        pairs = hq * sum(_pairs(sq, sk, case["causal"], sk - sq, n) for n in lens)
        nbytes = b * hq * sq * d * (e + o) + 2 * hkv * d * e * sum(lens)
        if case["mask"] == "keep":
            nbytes += sq * sk
        return {"bytes": nbytes, "flops": 4 * d * pairs}
    if kind == "chunk":
        t, hq, hkv, d, e = case["tokens"], case["heads"], case["kv_heads"], case["dim"], BYTES[case["dtype"]]
        keys = case["start"] + t
        pairs = hq * _pairs(t, keys, True, case["start"], keys)
        # new rows read and written, the rows before them read, queries and outputs
        return {"bytes": 2 * hkv * d * e * (2 * t + case["start"]) + 2 * t * hq * d * e, "flops": 4 * d * pairs}
    if kind == "step":
        n, hq, hkv, d, e = case["batch"], case["heads"], case["kv_heads"], case["dim"], BYTES[case["dtype"]]
        model = hq * d
        rows = (hq + 2 * hkv) * d
        lens = _lengths(n, case["shortest"], case["longest"])
        nbytes = rows * model * 2 + n * model * 4 + 2 * hkv * d * e * sum(lens) + n * hq * d * e
        return {"bytes": nbytes, "flops": 2 * n * rows * model + 4 * d * hq * sum(lens)}
    if kind == "token":
        model, keys = case["heads"] * 64, case["position"] + 1
        nbytes = 3 * model * model * BYTES[case["weights"]] + 2 * keys * model * BYTES[case["cache"]] + 4 * 2 * model
        return {"bytes": nbytes, "flops": 6 * model * model + 4 * keys * model}
    if kind == "train":
        b, h, s, d = case["batch"], case["heads"], case["seq"], case["dim"]
        e, o = BYTES[case["dtype"]], BYTES[case["out"]]
        pairs = b * h * _pairs(s, s, case["causal"], 0, s)
        # Q, K, V and dO in; O, the statistics and three fp32 gradients out; the bias once
        nbytes = b * h * s * d * (3 * e + 2 * o + 12) + b * h * s * 4 + (h * s * s * 4 if case["bias"] else 0)
        return {"bytes": nbytes, "flops": 14 * d * pairs}
    b, s, h, d = case["batch"], case["seq"], case["heads"], case["dim"]
    e, o, model = BYTES[case["dtype"]], BYTES[case["out"]], case["heads"] * case["dim"]
    nbytes = b * s * model * (e + o) + 4 * model * model * e + (b * s if case["mask"] else 0)
    return {"bytes": nbytes, "flops": 8 * b * s * model * model + 4 * b * h * s * s * d}


# ---- inputs -----------------------------------------------------------------------------------------------------------

class _Inputs:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, count, dtype, scale=None):
        if scale is None:
            scale = 1.0 if dtype == "f32" else 0.5
        return GpuBuffer(torch.randn(count, generator=self.g, device="cuda", dtype=TORCH[dtype]).mul_(scale))

    def order(self, count):
        return torch.randperm(count, generator=self.g, device="cuda")

    def lengths(self, values):
        t = torch.tensor(values, dtype=torch.int32, device="cuda")
        return GpuBuffer(t[self.order(len(values))].contiguous())

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda")


def _rope_tables(positions, dim):
    angle = torch.arange(positions, device="cuda", dtype=torch.float32)[:, None] * torch.pow(
        10000.0, -torch.arange(dim // 2, device="cuda", dtype=torch.float32) * 2 / dim)[None, :]
    return GpuBuffer(torch.cos(angle).contiguous().view(-1)), GpuBuffer(torch.sin(angle).contiguous().view(-1))


def prepare(case, seed):
    inputs = _Inputs(seed)
    backend = _backend()
    kind = case["kind"]
    st = {"case": case, "backend": backend}
    if kind == "sdpa":
        b, hq, hkv, sq, sk, d, dt = (case[k] for k in ("batch", "heads", "kv_heads", "seq_q", "seq_k", "dim", "dtype"))
        st.update(q=inputs.normal(b * hq * sq * d, dt), k=inputs.normal(b * hkv * sk * d, dt),
                  v=inputs.normal(b * hkv * sk * d, dt), mask=None, lengths=None,
                  out=backend.AllocateBuffer(b * hq * sq * d, TORCH[case["out"]]))
        if case["mask"] == "lengths":
            st["lengths"] = inputs.lengths(_sdpa_lengths(case))
        elif case["mask"] == "keep":                                       # one boolean mask shared by all heads
            keep = inputs.uniform(sq, sk) < 0.9
            keep[:, 0] = True
            st["mask"] = GpuBuffer(keep.to(torch.uint8).view(-1))
    elif kind == "chunk":
        t, hq, hkv, d, dt, bs = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "dtype", "block"))
        blocks = (case["start"] + t + bs - 1) // bs
        pool = blocks + blocks // 4 + 1
        st.update(q=inputs.normal(t * hq * d, dt), new_k=inputs.normal(t * hkv * d, dt),
                  new_v=inputs.normal(t * hkv * d, dt), k=inputs.normal(pool * bs * hkv * d, dt),
                  v=inputs.normal(pool * bs * hkv * d, dt), blocks=pool,
                  table=GpuBuffer(inputs.order(pool)[:blocks].to(torch.int32).contiguous()))
    elif kind == "step":
        n, hq, hkv, d, dt, bs = (case[k] for k in ("batch", "heads", "kv_heads", "dim", "dtype", "block"))
        model, rows = hq * d, (hq + 2 * hkv) * d
        per_seq = (case["longest"] + bs - 1) // bs
        lens = inputs.lengths(_lengths(n, case["shortest"], case["longest"]))
        table = inputs.order(n * per_seq).to(torch.int32).view(n, per_seq).contiguous()
        last = (lens.tensor - 1).long()
        cache_rows = table.long().gather(1, (last // bs)[:, None])[:, 0] * bs + last % bs
        cos, sin = _rope_tables(case["longest"], d)
        st.update(x=inputs.normal(n * model, "f32"), w=inputs.normal(rows * model, "bf16", 1 / math.sqrt(model)),
                  bias=inputs.normal(rows, "f32", 0.1), cos=cos, sin=sin,
                  q=backend.AllocateBuffer(n * model, TORCH[dt]), k=inputs.normal(n * per_seq * bs * hkv * d, dt),
                  v=inputs.normal(n * per_seq * bs * hkv * d, dt), lengths=lens,
                  positions=GpuBuffer(last.to(torch.int32).contiguous()),
                  cache_rows=GpuBuffer(cache_rows.to(torch.int32).contiguous()),
                  table=GpuBuffer(table.view(-1)), per_seq=per_seq)
    elif kind == "token":
        model, cap = case["heads"] * 64, case["capacity"]
        cos, sin = _rope_tables(cap, 64)
        st.update(x=inputs.normal(model, "f32"), w=inputs.normal(3 * model * model, case["weights"], 1 / math.sqrt(model)),
                  bias=inputs.normal(3 * model, "f32", 0.1), cos=cos, sin=sin,
                  q=backend.AllocateBuffer(model, TORCH[case["cache"]]), k=inputs.normal(cap * model, case["cache"]),
                  v=inputs.normal(cap * model, case["cache"]))
    elif kind == "train":
        b, h, s, d, dt = (case[k] for k in ("batch", "heads", "seq", "dim", "dtype"))
        n = b * h * s * d
        st.update(q=inputs.normal(n, dt), k=inputs.normal(n, dt), v=inputs.normal(n, dt),
                  dout=inputs.normal(n, case["out"], 1.0), out=backend.AllocateBuffer(n, TORCH[case["out"]]),
                  stats=backend.AllocateBuffer(b * h * s), dq=backend.AllocateBuffer(n), dk=backend.AllocateBuffer(n),
                  dv=backend.AllocateBuffer(n), bias=inputs.normal(h * s * s, "f32", 0.5) if case["bias"] else None)
    else:
        b, s, h, d, dt = (case[k] for k in ("batch", "seq", "heads", "dim", "dtype"))
        model = h * d
        st.update(x=inputs.normal(b * s * model, dt),
                  w=[inputs.normal(model * model, dt, 1 / math.sqrt(model)) for _ in range(4)],
                  out=backend.AllocateBuffer(b * s * model, TORCH[case["out"]]), mask=None, mask_shape=None)
        if case["mask"]:                                                   # key padding, one row per sequence
            lens = inputs.lengths(_lengths(b, max(1, s // 2), s)).tensor
            st["mask"] = GpuBuffer((torch.arange(s, device="cuda")[None, :] < lens[:, None]).to(torch.uint8).view(-1))
            st["mask_shape"] = (b, 1, 1, s)
    return st


# ---- one pass ---------------------------------------------------------------------------------------------------------

def run(st):
    case, be = st["case"], st["backend"]
    kind = case["kind"]
    if kind == "sdpa":
        be.ScaledDotProductAttention(st["q"], st["k"], st["v"], st["out"], None, st["mask"], case["batch"], case["heads"],
                                     case["seq_q"], case["seq_k"], case["dim"], case["dim"] ** -0.5, case["causal"],
                                     case["softcap"], case["kv_heads"], st["lengths"])
        return st["out"].tensor
    if kind == "chunk":
        row_bytes = case["kv_heads"] * case["dim"] * BYTES[case["dtype"]]
        native.paged_kv_append(st["new_k"].Handle, st["new_v"].Handle, st["k"].Handle, st["v"].Handle, st["table"].Handle,
                               case["start"], case["tokens"], case["block"], st["blocks"], row_bytes,
                               be.stream.cuda_stream)
        out = be.PagedAttentionPrefillGqa(st["q"], st["k"], st["v"], st["table"], case["heads"], case["kv_heads"],
                                          case["dim"], case["block"], case["tokens"], case["start"], case["dim"] ** -0.5)
        return {"out": out.tensor, "keys": st["k"].tensor, "values": st["v"].tensor}
    if kind == "step":
        n, hq, hkv, d = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        native.qkv_rope_cache(input=st["x"].Handle, weights=st["w"].Handle, bias=st["bias"].Handle, cosine=st["cos"].Handle,
                              sine=st["sin"].Handle, query=st["q"].Handle, key_cache=st["k"].Handle,
                              value_cache=st["v"].Handle, tokens=n, heads=hq, kv_heads=hkv, head_dim=d,
                              positions=st["positions"].Handle, cache_rows=st["cache_rows"].Handle,
                              weight_dtype=native.BF16, query_dtype=NATIVE[case["dtype"]],
                              cache_dtype=NATIVE[case["dtype"]], cache_capacity=n * st["per_seq"] * case["block"],
                              max_position=case["longest"], stream=be.stream.cuda_stream)
        out = be.PagedAttentionDecodeBatched(st["q"], st["k"], st["v"], st["table"], st["lengths"], n, hq, hkv, d,
                                             case["block"], case["longest"], st["per_seq"], d ** -0.5)
        return {"out": out.tensor, "query": st["q"].tensor, "keys": st["k"].tensor, "values": st["v"].tensor}
    if kind == "token":
        be.QkvProjectionRoPECacheD64(st["x"], st["w"], st["bias"], st["cos"], st["sin"], st["q"], st["k"], st["v"],
                                     case["heads"], case["capacity"], case["position"])
        out = be.FlashDecode(st["q"], st["k"], st["v"], case["heads"], case["heads"], 64, case["position"] + 1, 0.125)
        return {"out": out.tensor, "query": st["q"].tensor, "keys": st["k"].tensor, "values": st["v"].tensor}
    if kind == "train":
        b, h, s, d = case["batch"], case["heads"], case["seq"], case["dim"]
        be.FlashAttentionV2(st["q"], st["k"], st["v"], st["out"], st["stats"], b, h, s, s, d, d ** -0.5, case["causal"],
                            st["bias"], 0)
        be.FlashAttentionBackward(st["dout"], st["q"], st["k"], st["v"], st["out"], st["stats"], st["dq"], st["dk"],
                                  st["dv"], b, h, s, s, d, d ** -0.5, case["causal"], st["bias"], 0)
        return {name: st[name].tensor for name in ("out", "stats", "dq", "dk", "dv")}
    be.MultiHeadAttentionForward(st["x"], *st["w"], st["out"], case["batch"], case["seq"], case["heads"] * case["dim"],
                                 case["heads"], st["mask"], st["mask_shape"], exact=case["dtype"] == "f32")
    return st["out"].tensor


def tolerance(case):
    """About four times the error of every output against a float64 evaluation, over the listed cases and forty drawn
    ones: fp32 1e-6 relative (8e-6 at most, of one element), fp16 4.2e-4 (7.6e-3), bf16 2.4e-3, through two projections
    2.9e-3 (an attention row that averages many keys is small beside its tensor's root mean square and is rounded once
    per key: 1.1e-1 at most; 1.8e-2 with one query row per head or an output projection)."""
    if "f32" in (case.get("dtype"), case.get("cache")):
        return {"rel": 4e-6, "max": 4e-5}
    if case.get("dtype") == "f16":
        return {"rel": 1.7e-3, "max": 3e-2}
    rows = case["kind"] == "train" or (case["kind"] == "sdpa" and case["seq_q"] > 1)
    return {"rel": 1.2e-2 if case["kind"] == "mha" else 1e-2, "max": 0.45 if rows else 7e-2}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------

def _attend(q, k, v, scale, visible=None, softcap=0.0, bias=None, dout=None):
    """softmax(scale q k^T) v of one (sequence, head) in float64, some rows at a time: q [Sq, D], k and v [Sk, D],
    ``visible(rows)`` and ``bias`` of [rows, Sk].  Returns the output and the log-sum-exp, and with ``dout`` the three
    gradients too."""
    rows = max(1, (1 << 26) // k.shape[0])
    out, lse, dq = torch.empty_like(q), torch.empty_like(q[:, 0]), torch.empty_like(q)
    dk, dv = torch.zeros_like(k), torch.zeros_like(v)
    for first in range(0, q.shape[0], rows):
        at = slice(first, min(q.shape[0], first + rows))
        s = (q[at] @ k.T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if bias is not None:
            s = s + bias[at].double()
        if visible is not None:
            s = s.masked_fill(~visible(torch.arange(at.start, at.stop, device=q.device)), float("-inf"))
        lse[at] = torch.logsumexp(s, 1)
        p = torch.exp(s - lse[at, None])
        out[at] = p @ v
        if dout is not None:
            ds = p * (dout[at] @ v.T - (dout[at] * out[at]).sum(1, keepdim=True))
            dq[at] = scale * (ds @ k)
            dk += scale * (ds.T @ q[at])
            dv += p.T @ dout[at]
    return (out, lse) if dout is None else (out, lse, dq, dk, dv)


def _rotated(x, cos, sin, positions):
    """Interleaved RoPE of x [tokens, heads, D] at the tokens' positions."""
    half = x.shape[2] // 2
    c, s = (t.tensor.view(-1, half)[positions].double()[:, None] for t in (cos, sin))
    even, odd = x[..., 0::2], x[..., 1::2]
    return torch.stack((even * c - odd * s, even * s + odd * c), -1).flatten(2)


def exact(case, seed):
    """What ``run`` returns, evaluated in float64 with no rounding in between."""
    st = prepare(case, seed)
    kind, scale = case["kind"], case.get("dim", 64) ** -0.5

    def wide(name, *shape):
        return st[name].tensor.double().view(*shape)

    if kind == "sdpa":
        b, hq, hkv, sq, sk, d = (case[k] for k in ("batch", "heads", "kv_heads", "seq_q", "seq_k", "dim"))
        q, out = st["q"].tensor.view(b, hq, sq, d), torch.empty(b, hq, sq, d, dtype=torch.float64, device="cuda")
        k, v = (st[name].tensor.view(b, hkv, sk, d) for name in ("k", "v"))
        keys = torch.arange(sk, device="cuda")
        keep = st["mask"].tensor.view(sq, sk) != 0 if st["mask"] is not None else None
        lens = st["lengths"].tensor.tolist() if st["lengths"] is not None else [sk] * b
        for i in range(b):
            def visible(rows):
                seen = (keys < lens[i])[None, :].expand(len(rows), sk)
                if case["causal"]:
                    seen = seen & (keys[None, :] <= rows[:, None] + (sk - sq))
                return seen if keep is None else seen & keep[rows]
            for h in range(hq):
                kv = h // (hq // hkv)
                out[i, h] = _attend(q[i, h].double(), k[i, kv].double(), v[i, kv].double(), scale, visible,
                                    case["softcap"])[0]
        return out.view(-1)
    if kind == "chunk":
        t, hq, hkv, d, bs, start = (case[k] for k in ("tokens", "heads", "kv_heads", "dim", "block", "start"))
        keys = torch.arange(start + t, device="cuda")
        rows = st["table"].tensor.long()[keys // bs] * bs + keys % bs
        k, v = wide("k", -1, hkv, d), wide("v", -1, hkv, d)
        k[rows[start:]], v[rows[start:]] = wide("new_k", t, hkv, d), wide("new_v", t, hkv, d)
        q, out = wide("q", t, hq, d), torch.empty(t, hq, d, dtype=torch.float64, device="cuda")
        for h in range(hq):
            kv = h // (hq // hkv)
            out[:, h] = _attend(q[:, h], k[rows, kv], v[rows, kv], scale,
                                lambda r: keys[None, :] <= r[:, None] + start)[0]
        return {"out": out.view(-1), "keys": k.view(-1), "values": v.view(-1)}
    if kind in ("step", "token"):
        if kind == "step":
            n, hq, hkv, d, bs = (case[k] for k in ("batch", "heads", "kv_heads", "dim", "block"))
            positions, cache_rows = st["positions"].tensor.long(), st["cache_rows"].tensor.long()
            table, lens = st["table"].tensor.long().view(n, -1), st["lengths"].tensor.tolist()
        else:
            n, hq, hkv, d = 1, case["heads"], case["heads"], 64
            positions = cache_rows = torch.tensor([case["position"]], device="cuda")
            lens = [case["position"] + 1]
        y = wide("x", n, -1) @ wide("w", (hq + 2 * hkv) * d, -1).T + st["bias"].tensor.double()
        q, new_k, new_v = y.view(n, hq + 2 * hkv, d).split((hq, hkv, hkv), 1)
        q, k, v = _rotated(q, st["cos"], st["sin"], positions), wide("k", -1, hkv, d), wide("v", -1, hkv, d)
        k[cache_rows], v[cache_rows] = _rotated(new_k, st["cos"], st["sin"], positions), new_v
        out = torch.empty(n, hq, d, dtype=torch.float64, device="cuda")
        for i in range(n):
            rows = torch.arange(lens[i], device="cuda")
            if kind == "step":
                rows = table[i, rows // bs] * bs + rows % bs
            for h in range(hq):
                kv = h // (hq // hkv)
                out[i, h] = _attend(q[i, h:h + 1], k[rows, kv], v[rows, kv], scale)[0][0]
        return {"out": out.view(-1), "query": q.reshape(-1), "keys": k.view(-1), "values": v.view(-1)}
    if kind == "train":
        b, h, s, d = (case[k] for k in ("batch", "heads", "seq", "dim"))
        got = {name: torch.empty(b, h, s, *size, dtype=torch.float64, device="cuda")
               for name, size in (("out", (d,)), ("stats", ()), ("dq", (d,)), ("dk", (d,)), ("dv", (d,)))}
        ins = [st[name].tensor.view(b, h, s, d) for name in ("q", "k", "v", "dout")]
        bias = st["bias"].tensor.view(h, s, s) if case["bias"] else None
        keys = torch.arange(s, device="cuda")
        visible = (lambda r: keys[None, :] <= r[:, None]) if case["causal"] else None
        for i in range(b):
            for j in range(h):
                q, k, v, dout = (t[i, j].double() for t in ins)
                for name, x in zip(got, _attend(q, k, v, scale, visible, bias=None if bias is None else bias[j],
                                                dout=dout)):
                    got[name][i, j] = x
        return {name: x.view(-1) for name, x in got.items()}
    b, s, h, d = (case[k] for k in ("batch", "seq", "heads", "dim"))
    x = wide("x", b * s, h * d)
    q, k, v = ((x @ w.tensor.double().view(h * d, h * d)).view(b, s, h, d) for w in st["w"][:3])
    keep = st["mask"].tensor.view(b, s) != 0 if case["mask"] else None
    out = torch.empty(b, s, h, d, dtype=torch.float64, device="cuda")
    for i in range(b):
        for j in range(h):
            out[i, :, j] = _attend(q[i, :, j], k[i, :, j], v[i, :, j], scale,
                                   None if keep is None else lambda r: keep[i][None, :].expand(len(r), s))[0]
    return (out.view(b * s, h * d) @ st["w"][3].tensor.double().view(h * d, h * d)).view(-1)
