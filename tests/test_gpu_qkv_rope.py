"""GPU parity of the decode-step front end (aidn_qkv_rope_cache, aidn_rope_interleaved) against the oracle's
restatement of the reference composition (CudaBackend.cs:8389-8439; rope_interleaved, CudaAttentionKernels.cs:1023-1050),
and the chain the fusion exists for: tokens projected and written into a 16-bit paged pool, then decoded from it."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import AIDN_DT, TORCH_DT

pytestmark = pytest.mark.gpu


def _rope_tables(max_pos, head_dim, rng):
    ang = rng.uniform(0, 2 * np.pi, (max_pos, head_dim // 2)).astype(np.float32)
    return np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)


def _run(x, w, b, cos, sin, *, heads, kv_heads, head_dim, capacity, position=0, positions=None, cache_rows=None,
         weight_dtype="f32", query_dtype="f32", cache_dtype="f32", kc=None, vc=None):
    dev = "cuda"
    tokens = x.shape[0]
    xd = torch.from_numpy(x).to(dev)
    wd = torch.from_numpy(w).to(dev).to(TORCH_DT[weight_dtype])
    bd = torch.from_numpy(b).to(dev) if b is not None else None
    cd, sd = torch.from_numpy(cos).to(dev), torch.from_numpy(sin).to(dev)
    q = torch.full((tokens, heads * head_dim), float("nan"), dtype=TORCH_DT[query_dtype], device=dev)
    kc = torch.zeros((capacity, kv_heads * head_dim), dtype=TORCH_DT[cache_dtype], device=dev) if kc is None else kc
    vc = torch.zeros((capacity, kv_heads * head_dim), dtype=TORCH_DT[cache_dtype], device=dev) if vc is None else vc
    pd = torch.from_numpy(np.asarray(positions, np.int32)).to(dev) if positions is not None else None
    rd = torch.from_numpy(np.asarray(cache_rows, np.int32)).to(dev) if cache_rows is not None else None
    N.qkv_rope_cache(input=xd.data_ptr(), weights=wd.data_ptr(), bias=bd.data_ptr() if bd is not None else None,
                     cosine=cd.data_ptr(), sine=sd.data_ptr(), query=q.data_ptr(), key_cache=kc.data_ptr(),
                     value_cache=vc.data_ptr(), tokens=tokens, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                     position=position, positions=pd.data_ptr() if pd is not None else None,
                     cache_rows=rd.data_ptr() if rd is not None else None, weight_dtype=AIDN_DT[weight_dtype],
                     query_dtype=AIDN_DT[query_dtype], cache_dtype=AIDN_DT[cache_dtype], cache_capacity=capacity,
                     max_position=cos.shape[0], stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return q, kc, vc


@pytest.mark.parametrize("heads,capacity,position", [(4, 16, 0), (8, 64, 17), (16, 128, 127), (32, 64, 63)])
def test_single_token_d64_reference_contract(heads, capacity, position):
    """The reference's contract and its test shapes (DirectGpu/DirectPtxWmmaTests.cs:2110-2113, tolerance 2e-5 at
    :2307-2309): one fp32 token, head_dim 64, cache [capacity, heads, 64], packed bias, `position` both the RoPE
    position and the cache row; the other cache rows stay untouched."""
    rng = np.random.default_rng(100 + heads)
    D, model = 64, heads * 64
    x = rng.uniform(-1, 1, (1, model)).astype(np.float32)
    w = (rng.uniform(-1, 1, (3 * model, model)) / np.sqrt(model)).astype(np.float32)
    b = rng.uniform(-0.1, 0.1, 3 * model).astype(np.float32)
    cos, sin = _rope_tables(capacity, D, rng)
    kref = np.full((capacity, model), 7.0, np.float32)
    vref = np.full((capacity, model), -3.0, np.float32)
    qref = O.qkv_rope_cache(x, w, b, cos, sin, heads=heads, kv_heads=heads, head_dim=D, positions=[position],
                            cache_rows=[position], key_cache=kref, value_cache=vref)
    kc = torch.full((capacity, model), 7.0, device="cuda")
    vc = torch.full((capacity, model), -3.0, device="cuda")
    q, kc, vc = _run(x, w, b, cos, sin, heads=heads, kv_heads=heads, head_dim=D, capacity=capacity, position=position,
                     kc=kc, vc=vc)
    for got, want in ((q, qref), (kc, kref), (vc, vref)):
        assert np.abs(got.cpu().numpy() - want).max() <= 2e-5
    untouched = np.arange(capacity) != position
    assert np.array_equal(kc.cpu().numpy()[untouched], kref[untouched])


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 7, 8, 11])
@pytest.mark.parametrize("weight_dtype,cache_dtype", [("f32", "f32"), ("bf16", "bf16"), ("bf16", "f16")])
def test_batched_tokens_gqa_positions_and_rows(tokens, weight_dtype, cache_dtype):
    """A decode batch: one token per sequence, each with its own position and its own cache row (as a paged pool hands
    them out), grouped-query projection, head_dim 128, bf16 weights and a 16-bit cache."""
    rng = np.random.default_rng(200 + tokens)
    heads, kv_heads, D, capacity, max_pos = 8, 2, 128, 40, 96
    model = heads * D
    x = rng.uniform(-1, 1, (tokens, model)).astype(np.float32)
    w = (rng.uniform(-1, 1, ((heads + 2 * kv_heads) * D, model)) / np.sqrt(model)).astype(np.float32)
    if weight_dtype == "bf16":
        w = torch.from_numpy(w).to(torch.bfloat16).to(torch.float32).numpy()   # the oracle sees the rounded weights
    b = rng.uniform(-0.1, 0.1, (heads + 2 * kv_heads) * D).astype(np.float32)
    cos, sin = _rope_tables(max_pos, D, rng)
    positions = rng.integers(0, max_pos, tokens).astype(np.int32)
    rows = rng.permutation(capacity)[:tokens].astype(np.int32)
    kref = np.zeros((capacity, kv_heads * D), np.float32)
    vref = np.zeros((capacity, kv_heads * D), np.float32)
    qref = O.qkv_rope_cache(x, w, b, cos, sin, heads=heads, kv_heads=kv_heads, head_dim=D, positions=positions,
                            cache_rows=rows, key_cache=kref, value_cache=vref)
    q, kc, vc = _run(x, w, b, cos, sin, heads=heads, kv_heads=kv_heads, head_dim=D, capacity=capacity,
                     positions=positions, cache_rows=rows, weight_dtype=weight_dtype, cache_dtype=cache_dtype)
    assert np.abs(q.cpu().numpy() - qref).max() <= 3e-5
    tol = 3e-5 if cache_dtype == "f32" else 2e-2     # one 16-bit rounding of values of magnitude <= ~2
    assert np.abs(kc.float().cpu().numpy() - kref).max() <= tol
    assert np.abs(vc.float().cpu().numpy() - vref).max() <= tol


def test_row_outside_the_cache_is_not_written():
    rng = np.random.default_rng(5)
    heads, D, capacity = 2, 64, 8
    model = heads * D
    x = rng.uniform(-1, 1, (2, model)).astype(np.float32)
    w = rng.uniform(-1, 1, (3 * model, model)).astype(np.float32)
    cos, sin = _rope_tables(16, D, rng)
    q, kc, vc = _run(x, w, None, cos, sin, heads=heads, kv_heads=heads, head_dim=D, capacity=capacity,
                     positions=[3, 5], cache_rows=[2, 99])
    assert torch.count_nonzero(kc[2]) > 0 and torch.count_nonzero(kc).item() == torch.count_nonzero(kc[2]).item()
    assert torch.isfinite(q).all()


def test_argument_errors():
    z = torch.zeros(64 * 192, device="cuda")
    kw = dict(input=z.data_ptr(), weights=z.data_ptr(), bias=None, cosine=z.data_ptr(), sine=z.data_ptr(),
              query=z.data_ptr(), key_cache=z.data_ptr(), value_cache=z.data_ptr(), tokens=1, heads=1, kv_heads=1,
              head_dim=64, cache_capacity=4, max_position=4, stream=0)
    for bad in (dict(position=4), dict(position=-1), dict(heads=0), dict(kv_heads=3), dict(head_dim=63),
                dict(tokens=0), dict(weight_dtype=N.F16)):
        with pytest.raises(N.AidnError) as e:
            N.qkv_rope_cache(**{**kw, **bad})
        assert e.value.status == N.EINVAL, bad


@pytest.mark.parametrize("rows,head_dim,seq_len,start", [(6, 64, 3, 5), (32, 128, 1, 9), (10, 8, 10, 0)])
def test_rope_interleaved(rows, head_dim, seq_len, start):
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1, 1, (rows, head_dim)).astype(np.float32)
    cos, sin = _rope_tables(start + seq_len, head_dim, rng)
    want = O.rope_interleaved(x, cos, sin, seq_len, start)
    xd, cd, sd = (torch.from_numpy(a).cuda() for a in (x, cos, sin))
    out = torch.empty_like(xd)
    N.rope_interleaved(xd.data_ptr(), cd.data_ptr(), sd.data_ptr(), out.data_ptr(), rows, head_dim, seq_len, start,
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-6


def test_projected_tokens_feed_the_paged_decode():
    """The chain the fusion exists for: every sequence of a decode batch appends one token to a bf16 paged pool through
    aidn_qkv_rope_cache, then aidn_sdpa_launch_paged decodes over the pool; checked against the oracle end to end."""
    rng = np.random.default_rng(77)
    B, heads, kv_heads, D, bs, max_len = 3, 8, 2, 128, 16, 64
    model = heads * D
    lens = np.array([37, 64, 1], np.int32)          # sequence lengths after the append
    nblocks = 16
    bps = max_len // bs
    perm = rng.permutation(nblocks)
    bt = np.full((B, bps), 0x3fffffff, np.int32)
    at = 0
    for b in range(B):
        n = (int(lens[b]) + bs - 1) // bs
        bt[b, :n] = perm[at:at + n]
        at += n
    # pools already hold the older tokens
    kpool = (rng.standard_normal((nblocks * bs, kv_heads * D)) * 0.5).astype(np.float32)
    vpool = (rng.standard_normal((nblocks * bs, kv_heads * D)) * 0.5).astype(np.float32)
    kpool = torch.from_numpy(kpool).to(torch.bfloat16)
    vpool = torch.from_numpy(vpool).to(torch.bfloat16)
    x = rng.uniform(-1, 1, (B, model)).astype(np.float32)
    w = torch.from_numpy((rng.uniform(-1, 1, ((heads + 2 * kv_heads) * D, model)) / np.sqrt(model)).astype(np.float32))
    w = w.to(torch.bfloat16).to(torch.float32).numpy()
    cos, sin = _rope_tables(max_len, D, rng)
    positions = lens - 1
    rows = np.array([bt[b, positions[b] // bs] * bs + positions[b] % bs for b in range(B)], np.int32)
    kref, vref = kpool.float().numpy().copy(), vpool.float().numpy().copy()
    qref = O.qkv_rope_cache(x, w, None, cos, sin, heads=heads, kv_heads=kv_heads, head_dim=D, positions=positions,
                            cache_rows=rows, key_cache=kref, value_cache=vref)
    q, kc, vc = _run(x, w, None, cos, sin, heads=heads, kv_heads=kv_heads, head_dim=D, capacity=nblocks * bs,
                     positions=positions, cache_rows=rows, weight_dtype="bf16", query_dtype="bf16", cache_dtype="bf16",
                     kc=kpool.cuda(), vc=vpool.cuda())
    # decode over the pool the projection just wrote
    out = torch.full((B, heads, D), float("nan"), device="cuda")
    h = N.Handle(device=0, qkv_dtype=N.BF16, head_dim=D, num_q_heads=heads, num_kv_heads=kv_heads)
    stream = torch.cuda.current_stream().cuda_stream
    nbytes = h.workspace_bytes(B, 1, max_len)
    ws = torch.empty(max(nbytes, 16), dtype=torch.uint8, device="cuda")
    btd, kl = torch.from_numpy(bt).cuda(), torch.from_numpy(lens).cuda()
    qo = (heads * D, D, heads * D)
    h.launch(q=q.data_ptr(), k=kc.data_ptr(), v=vc.data_ptr(), out=out.data_ptr(), batch=B, seq_q=1, seq_kv=max_len,
             stream=stream, kv_len=kl.data_ptr(), q_stride=qo, o_stride=qo, workspace=ws.data_ptr() if nbytes else None,
             workspace_bytes=nbytes, block_table=btd.data_ptr(), block_table_stride=bps, block_size=bs, num_blocks=nblocks)
    h.poll(stream)
    h.close()
    bf = lambda a: torch.from_numpy(a).to(torch.bfloat16).to(torch.float32).numpy()
    ref = O.paged_sdpa(bf(qref).reshape(B, 1, heads, D).transpose(0, 2, 1, 3), bf(kref).reshape(nblocks, bs, kv_heads, D),
                       bf(vref).reshape(nblocks, bs, kv_heads, D), np.where(bt == 0x3fffffff, 0, bt), block_size=bs,
                       seq_kv=max_len, kv_len=lens)
    got = out.cpu().numpy().reshape(B, heads, 1, D)
    assert np.abs(got - ref).max() <= 2e-2 and np.abs(got - ref).mean() <= 2e-3


def test_backend_mirror_methods():
    """QkvProjectionRoPECacheD64 / RopeInterleaved through the backend mirror, with the reference's argument checks."""
    from aidotnet.tensors_b200.backend import CudaBackend, GpuBuffer
    rng = np.random.default_rng(31)
    heads, capacity, position, D = 8, 64, 17, 64
    model = heads * D
    x = rng.uniform(-1, 1, (1, model)).astype(np.float32)
    w = (rng.uniform(-1, 1, (3 * model, model)) / np.sqrt(model)).astype(np.float32)
    b = rng.uniform(-0.1, 0.1, 3 * model).astype(np.float32)
    cos, sin = _rope_tables(capacity, D, rng)
    kref = np.zeros((capacity, model), np.float32)
    vref = np.zeros((capacity, model), np.float32)
    qref = O.qkv_rope_cache(x, w, b, cos, sin, heads=heads, kv_heads=heads, head_dim=D, positions=[position],
                            cache_rows=[position], key_cache=kref, value_cache=vref)
    be = CudaBackend(0)
    buf = lambda a: GpuBuffer(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1).cuda())
    q, kc, vc = buf(np.zeros(model, np.float32)), buf(np.zeros_like(kref)), buf(np.zeros_like(vref))
    args = (buf(x), buf(w), buf(b), buf(cos), buf(sin), q, kc, vc)
    be.QkvProjectionRoPECacheD64(*args, heads, capacity, position)
    be.Synchronize()
    assert np.abs(q.tensor.cpu().numpy() - qref[0]).max() <= 2e-5
    assert np.abs(kc.tensor.cpu().numpy().reshape(capacity, model) - kref).max() <= 2e-5
    assert np.abs(vc.tensor.cpu().numpy().reshape(capacity, model) - vref).max() <= 2e-5
    with pytest.raises(ValueError):
        be.QkvProjectionRoPECacheD64(*args, heads, capacity, capacity)
    with pytest.raises(ValueError):
        be.QkvProjectionRoPECacheD64(*args, heads, capacity, -1)
    with pytest.raises(ValueError):
        be.QkvProjectionRoPECacheD64(None, *args[1:], heads, capacity, position)
    with pytest.raises(ValueError):
        be.QkvProjectionRoPECacheD64(*args, heads * 2, capacity, position)      # buffers too small for 16 heads
    xin = rng.uniform(-1, 1, (18, 8)).astype(np.float32)
    c2, s2 = _rope_tables(32, 8, rng)
    out = buf(np.zeros_like(xin))
    be.RopeInterleaved(buf(xin), buf(c2), buf(s2), out, 18, 8, 6, 5)
    be.Synchronize()
    assert np.abs(out.tensor.cpu().numpy().reshape(18, 8) - O.rope_interleaved(xin, c2, s2, 6, 5)).max() <= 1e-6
    with pytest.raises(ValueError):
        be.RopeInterleaved(buf(xin), buf(c2), buf(s2), out, 18, 8, 6, 30)
    be.Dispose()


@pytest.mark.parametrize("weights,cache,D,heads,kv_heads,chunk", [("f32", "f32", 64, 8, 8, 64), ("bf16", "bf16", 64, 8, 8, 64),
                                                                  ("bf16", "bf16", 128, 8, 2, 1024), ("bf16", "bf16", 64, 40, 2, 128),
                                                                  ("f32", "f32", 128, 6, 6, 1024)])
@pytest.mark.parametrize("tokens", [1, 2])
def test_steps_follow_each_other_without_synchronisation(weights, cache, D, heads, kv_heads, chunk, tokens):
    """Projection, attention, projection of what the attention wrote, ...: the kernels of a step start before the ones in front
    of them have ended, and each reads what those write (cache rows, partial results, activations).  The chain gives the bits
    that it gives with a synchronisation after every call."""
    types = {"f32": (torch.float32, N.F32), "bf16": (torch.bfloat16, N.BF16)}
    model, capacity, start, steps = heads * D, 1024, 700, 60
    rng = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *shape: torch.randn(*shape, generator=rng, device="cuda")
    x0 = rnd(tokens, model)
    w = (rnd((heads + 2 * kv_heads) * D, model) * (2.0 / model ** 0.5)).to(types[weights][0])
    bias, cos, sin = rnd((heads + 2 * kv_heads) * D), torch.cos(rnd(capacity, D // 2)), torch.sin(rnd(capacity, D // 2))
    k0, v0 = (rnd(tokens, capacity, kv_heads, D).to(types[cache][0]) for _ in range(2))
    q = torch.empty(tokens, model, device="cuda", dtype=types[cache][0])
    positions = [torch.arange(tokens, device="cuda", dtype=torch.int32) * 0 + start + i for i in range(steps)]
    rows = [torch.arange(tokens, device="cuda", dtype=torch.int32) * capacity + start + i for i in range(steps)]
    h = N.Handle(device=0, qkv_dtype=types[cache][1], out_dtype=N.F32, head_dim=D, num_q_heads=heads, num_kv_heads=kv_heads,
                 decode_chunk=chunk)
    ws = torch.empty(max(16, h.workspace_bytes(tokens, 1, capacity)), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def chain(synchronise):
        x, k, v = x0.clone(), k0.clone(), v0.clone()
        torch.cuda.synchronize()
        for i in range(steps):
            N.qkv_rope_cache(input=x.data_ptr(), weights=w.data_ptr(), bias=bias.data_ptr(), cosine=cos.data_ptr(), sine=sin.data_ptr(),
                             query=q.data_ptr(), key_cache=k.data_ptr(), value_cache=v.data_ptr(), tokens=tokens, heads=heads,
                             kv_heads=kv_heads, head_dim=D, positions=positions[i].data_ptr(), cache_rows=rows[i].data_ptr(),
                             weight_dtype=types[weights][1], query_dtype=types[cache][1], cache_dtype=types[cache][1],
                             cache_capacity=tokens * capacity, max_position=capacity, stream=stream)
            if synchronise:
                torch.cuda.synchronize()
            # the new key is the last one that the query sees; the output is the next step's input
            h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=x.data_ptr(), batch=tokens, seq_q=1, seq_kv=start + i + 1,
                     k_stride=(capacity * kv_heads * D, D, kv_heads * D), v_stride=(capacity * kv_heads * D, D, kv_heads * D),
                     stream=stream, workspace=ws.data_ptr(), workspace_bytes=ws.numel())
            if synchronise:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return x, k, v

    want = chain(True)
    assert torch.isfinite(want[0]).all() and not torch.equal(want[0], x0)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(False), want))
    h.close()


@pytest.mark.parametrize("tokens", [2, 15, 16, 17, 33, 64, 65, 130])
@pytest.mark.parametrize("heads,kv_heads,D", [(4, 4, 64), (5, 1, 72), (6, 3, 20), (40, 8, 128)])
def test_several_tokens_bf16_weights(tokens, heads, kv_heads, D):
    """The tensor-core projection at its edges: passes of up to 64 tokens padded to 16, row tiles of 128, K blocks of 64 and
    splits of K that do not divide.  An element is a sum of `model` products with exact bf16 weights; the accumulation truncates
    (2^-23 of a partial sum) over chains of at most model / 96 + 8 additions per split: 2^-23 x (model / 96 + 16) of the sum of magnitudes,
    twice for the rotation."""
    rng = np.random.default_rng(300 + tokens)
    model, rows, capacity, max_pos = heads * D, (heads + 2 * kv_heads) * D, 200, 96
    x = rng.standard_normal((tokens, model)).astype(np.float32)
    w = torch.from_numpy((rng.standard_normal((rows, model)) / np.sqrt(model)).astype(np.float32)).to(torch.bfloat16).float().numpy()
    b = rng.uniform(-0.1, 0.1, rows).astype(np.float32)
    cos, sin = _rope_tables(max_pos, D, rng)
    positions = rng.integers(0, max_pos, tokens).astype(np.int32)
    cache_rows = rng.permutation(capacity)[:tokens].astype(np.int32)
    q, kc, vc = _run(x, w, b, cos, sin, heads=heads, kv_heads=kv_heads, head_dim=D, capacity=capacity, positions=positions,
                     cache_rows=cache_rows, weight_dtype="bf16")
    y = x.astype(np.float64) @ w.T.astype(np.float64) + b
    y = y.reshape(tokens, -1, D)
    c, s = cos[positions].astype(np.float64)[:, None], sin[positions].astype(np.float64)[:, None]
    even, odd = y[:, :heads + kv_heads, 0::2].copy(), y[:, :heads + kv_heads, 1::2].copy()
    y[:, :heads + kv_heads, 0::2], y[:, :heads + kv_heads, 1::2] = even * c - odd * s, even * s + odd * c
    want = y.reshape(tokens, rows)
    got = torch.cat([q, kc[torch.from_numpy(cache_rows).long()], vc[torch.from_numpy(cache_rows).long()]], 1).cpu().numpy()
    bound = 2 * 2.0 ** -23 * (model / 96 + 16) * (np.abs(x) @ np.abs(w).T).max()
    assert np.abs(got - want).max() <= bound, (np.abs(got - want).max(), bound)
    unused = np.setdiff1d(np.arange(capacity), cache_rows)
    assert torch.count_nonzero(kc[torch.from_numpy(unused).long()]) == 0


def test_infinite_activations_and_weights_of_several_tokens():
    """An infinity or a NaN stays in its token or its row, and an infinite sum is an infinity, as with fp32 multiply-adds."""
    rng = np.random.default_rng(6)
    heads, D, tokens = 2, 64, 3
    model = heads * D
    x = rng.uniform(0.5, 1, (tokens, model)).astype(np.float32)
    w = rng.uniform(0.5, 1, (3 * model, model)).astype(np.float32)
    x[0, 5] = np.inf
    x[1, 7] = 1.0                      # mid and lo of it are 0
    w[9, 7] = -np.inf
    w[300, 3] = np.nan
    w = torch.from_numpy(w).to(torch.bfloat16).float().numpy()
    cos, sin = np.ones((4, D // 2), np.float32), np.zeros((4, D // 2), np.float32)
    q, kc, vc = _run(x, w, None, cos, sin, heads=heads, kv_heads=heads, head_dim=D, capacity=4, positions=[0, 1, 2],
                     cache_rows=[0, 1, 2], weight_dtype="bf16")
    v = vc.cpu().numpy()[:tokens]      # no rotation, which would mix the elements of a pair
    want = x @ w[2 * model:].T
    assert np.array_equal(np.isnan(v), np.isnan(want)) and np.array_equal(np.isinf(v), np.isinf(want))
    assert np.array_equal(v[np.isinf(v)], want[np.isinf(want)])
    got = q.cpu().numpy()
    assert np.isneginf(got[1, 9]) or np.isnan(got[1, 9])     # -inf through the rotation's 0 * x of the pair
    assert np.isfinite(np.delete(got[1:], [8, 9], axis=1)).all()


_EXPIRE = '''
import sys
import numpy as np, torch
from aidotnet.tensors_b200 import native as N
check = sys.argv[1] == "1"
torch.cuda.set_device(0)
st = torch.cuda.current_stream().cuda_stream
heads, kv, D, T, cap = 40, 8, 128, 16, 64
model, rows = heads * D, (heads + 2 * kv) * D
g = torch.Generator("cuda").manual_seed(1)
x = torch.randn((T, model), device="cuda", generator=g)
w = (torch.randn((rows, model), device="cuda", generator=g) / model ** 0.5).to(torch.bfloat16)
cos, sin = torch.ones((cap, D // 2), device="cuda"), torch.zeros((cap, D // 2), device="cuda")
q = torch.full((T, model), 7.0, device="cuda")
kc, vc = (torch.full((cap, kv * D), 7.0, device="cuda") for _ in range(2))
def call(tokens=T, weights=w, dtype=N.BF16):
    N.qkv_rope_cache(input=x.data_ptr(), weights=weights.data_ptr(), bias=None, cosine=cos.data_ptr(), sine=sin.data_ptr(), query=q.data_ptr(),
                     key_cache=kc.data_ptr(), value_cache=vc.data_ptr(), tokens=tokens, heads=heads, kv_heads=kv, head_dim=D, position=0,
                     weight_dtype=dtype, cache_capacity=cap, max_position=cap, stream=st)
def timed_out(f):
    try:
        f()
    except N.AidnError as e:
        assert e.status == N.ETIMEOUT, (e.status, e.message)
        return True
    return False
arm = lambda: N.load().aidn_sdpa_debug_set(None, None, 3)
poll = lambda: N.qkv_rope_poll(st)
assert arm() == 0
if check:
    assert timed_out(call)             # by the call itself, which clears the word:
    assert not timed_out(poll)
else:
    call()
    call(tokens=1)                     # a kernel without such waits, between the failure and its report
    torch.cuda.synchronize()
    assert torch.equal(q[1:], torch.full_like(q[1:], 7.0)) and (kc[1:] == 7).all() and (vc[1:] == 7).all()
    assert timed_out(poll)
    assert not timed_out(poll)
assert torch.equal(q[1:], torch.full_like(q[1:], 7.0)) and (kc[1:] == 7).all() and (vc[1:] == 7).all()   # nothing was stored
assert not timed_out(call) and not timed_out(poll)
want = x.double() @ w.double().T
got = torch.cat([q.double(), kc[:T].double(), vc[:T].double()], 1)
assert (got - want).abs().max() <= 1e-5 * want.abs().max()
wf = w.float()
assert not timed_out(lambda: call(tokens=2, weights=wf, dtype=N.F32)) and not timed_out(poll)
print("expired cleanly")
'''


@pytest.mark.parametrize("launch_check", ["0", "1"])
def test_several_tokens_bounded_waits_expire_cleanly(launch_check):
    """Failure detection without a fault: with the test hook the producer withholds its loads and the waits (20 ms) run out.  No row is
    stored, the failure is reported once - by the poll, or with AIDOTNET_KERNEL_LAUNCH_CHECK by the call itself - and calls after
    it are correct and succeed."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=root)
    env.pop("AIDOTNET_KERNEL_LAUNCH_CHECK", None)
    if launch_check == "1":
        env["AIDOTNET_KERNEL_LAUNCH_CHECK"] = "1"
    r = subprocess.run([sys.executable, "-c", _EXPIRE, launch_check], capture_output=True, text=True, timeout=300, env=env, cwd=root)
    assert r.returncode == 0 and "expired cleanly" in r.stdout, f"stdout:\n{r.stdout}\nstderr:\n{r.stderr[-2000:]}"
