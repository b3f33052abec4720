"""tcgen05 prefill with the keys of every work item cut into parts (fewer items than SMs): parity where a part can be empty,
end inside a sub-tile, or see nothing of a row, and what decides whether a launch is split."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import compare, compare_lse, gen, run_gpu

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Sq, Sk, D): 1024 keys are the fewest that are split; 16 parts at most
SHAPES = [(1, 2, 1, 128, 1024, 64), (1, 1, 1, 1, 1025, 128), (2, 3, 3, 130, 2113, 64), (1, 4, 2, 257, 3007, 128), (1, 8, 1, 97, 8200, 128)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype,out", [("bf16", "f32"), ("f16", "f16")])
@pytest.mark.parametrize("variant", ["plain", "causal", "lengths", "keep_softcap"])
def test_split_prefill(shape, dtype, out, variant):
    B, Hq, Hkv, Sq, Sk, D = shape
    q, qf = gen((B, Hq, Sq, D), dtype, 1)
    k, kf = gen((B, Hkv, Sk, D), dtype, 2)
    v, vf = gen((B, Hkv, Sk, D), dtype, 3)
    kw, okw = {}, {}
    rng = np.random.default_rng(4)
    if variant == "causal":     # top-left: the first parts hold all that the rows see, the others are empty
        kw, okw = dict(causal=True, bottom_right=False, causal_offset=70), dict(causal=True, causal_offset=70)
    elif variant == "lengths":
        lens = np.array([Sk // 3 + 1, 0][:B], np.int32)
        for b in range(B):
            v[b, :, lens[b]:] = float("nan")
        kw, okw = dict(kv_len=torch.from_numpy(lens).cuda()), dict(kv_len=lens)
    elif variant == "keep_softcap":
        keep = (rng.random((1, 1, Sq, Sk)) < 0.5).astype(np.uint8)
        keep[..., Sq // 2, :] = 0
        keep[..., 0, : Sk // 2] = 0
        kw = dict(mask=torch.from_numpy(keep).cuda(), mask_kind=N.MASK_KEEP_U8, softcap=15.0)
        okw = dict(mask=keep, mask_kind=O.MASK_KEEP_U8, softcap=15.0)
    got, lse, info = run_gpu(q, k, v, dtype=dtype, out_dtype=out, want_lse=True, path=N.PATH_PREFILL_SM100, **kw)
    assert info["launches"] == 2
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, **({"causal": False} | okw))
    compare(got, ref, dtype, f"{shape} {variant}")
    compare_lse(lse, ref_lse, dtype, f"{shape} {variant}")


def test_bottom_right_causal_parts_match_one_piece():
    """A chunk at the end of its keys, with and without a workspace: one is split, the other is not, and they differ by the
    rounding of P alone.  A weight near 1 / n is off by at most 2^-9 of itself in bf16 on either side, independently, and n
    of them are averaged over values of standard deviation 0.5: sqrt(2) 2^-9 0.5 / sqrt(n) per output (n >= 3901 visible
    keys), of which 100 000 outputs stay within six."""
    q, _ = gen((1, 4, 200, 128), "bf16", 1)
    k, _ = gen((1, 2, 4100, 128), "bf16", 2)
    v, _ = gen((1, 2, 4100, 128), "bf16", 3)
    split, _, info = run_gpu(q, k, v, dtype="bf16", causal=True)
    assert info["launches"] == 2
    h = N.Handle(device=0, qkv_dtype=N.BF16, out_dtype=N.F32, head_dim=128, num_q_heads=4, num_kv_heads=2, causal=True)
    whole = torch.empty(1, 4, 200, 128, device="cuda")
    args = dict(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=whole.data_ptr(), batch=1, seq_q=200, seq_kv=4100,
                stream=torch.cuda.current_stream().cuda_stream)
    h.launch(**args)
    h.poll(args["stream"])
    assert h.last_launch_count == 1
    assert (split - whole).abs().max().item() <= 6 * 2 ** 0.5 * 2.0 ** -9 * 0.5 / 3901 ** 0.5
    small = torch.empty(4096, dtype=torch.uint8, device="cuda")            # too small a workspace: not split either
    h.launch(workspace=small.data_ptr(), workspace_bytes=4096, **args)
    assert h.last_launch_count == 1
    h.close()


def test_many_items_or_few_keys_are_not_split():
    h = N.Handle(device=0, qkv_dtype=N.BF16, out_dtype=N.F32, head_dim=128, num_q_heads=32, num_kv_heads=8)
    assert h.workspace_bytes(4, 2048, 2048) == 0
    assert h.workspace_bytes(1, 512, 1023) == 0
    assert h.workspace_bytes(1, 512, 8112) > 0
    h.close()
    shard = N.Handle(device=0, qkv_dtype=N.BF16, out_dtype=N.F32, head_dim=128, num_q_heads=32, num_kv_heads=8, head_begin=8, head_count=8)
    assert shard.workspace_bytes(1, 512, 8112) == 0
    shard.close()


@pytest.mark.parametrize("batch", [1, 7, 32, 33])
@pytest.mark.parametrize("causal", [False, True])
def test_items_ordered_by_length(batch, causal):
    """More items than SMs, lengths with ties, zeros and values past the tensor: every sequence is computed once, in whatever
    order the lengths give (33 sequences are not sorted)."""
    rng = np.random.default_rng(batch)
    Hq, Hkv, Sq, Sk, D = 12, 6, 140, 150, 64
    lens = rng.choice([0, 1, 64, 65, 150, 4000], batch).astype(np.int32)
    q, qf = gen((batch, Hq, Sq, D), "bf16", 1)
    k, kf = gen((batch, Hkv, Sk, D), "bf16", 2)
    v, vf = gen((batch, Hkv, Sk, D), "bf16", 3)
    got, lse, _ = run_gpu(q, k, v, dtype="bf16", want_lse=True, path=N.PATH_PREFILL_SM100, causal=causal, kv_len=torch.from_numpy(lens).cuda())
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, causal=causal, kv_len=np.minimum(lens, Sk))
    compare(got, ref, "bf16", f"{batch} {causal}")
    compare_lse(lse, ref_lse, "bf16", f"{batch} {causal}")


@pytest.mark.parametrize("block", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("seq_q,start", [(130, 1000), (300, 2900)])
def test_paged_split_windows(block, seq_q, start):
    """Paged K and V, one loader each, over parts that begin anywhere in a 32-entry window of the block table."""
    from aidotnet.tensors_b200.backend import CudaBackend, GpuBuffer
    heads, kv_heads, D, keys = 4, 2, 128, start + seq_q
    blocks = (keys + block - 1) // block
    pool = blocks + 5
    q, qf = gen((seq_q, heads, D), "bf16", 1)
    k, kf = gen((pool * block, kv_heads, D), "bf16", 2)
    v, vf = gen((pool * block, kv_heads, D), "bf16", 3)
    table = np.random.default_rng(block).permutation(pool)[:blocks].astype(np.int32)
    rows = table[np.arange(keys) // block] * block + np.arange(keys) % block
    unused = np.setdiff1d(np.arange(pool * block), rows)
    v[torch.from_numpy(unused).cuda()] = float("nan")
    backend = CudaBackend(0)
    buf = lambda t: GpuBuffer(t.reshape(-1))
    out = backend.PagedAttentionPrefillGqa(buf(q), buf(k), buf(v), GpuBuffer(torch.from_numpy(table).cuda()), heads, kv_heads, D, block,
                                           seq_q, start, D ** -0.5)
    ref = O.sdpa(qf.transpose(1, 0, 2)[None], kf[rows].transpose(1, 0, 2)[None], vf[rows].transpose(1, 0, 2)[None], causal=True,
                 causal_offset=start)
    compare(out.tensor.float().view(seq_q, heads, D), ref[0].transpose(1, 0, 2), "bf16", f"block {block}")
    backend.Dispose()


def _chunk(backend, case):
    q, k, v, out, heads, kv_heads, sq, sk, D = case
    backend.ScaledDotProductAttention(q, k, v, out, None, None, 1, heads, sq, sk, D, D ** -0.5, True, 0.0, kv_heads)


def _chunk_case(D, seed):
    from aidotnet.tensors_b200.backend import GpuBuffer
    heads, kv_heads, sq, sk = 4, 2, 200, 4100
    q, k, v = (gen(s, "bf16", seed + i)[0].reshape(-1) for i, s in
               enumerate([(1, heads, sq, D), (1, kv_heads, sk, D), (1, kv_heads, sk, D)]))
    return (GpuBuffer(q), GpuBuffer(k), GpuBuffer(v), GpuBuffer(torch.zeros(heads * sq * D, device="cuda")), heads, kv_heads, sq, sk, D)


def test_overlapping_streams_do_not_share_a_workspace():
    from aidotnet.tensors_b200.backend import CudaBackend
    backend = CudaBackend(0)
    cases = [_chunk_case(64, 1), _chunk_case(128, 5)]           # two handles: a handle's launches do not overlap
    for c in cases:
        _chunk(backend, c)
    torch.cuda.synchronize()
    want = [c[3].tensor.clone() for c in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    for c in cases:
        c[3].tensor.zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for c, s in zip(cases, streams):
            with torch.cuda.stream(s):
                _chunk(backend, c)
    torch.cuda.synchronize()
    assert all(torch.equal(c[3].tensor, w) for c, w in zip(cases, want))
    assert len({backend._scratch[s.cuda_stream].data_ptr() for s in streams}) == 2
    backend.Dispose()


def test_split_prefill_in_a_graph():
    from aidotnet.tensors_b200.backend import CudaBackend
    backend, case = CudaBackend(0), _chunk_case(128, 9)
    _chunk(backend, case)
    torch.cuda.synchronize()
    want = case[3].tensor.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _chunk(backend, case)
    case[3].tensor.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(case[3].tensor, want)
    backend.Dispose()


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bias", [-1e9, -1e6, 1e9])
def test_merge_of_parts_with_large_logits(bias, D, group):
    """An additive bias whose ulp is as large as the row sums' logarithm (64 at 1e9): every visible key of the even rows
    carries it and those rows are the plain mean over their keys, however the keys fall into parts - 129 keys put a single one into
    the second part.  The odd rows hide half of their keys behind it."""
    lens = np.array([129, 1, 193, 2113], np.int32)
    B, H, Sq, Sk = 4, 2, 130, 2113
    q, qf = gen((B, H, Sq, D), "bf16", 1)
    k, kf = gen((B, H // group, Sk, D), "bf16", 2)
    v, vf = gen((B, H // group, Sk, D), "bf16", 3)
    mask = np.full((1, 1, Sq, Sk), bias, np.float32)
    mask[..., 1::2, :] = np.where(np.random.default_rng(5).random((Sq // 2, Sk)) < 0.5, 0.0, -abs(bias))
    got, lse, info = run_gpu(q, k, v, dtype="bf16", want_lse=True, path=N.PATH_PREFILL_SM100, mask=torch.from_numpy(mask).cuda(),
                             mask_kind=N.MASK_ADD_F32, kv_len=torch.from_numpy(lens).cuda())
    assert info["launches"] == 2
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, causal=False, mask=mask, mask_kind=O.MASK_ADD_F32, kv_len=lens)
    compare(got, ref, "bf16", f"{bias} {D}")
    # both round m + log(l) once: an ulp of the bias on top of the contract's 2e-2
    got, ref = lse.cpu().numpy(), ref_lse
    assert (np.abs(got - ref) <= 2e-2 + np.spacing(np.abs(ref))).all()


def _unsplit(q, k, v, **kw):
    """The same launch without a workspace: one part."""
    B, Hq, Sq, D = q.shape
    out = torch.empty(B, Hq, Sq, D, device="cuda")
    lse = torch.empty(B, Hq, Sq, device="cuda")
    h = N.Handle(device=0, qkv_dtype=N.F16 if q.dtype == torch.float16 else N.BF16, out_dtype=N.F32, head_dim=D, num_q_heads=Hq,
                 num_kv_heads=k.shape[1], emit_lse=True, **kw)
    stream = torch.cuda.current_stream().cuda_stream
    h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), lse=lse.data_ptr(), batch=B, seq_q=Sq,
             seq_kv=k.shape[2], stream=stream)
    h.poll(stream)
    assert h.last_launch_count == 1
    h.close()
    return out, lse


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("causal", [False, True])
def test_rows_of_nan_stay_nan(causal, group):
    """A NaN in a query row, an infinity in another, and one in a key and in a value of the second part: NaN comes out wherever it
    does without the split, and nowhere else."""
    H, Sq, Sk, D = 2, 130, 2113, 128
    q, _ = gen((1, H, Sq, D), "f16", 1)
    k, _ = gen((1, H // group, Sk, D), "f16", 2)
    v, _ = gen((1, H // group, Sk, D), "f16", 3)
    q[0, 1, 5] = float("nan")
    q[0, 0, 77, 3] = float("inf")
    for change in (lambda: None, lambda: v[0, 0, 1500, 9].fill_(float("nan")), lambda: k[0, 0, 1400].fill_(float("inf"))):
        change()
        got, lse, info = run_gpu(q, k, v, dtype="f16", want_lse=True, path=N.PATH_PREFILL_SM100, causal=causal)
        assert info["launches"] == 2
        whole, whole_lse = _unsplit(q, k, v, causal=causal)
        assert torch.isnan(whole[0, 1, 5]).all() and torch.isnan(whole[0, 0, 77]).all()
        assert torch.equal(torch.isnan(got), torch.isnan(whole))
        assert torch.equal(torch.isneginf(lse), torch.isneginf(whole_lse))


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("how", ["right", "left", "causal", "rows"])
def test_bias_of_the_lowest_float(how, D, group):
    """Masks written as an additive bias of the lowest float: hidden keys get weight 0 wherever they stand - a whole part or the
    first sub-tiles of a row can consist of them - and a row of nothing else is the mean over its keys."""
    low = np.finfo(np.float32).min
    H, Sq, Sk = 2, 130, 2113
    q, qf = gen((1, H, Sq, D), "bf16", 1)
    k, kf = gen((1, H // group, Sk, D), "bf16", 2)
    v, vf = gen((1, H // group, Sk, D), "bf16", 3)
    mask = np.zeros((1, 1, Sq, Sk), np.float32)
    if how == "right":
        mask[..., 300:] = low
    elif how == "left":
        mask[..., :1500] = low
    elif how == "causal":
        mask[0, 0] = np.where(np.arange(Sk)[None] > np.arange(Sq)[:, None], low, 0)
    else:
        mask[0, 0, ::3] = low
    tmask = torch.from_numpy(mask).cuda()
    got, lse, info = run_gpu(q, k, v, dtype="bf16", want_lse=True, path=N.PATH_PREFILL_SM100, mask=tmask, mask_kind=N.MASK_ADD_F32)
    assert info["launches"] == 2
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, causal=False, mask=mask, mask_kind=O.MASK_ADD_F32)
    compare(got, ref, "bf16", f"{how} {D}")
    compare_lse(lse, ref_lse, "bf16", f"{how} {D}")
    few, _, info = run_gpu(q, k[:, :, :900].contiguous(), v[:, :, :900].contiguous(), dtype="bf16", path=N.PATH_PREFILL_SM100,
                           mask=tmask[..., -900:].contiguous(), mask_kind=N.MASK_ADD_F32)
    assert info["launches"] == 1
    ref = O.sdpa(qf, np.ascontiguousarray(kf[:, :, :900]), np.ascontiguousarray(vf[:, :, :900]), causal=False,
                 mask=np.ascontiguousarray(mask[..., -900:]), mask_kind=O.MASK_ADD_F32)
    compare(few, ref, "bf16", f"{how} {D} in one part")


def test_graphs_own_their_workspaces():
    """Two graphs captured on one stream and replayed on two, after a larger call and more streams than the backend keeps a
    buffer for; new tensors take whatever memory the backend let go.  The graphs' memory comes back with them."""
    from aidotnet.tensors_b200.backend import CudaBackend
    backend = CudaBackend(0)
    cases = [_chunk_case(64, 1), _chunk_case(128, 5)]           # two handles: a handle's launches do not overlap
    stream = torch.cuda.Stream()
    graphs = []
    with torch.cuda.stream(stream):
        for c in cases:
            _chunk(backend, c)
    torch.cuda.synchronize()
    want = [c[3].tensor.clone() for c in cases]
    for c in cases:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            _chunk(backend, c)
        graphs.append(graph)
    assert len(backend._captured) == 2
    from aidotnet.tensors_b200.backend import GpuBuffer
    q, k, v = (GpuBuffer(gen(s, "bf16", 20)[0].reshape(-1)) for s in ((1, 8, 1024, 64), (1, 8, 4096, 64), (1, 8, 4096, 64)))
    larger = (q, k, v, GpuBuffer(torch.zeros(8 * 1024 * 64, device="cuda")), 8, 8, 1024, 4096, 64)
    torch.cuda.synchronize()
    for s in [stream] + [torch.cuda.Stream() for _ in range(20)]:
        with torch.cuda.stream(s):
            _chunk(backend, larger)
            _chunk(backend, cases[0])
    torch.cuda.synchronize()
    taken = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for n in (1 << 20, 1 << 22, 1 << 24) for _ in range(8)]
    for c in cases:
        c[3].tensor.zero_()
    torch.cuda.synchronize()
    sides = [torch.cuda.Stream() for _ in graphs]
    for _ in range(20):
        for graph, s in zip(graphs, sides):
            with torch.cuda.stream(s):
                graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(c[3].tensor, w) for c, w in zip(cases, want))
    assert all((t == 7).all() for t in taken)
    import time
    graphs.clear()
    graph = None
    torch.cuda.synchronize()
    for _ in range(100):                                        # the note comes from a thread of CUDA's
        backend._give_back()
        if not backend._captured:
            break
        time.sleep(0.05)
    assert not backend._captured
    backend.Dispose()


def test_head_shards_give_the_rows_of_the_call_in_one_piece():
    """A head shard is never split, whatever workspace it is given, so its bits are those of the same rows of the full call
    without a workspace; with one the full call is split here and differs by the rounding of P."""
    q, _ = gen((1, 8, 200, 128), "bf16", 1)
    k, _ = gen((1, 4, 2100, 128), "bf16", 2)
    v, _ = gen((1, 4, 2100, 128), "bf16", 3)
    split, _, info = run_gpu(q, k, v, dtype="bf16", causal=True)
    assert info["launches"] == 2
    whole, _ = _unsplit(q, k, v, causal=True)
    for begin in (0, 4):
        out = torch.zeros(1, 8, 200, 128, device="cuda")
        _, _, info = run_gpu(q, k, v, dtype="bf16", causal=True, head_begin=begin, head_count=4, out=out)
        assert info["launches"] == 1
        assert torch.equal(out[:, begin:begin + 4], whole[:, begin:begin + 4])
    assert not torch.equal(split, whole)
