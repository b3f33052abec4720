"""Launches that are set up under the end of the one before (csrc/common.cuh, launch_dependent), back to back on one stream: what a launch reads was
written by the one in front of it, and what it writes is read by that one.  Every result is the same bits as with a synchronisation
behind every call."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N

from tests._harness import AIDN_DT, gen

pytestmark = pytest.mark.gpu


def _same_bits(steps, results):
    """Runs the steps with a synchronisation behind each, then three times without; `results()` are the tensors that they leave."""
    def run(synchronise):
        for t in results():
            t.fill_(float("nan"))
        torch.cuda.synchronize()
        for step in steps:
            step()
            if synchronise:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [t.clone() for t in results()]
    want = run(True)
    assert all(torch.isfinite(t).all() for t in want)
    for _ in range(3):
        for got, ref in zip(run(False), want):
            assert torch.equal(got, ref)


# (dtype, B, Hq, Hkv, Sq, Sk, D): dK / dV long done while dQ walks the keys, dQ long done, and both of a length; 16 bits and fp32 on tcgen05
BACKWARD = [("bf16", 1, 4, 4, 40, 4100, 64), ("bf16", 1, 4, 1, 4100, 40, 128), ("f16", 2, 8, 2, 700, 700, 64), ("f32", 1, 4, 4, 330, 4000, 64),
            ("f32", 2, 4, 2, 600, 600, 32)]


@pytest.mark.parametrize("case", BACKWARD)
@pytest.mark.parametrize("bias", [False, True])
def test_gradients_are_read_behind_the_backward(case, bias):
    """Two sets of inputs in turn through one workspace, where the row sums of the set before still lie, and gradients that the next set
    overwrites: a copy by aidn_paged_kv_append, which starts as early as it may, takes them out in between."""
    dtype, B, Hq, Hkv, Sq, Sk, D = case
    stream = torch.cuda.current_stream().cuda_stream
    h = N.Handle(device=0, qkv_dtype=AIDN_DT[dtype], out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv, emit_lse=True,
                 mask_kind=N.MASK_ADD_F32 if bias else N.MASK_NONE)
    ws = torch.empty(h.backward_workspace_bytes(B, Sq), dtype=torch.uint8, device="cuda")
    fws = torch.empty(max(h.workspace_bytes(B, Sq, Sk), 16), dtype=torch.uint8, device="cuda")
    dq = torch.empty(B * Hq * Sq, D, device="cuda")
    dk, dv = (torch.empty(B * Hkv * Sk, D, device="cuda") for _ in range(2))
    sets = []
    for i in range(2):
        q, k, v = (gen((B, n, s, D), dtype, 10 * i + j)[0] for j, (n, s) in enumerate(((Hq, Sq), (Hkv, Sk), (Hkv, Sk))))
        sets.append(dict(q=q, k=k, v=v, dout=gen((B, Hq, Sq, D), "f32", 10 * i + 4, 1.0)[0], out=torch.empty(B, Hq, Sq, D, device="cuda"),
                         lse=torch.empty(B, Hq, Sq, device="cuda"), mask=gen((Hq, Sq, Sk), "f32", 10 * i + 5, 1.0)[0] if bias else None))
    common = lambda s: dict(q=s["q"].data_ptr(), k=s["k"].data_ptr(), v=s["v"].data_ptr(), out=s["out"].data_ptr(), lse=s["lse"].data_ptr(), batch=B, seq_q=Sq,
                            seq_kv=Sk, stream=stream, mask=s["mask"].data_ptr() if bias else None, mask_stride=(0, Sq * Sk, Sk, 1) if bias else (0, 0, 0, 0))
    for s in sets:
        h.launch(workspace=fws.data_ptr(), workspace_bytes=fws.numel(), **common(s))
    taken = [[torch.empty_like(dq), torch.empty_like(dq), torch.empty_like(dk), torch.empty_like(dv)] for _ in range(6)]
    table = torch.zeros(1, dtype=torch.int32, device="cuda")

    def take(a, b, to_a, to_b):
        N.paged_kv_append(a.data_ptr(), b.data_ptr(), to_a.data_ptr(), to_b.data_ptr(), table.data_ptr(), 0, a.shape[0], a.shape[0], 1, D * 4, stream)

    steps = []
    for i, out in enumerate(taken):
        s = sets[i % 2]
        steps.append(lambda s=s: h.backward(dout=s["dout"].data_ptr(), dq=dq.data_ptr(), dk=dk.data_ptr(), dv=dv.data_ptr(), workspace=ws.data_ptr(),
                                            workspace_bytes=ws.numel(), **common(s)))
        steps.append(lambda out=out: take(dq, dq, out[0], out[1]))
        if i % 2:                                              # without it the next backward comes right behind dQ's copy
            steps.append(lambda out=out: take(dk, dv, out[2], out[3]))
    _same_bits(steps, lambda: [t for i, out in enumerate(taken) for t in (out if i % 2 else out[:1])])
    h.poll(stream)
    h.close()


@pytest.mark.parametrize("dtype,heads,kv_heads,D,tokens,start", [("bf16", 8, 2, 128, 130, 300), ("f16", 4, 4, 64, 40, 1000)])
def test_append_prefill_append(dtype, heads, kv_heads, D, tokens, start):
    """New rows over the same positions of a pool, each set read by the prefill behind it."""
    stream = torch.cuda.current_stream().cuda_stream
    bs, keys = 16, start + tokens
    blocks = (keys + bs - 1) // bs
    table = torch.randperm(blocks, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).to(torch.int32)
    pool_k, pool_v = (gen((blocks, bs, kv_heads, D), dtype, i)[0] for i in range(2))
    new = [[gen((tokens, kv_heads, D), dtype, 10 + 2 * i + j)[0] for j in range(2)] for i in range(4)]
    q = gen((tokens, heads, D), dtype, 3)[0]
    outs = [torch.empty(tokens, heads, D, device="cuda") for _ in range(4)]
    h = N.Handle(device=0, qkv_dtype=AIDN_DT[dtype], out_dtype=N.F32, head_dim=D, num_q_heads=heads, num_kv_heads=kv_heads, causal=True, causal_bottom_right=False,
                 causal_offset=start)
    ws = torch.empty(max(h.workspace_bytes(1, tokens, keys), 16), dtype=torch.uint8, device="cuda")
    steps = []
    for (nk, nv), out in zip(new, outs):
        steps.append(lambda nk=nk, nv=nv: N.paged_kv_append(nk.data_ptr(), nv.data_ptr(), pool_k.data_ptr(), pool_v.data_ptr(), table.data_ptr(), start, tokens, bs, blocks,
                                                            kv_heads * D * 2, stream))
        steps.append(lambda out=out: h.launch(q=q.data_ptr(), k=pool_k.data_ptr(), v=pool_v.data_ptr(), out=out.data_ptr(), batch=1, seq_q=tokens, seq_kv=keys, stream=stream,
                                              q_stride=(0, D, heads * D), o_stride=(0, D, heads * D), block_table=table.data_ptr(), block_table_stride=blocks, block_size=bs,
                                              num_blocks=blocks, workspace=ws.data_ptr(), workspace_bytes=ws.numel()))
    _same_bits(steps, lambda: outs)
    h.poll(stream)
    h.close()


@pytest.mark.parametrize("B,Hq,Hkv,Sk,D", [(70, 4, 4, 353, 128), (40, 24, 3, 1500, 64), (16, 4, 2, 900, 128)])
@pytest.mark.parametrize("rewritten", [False, True])
def test_decodes_of_changing_lengths(B, Hq, Hkv, Sk, D, rewritten):
    """Decodes through one workspace with other lengths each, in tensors of their own or in one that a copy rewrites between the calls."""
    stream = torch.cuda.current_stream().cuda_stream
    q, k, v = (gen(shape, "bf16", i)[0] for i, shape in enumerate(((B, Hq, 1, D), (B, Hkv, Sk, D), (B, Hkv, Sk, D))))
    rng = np.random.default_rng(2)
    lens = [torch.from_numpy(rng.integers(1, Sk + 1, B).astype(np.int32)).cuda() for _ in range(5)]
    shared = torch.empty_like(lens[0])
    outs = [torch.empty(B, Hq, D, device="cuda") for _ in lens]
    h = N.Handle(device=0, qkv_dtype=N.BF16, out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv)
    ws = torch.empty(max(h.workspace_bytes(B, 1, Sk), 16), dtype=torch.uint8, device="cuda")
    steps = []
    for n, out in zip(lens, outs):
        if rewritten:
            steps.append(lambda n=n: shared.copy_(n))
        steps.append(lambda n=n, out=out: h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=1, seq_kv=Sk, stream=stream,
                                                   kv_len=(shared if rewritten else n).data_ptr(), workspace=ws.data_ptr(), workspace_bytes=ws.numel()))
    _same_bits(steps, lambda: outs)
    h.poll(stream)
    h.close()


@pytest.mark.parametrize("B,S,heads,d", [(8, 197, 16, 32), (13, 100, 20, 40), (1, 100, 20, 20)])
def test_layers_of_different_weights(B, S, heads, d):
    """fp32 layers through one workspace, where the terms of the weights of the layer before still lie, each on the output of the one before."""
    stream = torch.cuda.current_stream().cuda_stream
    Dm = heads * d
    weights = [[gen((Dm, Dm), "f32", 10 * i + j, 2.0 * Dm ** -0.5)[0] for j in range(4)] for i in range(4)]
    acts = [gen((B, S, Dm), "f32", 1, 1.0)[0]] + [torch.empty(B, S, Dm, device="cuda") for _ in weights]
    h = N.Handle(device=0, qkv_dtype=N.F32, out_dtype=N.F32, head_dim=d, num_q_heads=heads, num_kv_heads=heads)
    nb = h.mha_workspace_bytes(B, S, N.F32, N.F32)
    ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) // 256 * 256
    steps = [lambda w=w, x=x, y=y: h.mha_forward(input=x.data_ptr(), q_weight=w[0].data_ptr(), k_weight=w[1].data_ptr(), v_weight=w[2].data_ptr(),
                                                 out_weight=w[3].data_ptr(), out=y.data_ptr(), batch=B, seq=S, input_dtype=N.F32, weight_dtype=N.F32, out_dtype=N.F32,
                                                 workspace=base, workspace_bytes=nb, stream=stream)
             for w, x, y in zip(weights, acts, acts[1:])]
    _same_bits(steps, lambda: acts[1:])
    h.poll(stream)
    h.close()


@pytest.fixture(scope="module")
def early_trigger(tmp_path_factory):
    """(milliseconds, stream): enqueues a launch of one thread that lets dependent ones begin and then takes that long."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    lib = str(tmp_path_factory.mktemp("cuda") / "early_trigger.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda", "early_trigger.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", lib, src], check=True, capture_output=True)
    call = ctypes.CDLL(lib).early_trigger
    call.argtypes = [ctypes.c_int, ctypes.c_void_p]

    def enqueue(ms, stream):
        assert call(ms, stream) == 0
    return enqueue


@pytest.mark.parametrize("kind", ["prefill", "layer", "fp32", "backward"])
def test_bounded_waits_count_their_own_time(kind, early_trigger):
    """A launch that is set up beside one of 2.4 s, above the 2 s that any wait may take: none of its waits runs out."""
    stream = torch.cuda.current_stream().cuda_stream
    B, H, S, D = 1, 4, 300, 64
    dtype = N.F32 if kind == "fp32" else N.BF16
    q, k, v, g = (gen((B, H, S, D), "f32" if kind == "fp32" else "bf16", i)[0] for i in range(4))
    weights = [gen((H * D, H * D), "bf16", 10 + i, (H * D) ** -0.5)[0] for i in range(4)]
    out, lse = torch.empty(B, H, S, D, device="cuda"), torch.empty(B, H, S, device="cuda")
    grads = [torch.empty(B, H, S, D, device="cuda") for _ in range(3)]
    h = N.Handle(device=0, qkv_dtype=dtype, out_dtype=N.BF16 if kind == "layer" else N.F32, head_dim=D, num_q_heads=H, num_kv_heads=H, emit_lse=kind == "backward")
    ws = torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 256 == 0
    common = dict(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=S, seq_kv=S, stream=stream,
                  lse=lse.data_ptr() if kind == "backward" else None)
    if kind == "layer":
        run = lambda: h.mha_forward(input=q.data_ptr(), q_weight=weights[0].data_ptr(), k_weight=weights[1].data_ptr(), v_weight=weights[2].data_ptr(),
                                    out_weight=weights[3].data_ptr(), out=out.data_ptr(), batch=B, seq=S, input_dtype=N.BF16, weight_dtype=N.BF16, out_dtype=N.F32,
                                    workspace=ws.data_ptr(), workspace_bytes=ws.numel(), stream=stream)
    elif kind == "backward":
        h.launch(**common)
        g = g.float()
        run = lambda: h.backward(dout=g.data_ptr(), dq=grads[0].data_ptr(), dk=grads[1].data_ptr(), dv=grads[2].data_ptr(), workspace=ws.data_ptr(),
                                 workspace_bytes=ws.numel(), **common)
    else:
        run = lambda: h.launch(**common)
    results = grads if kind == "backward" else [out]
    run()
    h.poll(stream)
    want = [t.clone() for t in results]
    for t in results:
        t.fill_(float("nan"))
    torch.cuda.synchronize()
    early_trigger(2400, stream)
    run()
    h.poll(stream)
    for got, ref in zip(results, want):
        assert torch.equal(got, ref)
    h.close()
