"""fp32 attention and projections from three bf16 terms (csrc/sdpa_f32_sm100.cu, sdpa_backward_f32_sm100.cu, proj_gemm_f32_sm100.cu) where
they can go wrong: one row or key more or less than a tile, every number of k steps, one to eight CTAs per tile, every mask kind,
values that are not finite, waits that run out, and the line between these kernels and the register-tiled ones."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import compare, compare_lse, gen, run_gpu

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Sq, Sk, D): many heads keep a tile in one CTA, few cut its keys over up to eight
SHAPES = [(2, 40, 40, 129, 257, 64), (1, 2, 1, 128, 520, 64), (1, 2, 2, 127, 449, 20), (2, 80, 20, 130, 321, 32), (1, 4, 2, 257, 511, 80),
          (3, 30, 30, 100, 385, 96), (1, 8, 4, 16, 1025, 128), (2, 40, 40, 200, 330, 100), (1, 3, 3, 320, 64, 64), (2, 4, 2, 330, 515, 64)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("variant", ["plain", "causal", "lengths", "keep", "keep_f32", "bias", "softcap", "bias_softcap"])
def test_forward(shape, variant):
    """Within the contract's tolerance of float64.  The log-sum-exp, which only long sequences get from these kernels, is that of
    the same call; the output without it is the kernels' own for every shape."""
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
        lens[0] = Sk - 1
        for b in range(B):                                    # what lies beyond a sequence's keys must never matter
            k[b, :, lens[b]:], v[b, :, lens[b]:] = float("nan"), float("inf")
        kw, okw = dict(kv_len=torch.from_numpy(lens).cuda()), dict(kv_len=lens)
    elif variant in ("keep", "keep_f32"):
        keep = (rng.random((1, Hq, Sq, Sk)) < 0.7).astype(np.uint8)
        keep[:, :, Sq // 2] = 0                               # a row that sees nothing
        keep[:, 0, :, : Sk // 2] = 0                          # a head whose first blocks hold nothing
        kind = N.MASK_KEEP_U8 if variant == "keep" else N.MASK_KEEP_F32
        dev = torch.from_numpy(keep).cuda()
        kw, okw = dict(mask=dev if variant == "keep" else dev.float(), mask_kind=kind), dict(mask=keep, mask_kind=O.MASK_KEEP_U8)
    elif variant == "bias" or variant == "bias_softcap":
        bias = rng.standard_normal((B, 1, Sq, Sk)).astype(np.float32)
        bias[..., ::7] = -np.inf
        bias[..., 1] = np.finfo(np.float32).min
        kw, okw = dict(mask=torch.from_numpy(bias).cuda(), mask_kind=N.MASK_ADD_F32), dict(mask=bias, mask_kind=O.MASK_ADD_F32)
    if "softcap" in variant:
        kw["softcap"] = okw["softcap"] = 20.0
    out, _, _ = run_gpu(q, k, v, dtype="f32", **kw)
    with_lse, lse, _ = run_gpu(q, k, v, dtype="f32", want_lse=True, **kw)
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, **okw)
    compare(out, ref, "f32", f"{shape} {variant}")
    compare(with_lse, ref, "f32", f"{shape} {variant}")
    compare_lse(lse, ref_lse, "f32", f"{shape} {variant}")
    again, _, _ = run_gpu(q, k, v, dtype="f32", **kw)
    assert torch.equal(out, again)


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("where", ["q", "k", "v", "v_masked", "k_masked"])
@pytest.mark.parametrize("heads", [2, 80])
def test_forward_non_finite(value, where, heads):
    """What is not a number or infinite in one row comes out where the fp32 kernels (path generic) bring it out."""
    B, S, D = 2, 300, 64
    q, _ = gen((B, heads, S, D), "f32", 1, 1.0)
    k, _ = gen((B, heads, S, D), "f32", 2, 1.0)
    v, _ = gen((B, heads, S, D), "f32", 3, 1.0)
    kw = {}
    if "masked" in where:
        keep = torch.ones((1, 1, S, S), dtype=torch.uint8, device="cuda")
        keep[..., 7] = 0
        kw = dict(mask=keep, mask_kind=N.MASK_KEEP_U8)
    {"q": q, "k": k, "v": v}[where[0]][1, 1, 7, 5] = value
    got, _, _ = run_gpu(q, k, v, dtype="f32", **kw)
    want, _, _ = run_gpu(q, k, v, dtype="f32", path=N.PATH_GENERIC, **kw)
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(test(got), test(want))
    fin = torch.isfinite(want)
    assert (got - want)[fin].abs().max() <= 1e-5


@pytest.mark.parametrize("D", [32, 64, 80, 128])
@pytest.mark.parametrize("heads", [2, 80])
@pytest.mark.parametrize("variant", ["plain", "bias", "softcap"])
def test_forward_keys_of_weight_zero(D, heads, variant):
    """Infinite keys whose logits are -infinity for every row, in either half of a block or in both: their weight is 0, and no row may
    become NaN, whichever of the two warps of a row is first.  (With a softcap tanh makes them -20, an ordinary logit.)"""
    B, Sq, Sk = 2, 200, 330
    q, _ = gen((B, heads, Sq, D), "f32", 1, 1.0)
    k, _ = gen((B, heads, Sk, D), "f32", 2, 1.0)
    v, vf = gen((B, heads, Sk, D), "f32", 3, 1.0)
    q[..., 0] = -q[..., 0].abs() - 0.1
    for key in (7, 8, 40, 100, 200, 205, 250, 329):
        k[..., key, 0] = float("inf")
    kw = dict(softcap=20.0) if variant == "softcap" else {}
    s = (q.double() @ k.double().transpose(-1, -2)) / np.sqrt(D)
    if variant == "bias":
        bias = torch.randn((1, 1, Sq, Sk), device="cuda", generator=torch.Generator("cuda").manual_seed(4))
        kw, s = dict(mask=bias, mask_kind=N.MASK_ADD_F32), s + bias
    if variant == "softcap":
        s = 20 * torch.tanh(s / 20)
    want = torch.softmax(s, -1) @ v.double()
    first = None
    for _ in range(20):
        got, _, _ = run_gpu(q, k, v, dtype="f32", **kw)
        assert (got - want).abs().max() <= 1e-5 * want.abs().max()
        first = got if first is None else first
        assert torch.equal(got, first)


@pytest.mark.parametrize("D", [32, 64, 80, 128])
@pytest.mark.parametrize("heads", [2, 80])
def test_forward_logits_from_the_largest_floats(D, heads):
    """Finite elements above the largest bf16 (3.39e38) against queries that make ordinary logits of them."""
    B, Sq, Sk = 2, 200, 330
    q, _ = gen((B, heads, Sq, D), "f32", 1, 1.0)
    k, _ = gen((B, heads, Sk, D), "f32", 2, 1.0)
    v, _ = gen((B, heads, Sk, D), "f32", 3, 1.0)
    q[..., 3] = q[..., 3] * 2e-38
    k[..., ::5, 3] = torch.finfo(torch.float32).max
    k[..., 1::7, 3] = torch.finfo(torch.float32).min
    want = torch.softmax((q.double() @ k.double().transpose(-1, -2)) / np.sqrt(D), -1) @ v.double()
    got, _, _ = run_gpu(q, k, v, dtype="f32")
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()


@pytest.mark.parametrize("D", [32, 64, 80, 128])
@pytest.mark.parametrize("heads", [2, 80])
@pytest.mark.parametrize("variant", ["plain", "keep", "bias_softcap"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 3.4e38])
def test_forward_values_reach_the_rows_that_see_them(D, heads, variant, value):
    """Under a causal mask with lengths, a value that is not finite, or above the largest bf16, in some columns of V: rows before
    the key come out as if it were not there, and those that see it as float64 has them."""
    B, Sq, Sk, offset = 2, 300, 330, 20
    q, _ = gen((B, heads, Sq, D), "f32", 1, 1.0)
    k, _ = gen((B, heads, Sk, D), "f32", 2, 1.0)
    v, _ = gen((B, heads, Sk, D), "f32", 3, 1.0)
    lens = torch.tensor([Sk, 290], dtype=torch.int32, device="cuda")
    s = (q.double() @ k.double().transpose(-1, -2)) / np.sqrt(D)
    key, row = torch.arange(Sk, device="cuda"), torch.arange(Sq, device="cuda")
    seen = (key[None, None, None] <= row[None, None, :, None] + offset) & (key[None, None, None] < lens[:, None, None, None])
    kw = {}
    if variant == "keep":
        keep = (torch.rand((1, 1, Sq, Sk), device="cuda", generator=torch.Generator("cuda").manual_seed(4)) < 0.9).to(torch.uint8)
        keep[..., [5, 77, 190, 299]] = 1
        kw, seen = dict(mask=keep, mask_kind=N.MASK_KEEP_U8), seen & (keep != 0)
    elif variant == "bias_softcap":
        bias = torch.randn((1, 1, Sq, Sk), device="cuda", generator=torch.Generator("cuda").manual_seed(4))
        kw, s = dict(mask=bias, mask_kind=N.MASK_ADD_F32, softcap=20.0), 20 * torch.tanh(s / 20) + bias
    w = torch.softmax(s.masked_fill(~seen, -torch.inf), -1)
    clean = w @ v.double()
    places = [(5, 0), (77, D - 1), (190, 9), (299, 17)]
    for j, c in places:
        v[:, :, j, c] = value
    want = clean.clone()
    for j, c in places:   # what the key adds (beside which its old value does not count), to the rows that see it
        want[..., c] = torch.where(seen[..., j].expand(B, heads, Sq), clean[..., c] + w[..., j] * value, clean[..., c])
    got, _, _ = run_gpu(q, k, v, dtype="f32", causal=True, bottom_right=False, causal_offset=offset, kv_len=lens, **kw)
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(test(got), test(want.float()))
    fin = torch.isfinite(want.float())
    assert ((got - want).abs()[fin] <= 1e-5 * want.abs()[fin].clamp(min=2.0)).all()


BWD_SHAPES = [(1, 4, 4, 320, 320, 64), (1, 4, 2, 321, 449, 64), (2, 30, 30, 400, 385, 64), (1, 2, 2, 513, 640, 32), (2, 12, 6, 511, 450, 36),
              (1, 8, 4, 390, 700, 20)]


@pytest.mark.parametrize("shape", BWD_SHAPES)
@pytest.mark.parametrize("variant", ["plain", "causal", "keep_lengths", "keep_f32", "bias"])
def test_backward(shape, variant):
    """dQ, dK, dV against float64: 16 x 2^-24 x sqrt(n) of the largest value, as for the register-tiled kernels."""
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
    elif variant == "keep_f32":
        keep = (rng.random((B, 1, Sq, Sk)) < 0.8).astype(np.uint8)
        kw, okw = dict(mask=torch.from_numpy(keep).cuda().float(), mask_kind=N.MASK_KEEP_F32), dict(keep=keep)
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


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("heads", [2, 30])
@pytest.mark.parametrize("where", ["q", "k", "v", "dout"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 3.4e38])
def test_backward_values_reach_the_pairs_that_take_part(D, heads, where, value):
    """Under a causal mask with lengths: the gradients of rows and keys that take no part with a row (of Q, dO) or a key (of K, V)
    that holds something that is not finite, or above the largest bf16, are those without it."""
    from tests.test_gpu_backward import _fwd_bwd
    B, Sq, Sk, offset, row, key, col = 2, 400, 420, 10, 150, 160, 9
    (q, qf), (k, kf), (v, vf), (g, gf) = [gen((B, heads, S, D), "f32", i + 1, 1.0) for i, S in enumerate([Sq, Sk, Sk, Sq])]
    lens = np.array([Sk, 330], np.int32)
    if where in ("q", "dout"):
        gf = gf.copy()
        gf[:, :, row] = 0                       # the row adds nothing
    want = [x.astype(np.float64) for x in O.sdpa_backward(qf, kf, vf, gf, causal=True, causal_offset=offset, kv_len=lens)[:3]]
    {"q": q, "k": k, "v": v, "dout": g}[where][:, :, row if where in ("q", "dout") else key, col] = value
    got = [x.cpu().numpy() for x in _fwd_bwd(q, k, v, g, dtype="f32", causal=True, causal_offset=offset, kv_len=lens)]
    if where in ("q", "dout"):
        rows, keys = np.arange(Sq) != row, np.arange(Sk) > row + offset
    else:
        rows, keys = np.arange(Sq) + offset < key, np.arange(Sk) < 0
    for x, y, name, part in zip(got, want, ("dQ", "dK", "dV"), (rows, keys, keys)):
        x, y = x[:, :, part], y[:, :, part]
        assert np.isfinite(x).all(), name
        assert np.abs(x - y).max(initial=0) <= 16 * 2.0 ** -24 * np.sqrt(Sk) * max(1.0, np.abs(y).max(initial=0)), name
    if where == "dout":                         # and in dV nothing but the value's column changes
        dv, seen = got[2], np.arange(Sk) <= row + offset
        other = np.delete(dv, col, axis=3)
        assert np.isfinite(other).all()
        if np.isfinite(value):
            assert (dv[:, :, seen, col] > 1e30).all()
        else:
            assert (np.isnan(dv[:, :, seen, col]) if np.isnan(value) else dv[:, :, seen, col] == value).all()


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("heads", [2, 30])
def test_backward_infinite_value_in_v(D, heads):
    """One infinity in V makes the row sums of dO * O infinite and with them dS of every other key: with positive Q and dO its dK is
    -infinity, not NaN; dV does not know of it."""
    from tests.test_gpu_backward import _fwd_bwd
    B, S, key = 1, 350, 200
    (q, qf), (k, kf), (v, vf), (g, gf) = [gen((B, heads, S, D), "f32", i + 1, 1.0) for i in range(4)]
    q, g, qf, gf = q.abs(), g.abs(), np.abs(qf), np.abs(gf)
    v[:, :, key, 5] = float("inf")
    dq, dk, dv = _fwd_bwd(q, k, v, g, dtype="f32")
    others = torch.arange(S, device="cuda") != key
    assert torch.isneginf(dk[:, :, others]).all() and torch.isnan(dk[:, :, key]).all() and torch.isnan(dq).all()
    want = O.sdpa_backward(qf, kf, vf, gf)[2]
    assert np.abs(dv.cpu().numpy() - want).max() <= 16 * 2.0 ** -24 * np.sqrt(S) * np.abs(want).max()


def _times_out(h, launch):
    """Whether the call runs on a tcgen05 kernel: with the time-out hook those load nothing, and their bounded waits (20 ms) run out,
    which poll reports.  The same call without the hook then has to succeed."""
    stream = torch.cuda.current_stream().cuda_stream
    h.debug_set(None, 3)
    launch()
    try:
        h.poll(stream)
        expired = False
    except N.AidnError as e:
        assert e.status == N.ETIMEOUT
        expired = True
    h.debug_set(None, 0)
    launch()
    h.poll(stream)
    return expired


# (B, H, Sq, Sk, D, softcap, with log-sum-exp) and whether the call is large enough for the tcgen05 kernel
ROUTES = [((1, 2, 16, 64, 64, 0.0, False), True), ((1, 2, 16, 63, 64, 0.0, False), False),
          ((2, 80, 128, 64, 64, 0.0, False), True), ((2, 80, 128, 63, 64, 0.0, False), False),
          ((1, 2, 16, 129, 128, 0.0, False), True), ((1, 2, 16, 128, 128, 0.0, False), False),
          ((2, 80, 16, 128, 128, 0.0, False), True), ((2, 80, 16, 127, 128, 0.0, False), False),
          ((1, 2, 16, 257, 128, 20.0, False), True), ((1, 2, 16, 256, 128, 20.0, False), False),
          ((2, 80, 32, 128, 128, 20.0, False), True), ((2, 80, 32, 127, 128, 20.0, False), False),
          ((1, 2, 16, 257, 32, 20.0, False), True), ((1, 2, 16, 256, 32, 20.0, False), False),
          ((1, 2, 320, 320, 64, 0.0, True), True), ((1, 2, 320, 319, 64, 0.0, True), False), ((1, 2, 319, 320, 64, 0.0, True), False),
          ((1, 2, 400, 400, 80, 0.0, True), False)]


@pytest.mark.parametrize("call,tcgen05", ROUTES)
@pytest.mark.parametrize("path", [N.PATH_AUTO, N.PATH_GENERIC])
def test_forward_route_and_bounded_waits(call, tcgen05, path):
    """Both sides of every line of the rule run where they should, path GENERIC on multiply-adds; and the tcgen05 kernel unwinds when its
    waits run out: TMEM is given back, clusters part, and the next call on the handle is correct."""
    B, H, Sq, Sk, D, softcap, want_lse = call
    (q, qf), (k, kf), (v, vf) = [gen((B, H, S, D), "f32", i + 1, 1.0) for i, S in enumerate([Sq, Sk, Sk])]
    out, lse = torch.zeros((B, H, Sq, D), device="cuda"), torch.zeros((B, H, Sq), device="cuda")
    h = N.Handle(device=0, qkv_dtype=N.F32, head_dim=D, num_q_heads=H, num_kv_heads=H, softcap=softcap, emit_lse=want_lse, path=path)
    launch = lambda: h.launch(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk,
                              lse=lse.data_ptr() if want_lse else None, stream=torch.cuda.current_stream().cuda_stream)
    assert _times_out(h, launch) == (tcgen05 and path == N.PATH_AUTO)
    h.close()
    compare(out, O.sdpa(qf, kf, vf, softcap=softcap), "f32", str(call))


@pytest.mark.parametrize("shape,tcgen05", [((1, 2, 320, 320, 64), True), ((1, 40, 320, 321, 32), True), ((1, 2, 319, 320, 64), False),
                                           ((1, 2, 320, 319, 64), False), ((1, 2, 400, 400, 68), False)])
@pytest.mark.parametrize("path", [N.PATH_AUTO, N.PATH_GENERIC])
def test_backward_route_and_bounded_waits(shape, tcgen05, path):
    B, H, Sq, Sk, D = shape
    (q, qf), (k, kf), (v, vf), (g, gf) = [gen((B, H, S, D), "f32", i + 1, 1.0) for i, S in enumerate([Sq, Sk, Sk, Sq])]
    out, lse = torch.zeros((B, H, Sq, D), device="cuda"), torch.zeros((B, H, Sq), device="cuda")
    grads = [torch.zeros_like(x) for x in (q, k, v)]
    h = N.Handle(device=0, qkv_dtype=N.F32, head_dim=D, num_q_heads=H, num_kv_heads=H, emit_lse=True, path=path)
    ws = torch.empty(h.backward_workspace_bytes(B, Sq), dtype=torch.uint8, device="cuda")
    common = dict(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), out=out.data_ptr(), lse=lse.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk,
                  stream=torch.cuda.current_stream().cuda_stream)
    h.launch(**common)
    launch = lambda: h.backward(dout=g.data_ptr(), dq=grads[0].data_ptr(), dk=grads[1].data_ptr(), dv=grads[2].data_ptr(),
                                workspace=ws.data_ptr(), workspace_bytes=ws.numel(), **common)
    assert _times_out(h, launch) == (tcgen05 and path == N.PATH_AUTO)
    h.close()
    for x, y, name in zip(grads, O.sdpa_backward(qf, kf, vf, gf)[:3], ("dQ", "dK", "dV")):
        assert np.abs(x.cpu().numpy() - y).max() <= 16 * 2.0 ** -24 * np.sqrt(max(Sq, Sk, D)) * max(1.0, np.abs(y).max()), name


def _layer(x, ws, heads, path=N.PATH_AUTO, workspace=None):
    B, S, Dm = x.shape
    out = torch.full((B, S, Dm), float("nan"), device="cuda")
    h = N.Handle(device=0, qkv_dtype=N.F32, out_dtype=N.F32, head_dim=Dm // heads, num_q_heads=heads, num_kv_heads=heads, path=path)
    nb = h.mha_workspace_bytes(B, S, N.F32, N.F32) if workspace is None else workspace
    scratch = torch.zeros(nb + 1024, dtype=torch.uint8, device="cuda")
    launch = lambda: h.mha_forward(input=x.data_ptr(), q_weight=ws[0].data_ptr(), k_weight=ws[1].data_ptr(), v_weight=ws[2].data_ptr(),
                                   out_weight=ws[3].data_ptr(), out=out.data_ptr(), batch=B, seq=S, input_dtype=N.F32, weight_dtype=N.F32,
                                   out_dtype=N.F32, workspace=(scratch.data_ptr() + 1023) // 1024 * 1024, workspace_bytes=nb,
                                   stream=torch.cuda.current_stream().cuda_stream)
    return h, launch, out


@pytest.mark.parametrize("heads,d,tcgen05", [(4, 64, True), (3, 84, False), (5, 52, True), (6, 62, True), (3, 100, True), (7, 54, False), (9, 36, True)])
@pytest.mark.parametrize("B,S", [(1, 1), (1, 127), (3, 43), (8, 197)])
def test_projections(heads, d, tcgen05, B, S):
    """Widths off the tiles of 64 or 128 columns and the K blocks of 64, head sizes that are not multiples of 4, rows on both sides of 128:
    the layer against float64.  Every matrix adds 2^-24 x sqrt(width) x 4 of its largest element (three terms are exact to 2^-26 of a
    product; four truncated additions a block), three of them in a row: 1e-5 of the largest output is above that at width 512."""
    Dm = heads * d
    x, xf = gen((B, S, Dm), "f32", 1, 1.0)
    ws, wfs = zip(*[gen((Dm, Dm), "f32", 2 + i, Dm ** -0.5) for i in range(4)])
    h, launch, out = _layer(x, ws, heads)
    want = O.mha_forward(xf, *wfs, heads)
    launch()
    h.poll(torch.cuda.current_stream().cuda_stream)
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    if S == 1:   # (one key: the attention itself is too small for a tcgen05 kernel)
        assert _times_out(h, launch) == tcgen05
    h.close()


@pytest.mark.parametrize("B,S,heads,d", [(1, 100, 20, 20), (1, 127, 25, 40), (1, 1, 241, 4), (2, 70, 32, 64), (27, 19, 17, 32), (8, 125, 20, 38), (13, 100, 20, 40),
                                         (4, 100, 32, 64), (7, 100, 8, 109), (5, 77, 16, 48), (8, 250, 41, 20), (8, 250, 11, 40), (3, 100, 137, 8), (12, 50, 20, 54),
                                         (8, 250, 37, 8)])
def test_projection_plans(B, S, heads, d):
    """Every tile width (32 to 160 columns), weights cut in place and by a launch of their own, K over 1, 2, 4 and 8 CTAs of a cluster, widths and
    K off the tiles: the layer against float64, and the same bits again.  Bound: test_projections' 2^-24 x sqrt(width) x 4 a matrix."""
    Dm = heads * d
    x, xf = gen((B, S, Dm), "f32", 1, 1.0)
    ws, wfs = zip(*[gen((Dm, Dm), "f32", 2 + i, Dm ** -0.5) for i in range(4)])
    h, launch, out = _layer(x, ws, heads)
    want = O.mha_forward(xf, *wfs, heads)
    launch()
    first = out.clone()
    out.fill_(float("nan"))
    launch()
    h.poll(torch.cuda.current_stream().cuda_stream)
    assert np.abs(first.cpu().numpy() - want).max() <= 12 * 2.0 ** -24 * Dm ** 0.5 * np.abs(want).max()
    assert torch.equal(first, out)
    # a cluster's merge, too, stores nothing that an expired wait left behind, and the next call is whole again
    out.fill_(7.0)
    h.debug_set(None, 3)
    launch()
    with pytest.raises(N.AidnError):
        h.poll(torch.cuda.current_stream().cuda_stream)
    assert (out == 7.0).all()
    h.debug_set(None, 0)
    launch()
    h.poll(torch.cuda.current_stream().cuda_stream)
    assert torch.equal(first, out)
    h.close()


@pytest.mark.parametrize("B,S,heads,d", [(8, 197, 16, 32), (13, 100, 20, 40), (8, 250, 11, 40)])
def test_projections_without_room_for_the_images(B, S, heads, d):
    """The weights' terms are an offer: a workspace of the activations alone (Q, K, V and the attention's output), or one byte short of
    what is asked for, gives the same layer with the weights cut in place; less is refused.  Bound: test_projection_plans'."""
    Dm = heads * d
    x, xf = gen((B, S, Dm), "f32", 1, 1.0)
    ws, wfs = zip(*[gen((Dm, Dm), "f32", 2 + i, Dm ** -0.5) for i in range(4)])
    want = O.mha_forward(xf, *wfs, heads)
    with N.Handle(device=0, qkv_dtype=N.F32, out_dtype=N.F32, head_dim=d, num_q_heads=heads, num_kv_heads=heads) as h:
        asked = h.mha_workspace_bytes(B, S, N.F32, N.F32)
    least = 4 * ((B * S * Dm * 4 + 1023) // 1024 * 1024)
    assert asked > least
    for nbytes, launches in ((asked, 4), (asked - 1, 3), (least, 3)):
        h, launch, out = _layer(x, ws, heads, workspace=nbytes)
        launch()
        h.poll(torch.cuda.current_stream().cuda_stream)
        assert h.last_launch_count == launches
        assert np.abs(out.cpu().numpy() - want).max() <= 12 * 2.0 ** -24 * Dm ** 0.5 * np.abs(want).max()
        h.close()
    h, launch, out = _layer(x, ws, heads, workspace=least - 1)
    with pytest.raises(N.AidnError) as error:
        launch()
    assert error.value.status == N.EWORKSPACE
    h.close()


@pytest.mark.parametrize("heads,d,S", [(4, 64, 130), (5, 52, 130), (16, 32, 1000)])
def test_projections_of_values_that_are_not_finite(heads, d, S):
    """In the output weight, in columns of their own: an infinity gives infinities of the sign of what it meets, NaN gives NaN, a value
    above the largest bf16 a finite sum, and no other column changes.  A row of NaN in one sequence leaves the others alone."""
    B, Dm = 2, heads * d
    x, xf = gen((B, S, Dm), "f32", 1, 1.0)
    ws, wfs = zip(*[gen((Dm, Dm), "f32", 2 + i, Dm ** -0.5) for i in range(4)])
    _, launch, attended = _layer(x, [*ws[:3], torch.eye(Dm, device="cuda")], heads)
    launch()
    torch.cuda.synchronize()
    w = ws[3].clone()
    for c, value in ((0, float("inf")), (Dm // 2 + 1, float("-inf")), (77, float("nan")), (Dm - 1, 3.4e38)):
        w[c // 2, c] = value
    _, launch, out = _layer(x, [*ws[:3], w], heads)
    launch()
    torch.cuda.synchronize()
    want = attended.double() @ w.double()
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(test(out), test(want.float()))
    fin = torch.isfinite(want)
    fin[..., Dm - 1] = False
    assert (out - want)[fin].abs().max() <= 1e-5 * want[fin].abs().max()
    assert (out - want)[..., Dm - 1].abs().max() <= 1e-5 * want[..., Dm - 1].abs().max()
    y = x.clone()
    y[1, S // 2] = float("nan")
    _, launch, out = _layer(y, ws, heads)
    launch()
    torch.cuda.synchronize()
    ref = O.mha_forward(xf[:1], *wfs, heads)
    assert np.abs(out[:1].cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max() and torch.isnan(out[1]).all()


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(1, 2, 2, 512, 640), (2, 6, 2, 350, 400), (2, 8, 8, 130, 700)])
@pytest.mark.parametrize("swapped", [False, True])
def test_backward_gradients_over_keys(B, Hq, Hkv, Sq, Sk, swapped):
    """dK and dV in the place of K and V, or of V and K: the same bits as in buffers of their own, dQ too."""
    D = 64
    q, k, v, g = (gen((B, H, S, D), "f32", i, 1.0)[0] for i, (H, S) in enumerate(((Hq, Sq), (Hkv, Sk), (Hkv, Sk), (Hq, Sq))))
    out, lse = torch.empty(B, Hq, Sq, D, device="cuda"), torch.empty(B, Hq, Sq, device="cuda")
    with N.Handle(device=0, qkv_dtype=N.F32, out_dtype=N.F32, head_dim=D, num_q_heads=Hq, num_kv_heads=Hkv, emit_lse=True) as h:
        stream = torch.cuda.current_stream().cuda_stream
        ws = torch.empty(h.backward_workspace_bytes(B, Sq), dtype=torch.uint8, device="cuda")
        dq = [torch.empty_like(q) for _ in range(2)]
        dk, dv = torch.empty_like(k), torch.empty_like(v)
        k2, v2 = k.clone(), v.clone()
        common = dict(q=q.data_ptr(), out=out.data_ptr(), lse=lse.data_ptr(), batch=B, seq_q=Sq, seq_kv=Sk, stream=stream)
        h.launch(k=k.data_ptr(), v=v.data_ptr(), **common)
        for dq_, k_, v_, dk_, dv_ in ((dq[0], k, v, dk, dv), (dq[1], k2, v2, *((v2, k2) if swapped else (k2, v2)))):
            h.backward(k=k_.data_ptr(), v=v_.data_ptr(), dout=g.data_ptr(), dq=dq_.data_ptr(), dk=dk_.data_ptr(), dv=dv_.data_ptr(), workspace=ws.data_ptr(),
                       workspace_bytes=ws.numel(), **common)
        h.poll(stream)
    assert torch.equal(dq[0], dq[1])
    assert torch.equal(dk, v2 if swapped else k2) and torch.equal(dv, k2 if swapped else v2)
