"""Decode launches whose splits are the CTAs of a cluster (csrc/sdpa_decode.cu, decode_plan_clusters): every plan - 8, 4 and 2 CTAs,
several clusters with the merge kernel, the FP32 units - at lengths where a CTA, a cluster or a whole sequence has no key, and
sequences that are not in the order in which they are started."""
import numpy as np
import pytest
import torch

from aidotnet.tensors_b200 import native as N
from oracle import sdpa_oracle as O

from tests._harness import compare, compare_lse, gen, run_gpu

pytestmark = pytest.mark.gpu

# (B, Hq, Hkv, Sk, D, dtype, launches)
CASES = [(1, 4, 4, 1237, 64, "bf16", 1), (3, 8, 2, 700, 128, "f16", 1), (1, 16, 1, 600, 128, "bf16", 1), (20, 4, 2, 500, 128, "bf16", 1),
         (16, 8, 8, 300, 128, "bf16", 1), (40, 12, 4, 200, 64, "f16", 1), (2, 4, 2, 4400, 128, "bf16", 2), (1, 8, 8, 9000, 64, "bf16", 2),
         (2, 4, 4, 500, 64, "f32", 1), (1, 6, 2, 400, 128, "f32", 1), (1, 4, 4, 4000, 64, "f32", 2),
         (9, 48, 4, 600, 64, "bf16", 1), (12, 36, 4, 500, 64, "f16", 1)]   # more than eight heads: up to two CTAs an SM, and three


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("lengths", [False, True])
def test_cluster_decode(case, lengths):
    B, Hq, Hkv, Sk, D, dtype, launches = case
    scale = 1.0 if dtype == "f32" else 0.5
    q, qf = gen((B, Hq, 1, D), dtype, 1, scale)
    k, kf = gen((B, Hkv, Sk, D), dtype, 2, scale)
    v, vf = gen((B, Hkv, Sk, D), dtype, 3, scale)
    kw, okw = {}, {}
    if lengths:
        lens = np.random.default_rng(5).integers(0, Sk + 1, B).astype(np.int32)
        lens[0], lens[-1] = 17, Sk - 1                 # most of the CTAs have no key
        if B > 2:
            lens[1] = 0
        for b in range(B):                             # what lies beyond a sequence's keys must never matter
            k[b, :, lens[b]:], v[b, :, lens[b]:] = float("nan"), float("inf")
        kw, okw = dict(kv_len=torch.from_numpy(lens).cuda()), dict(kv_len=lens)
    out, lse, info = run_gpu(q, k, v, dtype=dtype, want_lse=True, path=N.PATH_DECODE, **kw)
    assert info["launches"] == launches
    ref, ref_lse, _ = O.sdpa(qf, kf, vf, want_lse=True, **okw)
    compare(out, ref, dtype, f"{case}")
    compare_lse(lse, ref_lse, dtype, f"{case}")
    again, _, _ = run_gpu(q, k, v, dtype=dtype, want_lse=True, path=N.PATH_DECODE, **kw)
    assert torch.equal(out, again)


@pytest.mark.parametrize("dtype,D,Sk", [("bf16", 64, 1200), ("f16", 128, 5000), ("f32", 64, 1200)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_clusters_keep_non_finite_values(dtype, D, Sk, value):
    """A visible NaN or infinity in V behind a weight that underflows to 0 (the largest logit, in another CTA, is 400 above it):
    0 * NaN is NaN, as in a launch of one split."""
    q, _ = gen((2, 4, 1, D), dtype, 1)
    k, _ = gen((2, 4, Sk, D), dtype, 2, 0.01)
    v, _ = gen((2, 4, Sk, D), dtype, 3)
    q[...] = 1.0
    k[:, :, 300] = 400.0 / D
    v[1, 3, Sk - 100, 7] = value
    split, _, info = run_gpu(q, k, v, dtype=dtype, path=N.PATH_DECODE, scale=1.0)
    one, _, info1 = run_gpu(q, k, v, dtype=dtype, path=N.PATH_DECODE, scale=1.0, decode_chunk=8192)
    assert info["launches"] == (2 if Sk == 5000 else 1) and info1["launches"] == 1
    assert torch.isnan(one[1, 3, 0, 7])
    assert torch.equal(torch.isnan(split), torch.isnan(one))


# (B, Hq, Hkv, D, dtype): keys on either side of a line of the plan, and the launches there (one: a cluster; two: a merge kernel)
LINES = [((33, 4, 1, 128, "bf16"), 3000, 1, 17000, 2), ((34, 2, 1, 128, "bf16"), 4000, 1, 8200, 2), ((50, 1, 1, 64, "bf16"), 4000, 1, 4200, 2),
         ((100, 1, 1, 128, "f16"), 2048, 1, 2049, 2), ((160, 1, 1, 128, "bf16"), 512, 1, 520, 2), ((8, 1, 1, 64, "f32"), 1280, 1, 1300, 2),
         ((74, 1, 1, 64, "f32"), 64, 1, 200, 2), ((6, 4, 1, 64, "f32"), 480, 1, 500, 2)]


@pytest.mark.parametrize("heads,below,launches_below,above,launches_above", LINES)
def test_plan_lines(heads, below, launches_below, above, launches_above):
    """Where clusters stop being faster than chunks with a merge kernel, both sides against float64."""
    B, Hq, Hkv, D, dtype = heads
    scale = 1.0 if dtype == "f32" else 0.5
    for Sk, launches in ((below, launches_below), (above, launches_above)):
        q, qf = gen((B, Hq, 1, D), dtype, 1, scale)
        k, kf = gen((B, Hkv, Sk, D), dtype, 2, scale)
        v, vf = gen((B, Hkv, Sk, D), dtype, 3, scale)
        out, _, info = run_gpu(q, k, v, dtype=dtype, path=N.PATH_DECODE)
        assert info["launches"] == launches, (heads, Sk)
        compare(out, O.sdpa(qf, kf, vf), dtype, f"{heads} {Sk}")
