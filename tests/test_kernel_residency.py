"""Register counts that the plans rely on, from the resource report of the build."""
import os
import re

import pytest

from aidotnet.tensors_b200 import build

REGISTERS, THREADS = 65536, 128   # of an SM; of a decode CTA


def _registers():
    """Kernel name (mangled) -> registers of a thread."""
    path = os.path.join(build.BUILD, "ptxas.log")
    if not os.path.exists(path):
        pytest.skip("no resource report: the library was not built here")
    with open(path) as f:
        report = f.read()
    return {name: int(n) for name, n in re.findall(r"Compiling entry function '(\w+)' for 'sm_100a'.*?Used (\d+) registers", report, re.S)}


@pytest.mark.parametrize("kernel", ["sdpa_decode_gqa_ring_kernel", "sdpa_decode_stream_kernel"])
@pytest.mark.parametrize("dim,ctas", [(64, 3), (128, 2)])
def test_decode_ctas_fit_the_register_file(kernel, dim, ctas):
    """decode_plan_clusters and decode_stream_bytes count on that many CTAs of an SM at once, for every instantiation (but those of the ring kernel for
    launches of two CTAs an SM, whose last template argument says so)."""
    found = {k: r for k, r in _registers().items() if kernel in k and f"Li{dim}E" in k and ("stream" in k or f"Li{ctas}EE" in k)}
    assert found
    for name, r in found.items():
        assert REGISTERS // (-(-r // 8) * 8 * THREADS) >= ctas, f"{name}: {r} registers"
