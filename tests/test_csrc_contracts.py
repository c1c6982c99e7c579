"""Properties of the CUDA sources that no run can show: what a kernel promises the compiler."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "ceo_b200" / "csrc"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


# Cluster barriers and TMEM release are warp-aligned: after per-lane loops and one-lane roles the
# warp has to be brought together first.
@pytest.mark.parametrize("name,call", [("skinny.cu", "cluster_sync_all();"),
                                       ("gemm_tcgen05.cu", "cluster_sync();")])
def test_warps_are_whole_at_aligned_instructions(name, call):
    lines = [x.strip() for x in _code(name).splitlines() if x.strip()]
    at = [i for i, x in enumerate(lines) if x.endswith(call)]
    assert len(at) == 2
    for i in at:
        assert "__syncwarp();" in lines[i - 1], lines[i - 2:i + 1]


# A programmatic dependent launch is resident while the kernel before it still writes its inputs:
# of a chain kernel's pointers only weights may be declared read-only.
@pytest.mark.parametrize("kernel,weights", [("decode_rmsnorm_kernel", {"w"}),
                                            ("decode_delta_kernel", {"beta_scalar"})])
def test_chain_kernels_promise_read_only_weights_alone(kernel, weights):
    text = _code("decode.cu")
    params = re.search(kernel + r"\(([^)]*)\)\s*\{", text).group(1)
    fixed = {p.split()[-1] for p in params.split(",") if "const" in p and "__restrict__" in p}
    assert fixed == weights
    body = text[text.index(params):].split("\n}\n")[0]
    assert "__ldg" not in body and "ld.global.nc" not in body
