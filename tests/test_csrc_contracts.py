"""Properties of the CUDA sources that no run can show: what a kernel promises the compiler."""
import re
from pathlib import Path

import pytest

from ceo_b200.runtime.fault import describe_status

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


# The limit of bounded waits is kept per translation unit: ceo_set_wait_limit has to reach each
# unit that waits, and each code such a unit writes needs a name.
def test_wait_limit_and_status_codes_reach_every_unit():
    forward = re.search(r"int ceo_set_wait_limit\(unsigned int iterations\) \{(.*?)\n\}",
                        _code("comm.cu"), re.S).group(1)
    for src in sorted(CSRC.glob("*.cu")):
        text = _code(src.name)
        if not re.search(r"\b(mbar_wait|wait_limit)\(", text):
            continue
        own = re.findall(r"(\w+)\(unsigned int iterations\) \{\s*return ceo::set_wait_limit", text)
        assert src.name == "comm.cu" or (len(own) == 1 and own[0] + "(iterations)" in forward), src
        for code in re.findall(r"\b\w*STATUS = (0x[0-9A-Fa-f]+);", text):
            assert "status" not in describe_status(int(code, 16)), (src, code)
