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
