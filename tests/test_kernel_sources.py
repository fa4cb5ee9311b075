"""Rules of the kernels' sources that no run can show (no GPU)."""

import os
import re

import pytest

from llm_pipeline_b200.ops.build import CSRC


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_a_warp_meets_before_an_aligned_cluster_barrier(name):
    """``barrier.cluster.arrive.aligned`` is for whole warps: behind a ``continue``, by which lanes leave an iteration early, the
    source says that they meet again first."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for barrier in re.finditer(r"cluster_sync_all\(\);|barrier\.cluster\.arrive", text):
        before = text[:barrier.start()]
        skip = max(before.rfind("continue;"), before.rfind("__global__"))
        if before[skip:].startswith("continue;"):
            assert re.search(r"__sync(warp|threads)\(|bar\.sync", before[skip:]), f"{name}:{before.count(chr(10)) + 1}"
