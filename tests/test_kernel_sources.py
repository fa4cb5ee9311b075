"""Rules of the kernels' sources that no run can show (no GPU)."""

import os
import re
import subprocess

import pytest

from llm_pipeline_b200.ops.build import CSRC, NVCC_FLAGS, find_nvcc


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


def test_the_scans_walk_keeps_its_registers(tmp_path):
    """At every number of state entries and in both types a walk's two sets of registers stay registers (the few bytes that are left are addresses of
    the copying warp)."""
    report = subprocess.run([find_nvcc(), *NVCC_FLAGS, "-I", CSRC, "-Xptxas", "-v", "-c", os.path.join(CSRC, "selective_scan.cu"), "-o", str(tmp_path / "x.o")],
                            capture_output=True, text=True, check=True).stderr
    spilled = dict(re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores", report, re.S))
    walks = {name: int(n) for name, n in spilled.items() if "selective_walk_kernel" in name}
    assert len(walks) == 24 and max(walks.values()) <= 48, walks
