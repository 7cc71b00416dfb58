"""bench.py's DRAM traffic comes from a capture of the kernel that the workload runs
on, or there is none."""
import re

import bench
from helpers import ROOT


def test_traffic_is_of_the_kernel_that_runs():
    tps, src = bench.traffic_per_source("batched", "rmat20")
    text = (ROOT / src).read_text()
    assert src == "profiles/batched_kernel_rmat20.md"
    assert tps == float(re.search(r"traffic_bytes_per_source: (\S+)", text).group(1))
    # the capture names the launch shape that the kernel is compiled for
    source = (ROOT / "centrality-gpu_b200" / "csrc" / "kernels_batched.cu").read_text()
    ctas = int(re.search(r"define BCGPU_BATCHED_MIN_CTAS (\d+)", source).group(1))
    assert f"| grid x block | {148 * ctas} x 256" in text
    # the per-source kernel of the R-MAT and grid workloads has no such capture
    assert bench.traffic_per_source("plain", "rmat20") == (None, None)
