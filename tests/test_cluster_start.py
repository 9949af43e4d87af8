"""A CTA's shared memory may be written or read by the other CTAs of its cluster
only once it runs, so every kernel that reaches into another CTA's shared memory
passes a barrier of the cluster first.  Nothing that a kernel computes shows a
missing barrier reliably, so the order is checked in the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc_gb300", "csrc")

# kernel: (file, its barrier of the cluster, its first remote access)
KERNELS = {
    "batched_fp64_kernel": ("batched_kernels.cu", "team_barrier<true>()", "next_team_system("),
    "batched_mixed_kernel": ("batched_kernels.cu", "team_barrier<true>()", "next_team_system("),
    "batch_cluster_fp64_kernel": ("batched_cluster.cu", "cluster_sync()", "system_sum<"),
    "batch_cluster_mixed_kernel": ("batched_cluster.cu", "cluster_sync()", "system_sum<"),
    "cg_cluster_kernel": ("cg_loop.cu", "cluster_sync()", "to_all("),
}


@pytest.mark.parametrize("name", list(KERNELS))
def test_a_cluster_barrier_comes_before_the_first_remote_access(name):
    file, barrier, remote = KERNELS[name]
    with open(os.path.join(CSRC, file)) as f:
        text = f.read()
    start = re.search(r"__global__[^;{]*\b%s\(" % name, text).end()
    body = text[start:text.index("\n}\n", start)]
    assert barrier in body and remote in body
    assert body.index(barrier) < body.index(remote)
