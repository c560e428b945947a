"""Rules of the kernels that no run can show to be kept, checked on their source."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "beamform_project_b200" / "csrc"


def _kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for part in text.split("__global__")[1:]:
            if "map_shared_rank" in part:
                yield pytest.param(part, id=path.stem + ":" + re.search(r"(\w+_kernel)\s*\(", part).group(1))


@pytest.mark.parametrize("kernel", list(_kernels()))
def test_cluster_runs_before_remote_shared_memory(kernel):
    """A CTA's shared memory may be reached from another CTA of its cluster
    only after a cluster barrier: only that says that every CTA has started."""
    before = kernel[:kernel.index("map_shared_rank")]
    assert "cluster.sync()" in before or \
        before.index("cluster.barrier_arrive()") < before.index("cluster.barrier_wait()")


def test_kernels_with_remote_shared_memory_are_found():
    assert len(list(_kernels())) >= 2
