"""A thread block may touch another one's shared memory only after a cluster
barrier has shown that the other one runs.  In every kernel that maps a peer's
shared memory a barrier's end (a sync, or the wait of a split one) comes first."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "afqmclab_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def kernels(text):
    """The bodies of the __global__ functions, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        i = text.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield text[i:j]


@pytest.mark.parametrize("name", SOURCES)
def test_a_barrier_comes_before_the_first_remote_access(name):
    with open(os.path.join(CSRC, name)) as f:
        bodies = [b for b in kernels(f.read()) if "map_shared_rank" in b]
    for b in bodies:
        barrier = re.search(r"\bcl\.sync\(\)|\bcluster_wait\(\)", b)
        assert barrier and barrier.start() < b.index("map_shared_rank")


def test_the_kernels_that_share_memory_are_found():
    found = []
    for name in SOURCES:
        with open(os.path.join(CSRC, name)) as f:
            found += [name for b in kernels(f.read()) if "map_shared_rank" in b]
    assert {"taylor_f64.cu", "lu_block.cu", "walker_kernels.cu"} <= set(found)
