"""Rules on the order of memory accesses in the device code that no run can show
to be broken: read from the sources.
"""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "compactles.jl_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


def _code(path):
    text = re.sub(r"/\*.*?\*/", " ", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_cluster_barriers_order_memory(path):
    """Blocks of a cluster read one another's shared memory, and a block's shared
    memory ends with the block: the arrival after such reads has to release them and
    the wait before the exit to acquire the others'."""
    code = _code(path)
    assert "barrier.cluster.arrive.relaxed" not in code
    if "ld.shared::cluster" in code:
        assert code.count('"barrier.cluster.arrive.release;"') == 1
        assert code.count('"barrier.cluster.wait.acquire;"') == 1
        body = code[code.index("__global__"):]
        # one pair publishes the end values, a second one keeps them
        assert len(re.findall(r"ln_cluster_arrive\(\);", body)) == 2
        assert len(re.findall(r"ln_cluster_wait\(\);", body)) == 2
