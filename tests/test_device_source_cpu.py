"""Rules on memory order and shared launch state that a run shows to be broken only
by chance: read from the sources.
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


def _kernels(code):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__", code):
        i = code.index("(", m.end())
        while True:   # attributes with arguments come before the name
            depth, j = 0, i
            while True:
                depth += {"(": 1, ")": -1}.get(code[j], 0)
                j += 1
                if depth == 0:
                    break
            rest = code[j:].lstrip()
            if rest.startswith("{"):
                break
            i = code.index("(", j)
        b = code.index("{", j)
        depth, e = 0, b
        while True:
            depth += {"{": 1, "}": -1}.get(code[e], 0)
            e += 1
            if depth == 0:
                break
        yield re.search(r"(\w+)\s*$", code[:i]).group(1), code[i + 1:j - 1], code[b:e]


# tables of a plan: written before the plan's first launch and never again
CONSTANT_TABLES = {"Gw", "Gg", "tab"}


def test_dependent_kernels_promise_nothing_before_their_wait():
    """A kernel that starts with grid_dependency_wait is alive while its predecessor
    still writes.  `__restrict__` on its parameters would promise that nobody else
    writes the memory while it lives, and let reads move above the wait."""
    seen = 0
    for path in SOURCES:
        for name, params, body in _kernels(_code(path)):
            if "grid_dependency_wait()" not in body:
                continue
            seen += 1
            bad = [n for n in re.findall(r"__restrict__\s+(\w+)", params) if n not in CONSTANT_TABLES]
            assert not bad, (path.name, name, bad)
    assert seen >= 16


def test_shared_memory_limits_are_only_raised_to_the_maximum():
    """A kernel's dynamic shared memory limit is shared by every plan and host thread of
    a device: set to one launch's size, it may undercut a larger launch that another
    thread is about to make.  It is set in one place, to the device's maximum."""
    calls = []
    for path in sorted(CSRC.iterdir()):
        if path.suffix in (".cu", ".cuh", ".cpp", ".h"):
            calls += [(path.name, m.group(1)) for m in
                      re.finditer(r"cudaFuncSetAttribute\(([^;]*)\);", _code(path))]
    assert [c[0] for c in calls] == ["cles_internal.h"], calls
    assert calls[0][1].rstrip(")").endswith("(int)kMaxDynamicSmem"), calls
    assert "kMaxDynamicSmem = 227 * 1024;" in _code(CSRC / "cles_internal.h")
