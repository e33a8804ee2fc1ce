"""A block of a cluster may touch another block's shared memory only once that
block is known to run, which a cluster barrier shows.  A store that comes
sooner hardly ever fails where it can be watched, so this reads the order of
the barriers and of the remote accesses off the kernels' source."""
from __future__ import annotations

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "nbody-sim_b200", "csrc")
KERNEL = re.compile(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*\)\s*\{")


def cluster_kernels():
    """(file, kernel, body) of every kernel that reaches into its cluster."""
    out = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in KERNEL.finditer(text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            body = text[m.end():end]
            if "map_shared_rank" in body:
                out.append((name, m.group(1), body))
        assert "map_shared_rank" not in text or any(o[0] == name for o in out), name
    return out


def test_the_kernels_are_found():
    assert {k for _, k, _ in cluster_kernels()} >= {"k_sorted_keys", "k_direct"}


@pytest.mark.parametrize("file,kernel,body",
                         [pytest.param(*k, id=k[1]) for k in cluster_kernels()])
def test_barrier_before_the_first_remote_access(file, kernel, body):
    first = body.index("map_shared_rank")
    seen = [m.start() for m in re.finditer(r"\bcl\.(sync|barrier_wait)\(\)", body)]
    assert seen and seen[0] < first, f"{file}: {kernel}"
    # each wait has its arrival before it, and none is left open
    calls = re.findall(r"\bcl\.(sync|barrier_arrive|barrier_wait)\(\)", body)
    open_ = 0
    for c in calls:
        if c == "sync":
            assert open_ == 0
        open_ += {"barrier_arrive": 1, "barrier_wait": -1}.get(c, 0)
        assert open_ in (0, 1)
    assert open_ == 0
