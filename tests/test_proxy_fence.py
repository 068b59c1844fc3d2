"""A kernel that holds one world after another in shared memory and fills it with
bulk copies has, in its loop over worlds, a fence between the ordinary accesses
to one world and the copies of the next (they go through different proxies, and
no barrier orders the two).  Read from the source; no GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fallingsand3d_gb300", "csrc")


def body_at(text, start):
    """The braces' content from the first { after start on."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def world_loops():
    """(kernel, its loop over worlds) of the kernels that load worlds by bulk copies."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            body = body_at(text, m.end())
            loop = re.search(r"for \(;;\)", body)
            if loop and "mbar_wait(" in body:
                out.append((m.group(1), body_at(body, loop.start())))
    return out


def test_every_such_kernel_is_found():
    assert {k for k, _ in world_loops()} == {"k_plane_segment_resident", "k_batch_slabs"}


@pytest.mark.parametrize("kernel", ["k_plane_segment_resident", "k_batch_slabs"])
def test_fence_between_worlds(kernel):
    loop = dict(world_loops())[kernel]
    assert "fence.proxy.async.shared::cta" in loop
    # followed, before the loop comes round to the next world's copies, by a barrier of all threads
    after = loop[loop.index("fence.proxy.async"):] + loop
    assert re.search(r"(__syncthreads|cluster\.sync)\(", after).start() < re.search(r"(bulk_load|\.load)\(", after).start()
