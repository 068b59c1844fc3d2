"""Chained kernels (those that begin with chain_wait() and are placed while the
kernel before them still runs) read what that kernel may write with ordinary
loads only: neither they nor the device functions they call use the read-only
path.  Read from the source; no GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fallingsand3d_gb300", "csrc")


def close(text, i, pair):
    """Index just past the bracket that closes the one at i."""
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return i


def functions():
    """name -> [(parameters, body)] of every device function and kernel."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"(?:__device__|__global__)[^;{}=]*?(?:__launch_bounds__\s*\([^{;]*?\)\s*)?\b(\w+)\s*(\()", text):
            end = close(text, m.start(2), "()")
            head = re.match(r"\s*(?:const)?\s*\{", text[end:])
            if head and m.group(1) not in ("__launch_bounds__", "defined"):
                start = end + head.end() - 1
                out.setdefault(m.group(1), []).append((text[m.start(2):end], text[start:close(text, start, "{}")]))
    return out


FUNCTIONS = functions()
CHAINED = sorted(n for n, defs in FUNCTIONS.items() if any("chain_wait();" in b for _, b in defs))


def reached(name):
    seen, todo = set(), [name]
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for _, body in FUNCTIONS[f]:
            todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[\w, ]*>)?\s*\(", body)) if c in FUNCTIONS]
    return seen


def test_the_chained_kernels_are_found():
    assert CHAINED == ["k_occupancy_bytes", "k_occupancy_counts", "k_occupancy_planes", "k_plane_step_skip", "k_render_dda",
                       "k_step_ragged", "k_step_rows"]
    # everything launched that way is one of them, and they wait before all else
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for k in re.findall(r"launch_(?:chained|occupancy|dda)\(\s*&?(k_\w+)", open(path).read()):
            assert k in CHAINED, k
    for k in CHAINED:
        for _, body in FUNCTIONS[k]:
            assert re.match(r"\{\s*chain_wait\(\);", body), k
    assert {"fetch", "filled", "material"} <= reached("k_render_dda")
    assert "rows_changed_recently" in reached("k_plane_step_skip")


@pytest.mark.parametrize("kernel", CHAINED)
def test_no_read_only_loads(kernel):
    for f in sorted(reached(kernel)):
        for params, body in FUNCTIONS[f]:
            assert "__ldg(" not in body and "ld.global.nc" not in body, f
            assert not re.search(r"const\s+\w+\s*\*\s*(?:const\s*)?__restrict__", params), f
