"""A value kept per device and context (fallingsand3d_gb300/csrc/per_context.h):
made once for each, again for another context of a device, never taken from one
device for another.  Compiled here with g++ and asked with made-up contexts; no
GPU.  The kernels' shared-memory limits are kept this way, not once per process."""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fallingsand3d_gb300", "csrc")

HARNESS = r"""
#include "per_context.h"
static fs3d::PerContext<int> kept;
static unsigned long long ctx_now;
static int made;
extern "C" int h_made() { return made; }
// device dev, context ctx current (become: the context that making it brings about)
extern "C" int h_get(int dev, unsigned long long ctx, unsigned long long become, int value) {
    ctx_now = ctx;
    return kept.get(dev, [] { return ctx_now; }, [&] { ctx_now = become; ++made; return value; });
}
"""


@pytest.fixture()
def kept(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-o", str(tmp_path / "h.so"),
                    str(tmp_path / "h.cpp"), "-lpthread"], check=True)
    L = C.CDLL(str(tmp_path / "h.so"))
    L.h_get.argtypes = [C.c_int, C.c_ulonglong, C.c_ulonglong, C.c_int]
    return L


def test_made_once_per_device_and_context(kept):
    assert kept.h_get(0, 7, 7, 10) == 10 and kept.h_get(0, 7, 7, 11) == 10 and kept.h_made() == 1
    assert kept.h_get(1, 9, 9, 20) == 20 and kept.h_made() == 2  # another device
    assert kept.h_get(0, 7, 7, 12) == 10 and kept.h_get(1, 9, 9, 21) == 20 and kept.h_made() == 2
    assert kept.h_get(0, 8, 8, 30) == 30 and kept.h_made() == 3  # another context of the first
    assert kept.h_get(0, 7, 7, 40) == 40 and kept.h_made() == 4
    assert kept.h_get(2, 0, 5, 50) == 50 and kept.h_get(2, 5, 5, 51) == 50 and kept.h_made() == 5  # none current before
    assert kept.h_get(64, 1, 1, 60) == 60 and kept.h_get(64, 1, 1, 61) == 61  # more devices than are kept


def test_function_attributes_are_set_per_context():
    """No kernel attribute is set under a once-per-process guard."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".cpp")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        if "cudaFuncSetAttribute" in text:
            assert "of_current_context" in text and "call_once" not in text, name
            assert not re.search(r"static const \w+ \w+ = \[\][^;]*?(?:\{[^}]*;)*[^}]*cudaFuncSetAttribute", text), name
