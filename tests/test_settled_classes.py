"""Which class of CTA a settled world of a batch gets: at every level the class
holds the world's layers (its shared memory has room for that many layers'
flags), and a level changes nothing else.  The rule is host arithmetic
(fallingsand3d_gb300/csrc/planes.h), compiled here with g++; no GPU."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fallingsand3d_gb300", "csrc")

HARNESS = r"""
#include "planes.h"
extern "C" int h_levels() { return fs3d::kWidestLevel + 1; }
extern "C" int h_table(int level, int own) { return fs3d::kWidened[level][own]; }
extern "C" int h_class_at(int level, int own, int Y) { return fs3d::gm_class_at(level, own, Y); }
extern "C" int h_holding(int c, int Y) { return fs3d::gm_class_holding(c, Y); }
extern "C" int h_max_layers(int c) { return fs3d::kGmMaxY[c]; }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda_inc, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not found")
    d = tmp_path_factory.mktemp("classes")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-w", "-I", cuda_inc, "-I", CSRC, "-o", str(d / "h.so"),
                    str(d / "h.cpp")], check=True)
    return C.CDLL(str(d / "h.so"))


@pytest.mark.parametrize("Y", [1, 40, 1023, 1024, 1025, 1500, 2047, 2048, 2049, 4095, 4096])
def test_every_level_holds_the_layers(rule, Y):
    for lanes_class in range(4):
        own = rule.h_holding(lanes_class, Y)
        assert rule.h_max_layers(own) >= Y
        if own > 3:
            continue
        for level in range(rule.h_levels()):
            c, table = rule.h_class_at(level, own, Y), rule.h_table(level, own)
            assert rule.h_max_layers(c) >= Y, (level, own, c)
            assert c == table or (c > table and rule.h_max_layers(c - 1) < Y), (level, own, c)
            if Y <= 1024:
                assert c == table


def test_more_layers_than_any_class(rule):
    assert rule.h_holding(0, 4097) == 5
