"""The library in a second context of the same device (an engine that makes its
own): what a context has to be given before a launch (the kernels' shared-memory
limits) is given to each.  Run in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import oracle_lib
import fallingsand3d_gb300 as f

orc = oracle_lib.load()
cu = C.CDLL("libcuda.so.1")
what = sys.argv[2]

def ok(r):
    assert r == 0, "driver call: %d" % r

def grid(X, Y, Z):
    return np.random.default_rng(X).choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])

def drop_in():
    f.World(np.zeros((2, 2, 2), np.uint8), 0).close()  # (makes a context current if none is)
    # 76.8 KB of planes a slab, and a small world
    for X, Y, Z in ((512, 300, 300), (70, 50, 60)):
        g = grid(X, Y, Z)
        for entry in ("fs3d_run_device", "fs3d_run_device_noalloc"):
            d = C.c_uint64()
            ok(cu.cuMemAlloc_v2(C.byref(d), C.c_size_t(g.size)))
            ok(cu.cuMemcpyHtoD_v2(d, C.c_void_p(g.ctypes.data), C.c_size_t(g.size)))
            f.check(getattr(f.lib(), entry)(d.value, X, Y, Z, 5, 2, 6, None))
            f.run_device_check()
            out = np.empty_like(g)
            ok(cu.cuMemcpyDtoH_v2(C.c_void_p(out.ctypes.data), d, C.c_size_t(g.size)))
            ok(cu.cuMemFree_v2(d))
            ref = g.copy()
            orc.run(ref, 5, 2, 6, nthreads=0)
            assert (out == ref).all(), (entry, X, Y, Z)

def world():
    g = grid(300, 200, 260)
    with f.World(g, 3) as w:
        w.step(6)
        w.sync()
        out = w.read()
    orc.run(g, 3, 0, 6, nthreads=0)
    assert (out == g).all()

def batch():
    # one CTA's classes and clusters, young and settled
    dims = [(128, 96, 128), (64, 64, 64), (100, 90, 96), (40, 20, 30)]
    for start in (0, 128):
        grids = [grid(*d) for d in dims]
        for mode in (1, 3):
            with f.Batch(1 << 30, steps_per_segment=20, use_smem=mode) as b:
                ts = b.admit_many(grids, list(range(4)), 20, start_steps=[start] * 4)
                b.run_segment()
                b.sync()
                outs = [b.retire(t, g.shape) for t, g in zip(ts, grids)]
            for i, (g, o) in enumerate(zip(grids, outs)):
                ref = g.copy()
                orc.run(ref, i, start, 20, nthreads=0)
                assert (o == ref).all(), (mode, start, dims[i])

run = {"drop_in": drop_in, "world": world, "batch": batch}[what]
ok(cu.cuInit(0))
dev = C.c_int()
ok(cu.cuDeviceGet(C.byref(dev), 0))
run()  # in the runtime's own context
for _ in range(2):
    ctx = C.c_void_p()
    ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, dev))
    run()
    ok(cu.cuCtxDestroy_v2(ctx))
run()
print("ok")
"""


@pytest.mark.parametrize("what", ["drop_in", "world", "batch"])
def test_second_context(what):
    t = subprocess.run([sys.executable, "-c", CHILD, HERE, what], capture_output=True, text=True, timeout=600,
                       cwd=os.path.dirname(HERE))
    assert t.returncode == 0 and "ok" in t.stdout, (t.stdout + t.stderr)[-3000:]
