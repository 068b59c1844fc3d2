"""A device that refuses the multi-step launch of a world (its SMs are shared out,
so not all CTAs could be resident): the steps are taken a launch at a time."""
import numpy as np
import pytest

from gpu_util import describe_diff, stream_ptr, to_device

pytestmark = pytest.mark.gpu

DIMS = [(64, 64, 64), (130, 90, 111), (1, 5, 7)]


@pytest.fixture
def refused(fs3d):
    fs3d.inject(fs3d.INJECT_COPY_STALL, 4)
    try:
        yield
    finally:
        fs3d.inject(fs3d.INJECT_NONE, 0)


def level(X, Y, Z):
    return np.random.default_rng(X).choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])


@pytest.mark.parametrize("entry", ["fs3d_run_device", "fs3d_run_device_noalloc"])
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_drop_in_run(fs3d, orc, cuda, refused, entry, dims):
    X, Y, Z = dims
    g, st = level(*dims), stream_ptr(cuda)
    d = to_device(cuda, g)
    assert getattr(fs3d.lib(), entry)(d.data_ptr(), X, Y, Z, 5, 3, 13, st) == 0
    fs3d.run_device_check(st)
    orc.run(g, 5, 3, 13, nthreads=0)
    got = d.cpu().numpy()
    assert (got == g).all(), describe_diff(got, g, 15)


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_world(fs3d, orc, dims):
    g, t = level(*dims), 0
    with fs3d.World(g, 6, 0, fs3d.LAYOUT_PLANES) as w:
        for n, what in ((9, 0), (12, 4), (1, 4), (8, 0)):  # taken, refused, a short call, taken again
            fs3d.inject(fs3d.INJECT_COPY_STALL if what else fs3d.INJECT_NONE, what)
            try:
                w.step(n)
                w.sync()
            finally:
                fs3d.inject(fs3d.INJECT_NONE, 0)
            orc.run(g, 6, t, n, nthreads=0)
            t += n
            assert w.step_counter == t
            assert (w.read() == g).all(), n
