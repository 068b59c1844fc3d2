"""The waits of one world's CTAs for one another.  The first CTA's bulk copy is
made to run into its limit (40 ms with the hook set); its neighbour's wait for
the first edge words runs out before (20 ms), CTAs farther on that have taken
the few steps of a short call wait for the verdict, and all give up together:
the world is as it was.  And several such launches at once, each of one world
of its own."""
import threading

import numpy as np
import pytest

from gpu_util import describe_diff, stream_ptr, to_device

pytestmark = pytest.mark.gpu

DIMS = [(96, 80, 112), (200, 300, 2), (448, 150, 160)]  # narrow slabs along z, along y, wide ones


def level(X, Y, Z, seed):
    r = np.random.default_rng(seed)
    return r.choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("n", [4, 50])
def test_world_is_as_it_was(fs3d, orc, dims, n):
    g = level(*dims, 5)
    with fs3d.World(g, 5, 3, fs3d.LAYOUT_PLANES) as w:
        w.step(6)
        w.sync()
        h = w.hash()
        fs3d.inject(fs3d.INJECT_COPY_STALL, 3)
        try:
            w.step(n)
            w.step(1)
            with pytest.raises(fs3d.Fs3dError) as e:
                w.sync()
            assert e.value.status == fs3d.ERR_TIMEOUT
        finally:
            fs3d.inject(fs3d.INJECT_NONE, 0)
        assert w.step_counter == 9 and w.hash() == h
        w.step(n)
        w.sync()
        orc.run(g, 5, 3, 6 + n, nthreads=0)
        got = w.read()
        assert (got == g).all(), describe_diff(got, g, 8 + n)


@pytest.mark.parametrize("entry", ["fs3d_run_device", "fs3d_run_device_noalloc"])
@pytest.mark.parametrize("n", [4, 50])
def test_drop_in_grid_is_as_it_was(fs3d, orc, cuda, entry, n):
    X, Y, Z = DIMS[0]
    g, st, fn = level(X, Y, Z, 6), stream_ptr(cuda), getattr(fs3d.lib(), entry)
    d = to_device(cuda, g)
    fs3d.inject(fs3d.INJECT_COPY_STALL, 3)
    try:
        assert fn(d.data_ptr(), X, Y, Z, 6, 1, n, st) == 0
        with pytest.raises(fs3d.Fs3dError) as e:
            fs3d.run_device_check(st)
        assert e.value.status == fs3d.ERR_TIMEOUT
    finally:
        fs3d.inject(fs3d.INJECT_NONE, 0)
    assert (d.cpu().numpy() == g).all()
    assert fn(d.data_ptr(), X, Y, Z, 6, 1, n, st) == 0
    fs3d.run_device_check(st)
    orc.run(g, 6, 1, n, nthreads=0)
    assert (d.cpu().numpy() == g).all()


@pytest.mark.parametrize("mode", [1, 3])
def test_cluster_world_is_as_it_was(fs3d, orc, mode):
    dims = [(128, 128, 128), (128, 100, 128)]
    grids = [level(*d, 7) for d in dims]
    with fs3d.Batch(1 << 30, steps_per_segment=30, use_smem=mode) as b:
        ts = b.admit_many(grids, [1, 2], 30)
        fs3d.inject(fs3d.INJECT_COPY_STALL, 3)
        try:
            b.run_segment()
            with pytest.raises(fs3d.Fs3dError) as e:
                b.sync()
            assert e.value.status == fs3d.ERR_TIMEOUT
        finally:
            fs3d.inject(fs3d.INJECT_NONE, 0)
        for t, g in zip(ts, grids):
            assert (b.retire(t, g.shape) == g).all()


@pytest.mark.parametrize("dims,calls", [((40, 41, 42), 30), ((200, 190, 201), 10), ((448, 150, 160), 6)],
                         ids=lambda d: str(d))
def test_several_launches_at_once(fs3d, orc, cuda, dims, calls):
    X, Y, Z = dims
    grids = [level(X, Y, Z, s) for s in range(4)]
    devs, errs = [to_device(cuda, g) for g in grids], []
    cuda.cuda.synchronize()

    def work(i):
        try:
            st = cuda.cuda.Stream()
            w = fs3d.World(grids[i], i) if i == 3 else None  # a world's stream among them
            for c in range(calls):
                if w:
                    w.step(5)
                else:
                    fs3d.run_device(devs[i].data_ptr(), X, Y, Z, i, 5 * c, 5, st.cuda_stream)
            if w:
                w.sync()
                devs[i] = w.read()
                w.close()
            else:
                fs3d.run_device_check(st.cuda_stream)
                devs[i] = devs[i].cpu().numpy()
        except Exception as e:  # noqa: BLE001
            errs.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errs
    for i, g in enumerate(grids):
        orc.run(g, i, 0, 5 * calls, nthreads=0)
        assert (devs[i] == g).all(), i
