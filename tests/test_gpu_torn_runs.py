"""Drop-in runs on one stream while a run on another gives up: each grid is left
whole, before or after a run, whenever the failure is recorded."""
import numpy as np
import pytest

from gpu_util import to_device

pytestmark = pytest.mark.gpu


def test_runs_beside_a_failing_run_leave_whole_grids(fs3d, orc, cuda):
    X, Y, Z, n, runs = 512, 60, 200, 3, 200  # (a launch a step: no copy of theirs can stall)
    g = np.random.default_rng(5).choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    small = orc.gen_c1(3)
    a, b = cuda.cuda.Stream(), cuda.cuda.Stream()
    grids, failing = [to_device(cuda, g) for _ in range(3)], to_device(cuda, small)
    warm = to_device(cuda, g)  # (a kernel's first launch may wait for the device)
    for k in (12, 3):
        fs3d.run_device(warm.data_ptr(), X, Y, Z, 3, 0, k, b.cuda_stream)
    cuda.cuda.synchronize()
    fs3d.inject(fs3d.INJECT_COPY_STALL, 1)
    try:
        fs3d.run_device(failing.data_ptr(), 64, 64, 64, 3, 0, 12, a.cuda_stream)  # gives up after 20 ms
        for r in range(runs):
            for d in grids:
                fs3d.run_device(d.data_ptr(), X, Y, Z, 8, n * r, n, b.cuda_stream)
        with pytest.raises(fs3d.Fs3dError) as e:
            b.synchronize()
            fs3d.run_device_check(a.cuda_stream)
        assert e.value.status == fs3d.ERR_TIMEOUT
    finally:
        fs3d.inject(fs3d.INJECT_NONE, 0)
    cuda.cuda.synchronize()
    assert (failing.cpu().numpy() == small).all()
    start = orc.hash(g)
    states = [start] + [int(h) for h in orc.run(g.copy(), 8, 0, n * runs, nthreads=0, hashes=True)][n - 1::n]
    for d in grids:  # a torn grid has none of the states' hashes
        assert orc.hash(d.cpu().numpy()) in states
