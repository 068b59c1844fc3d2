"""Scratch of a call's own duration: calls on several streams and threads at
once, captured into a graph, and larger than what the pool keeps."""
import threading

import numpy as np
import pytest

from gpu_util import to_device

pytestmark = pytest.mark.gpu


def world(n, seed):
    return np.random.default_rng(seed).choice(np.array([0, 1, 2, 3, 9], np.uint8), (n, n + 1, n + 2), p=[0.5, 0.1, 0.2, 0.15, 0.05])


@pytest.mark.parametrize("n,calls", [(17, 20), (120, 8), (430, 2)])
def test_runs_of_several_threads(fs3d, orc, cuda, n, calls):
    import torch
    grids = [world(n, s) for s in range(4)]
    devs, errs = [to_device(torch, g) for g in grids], []
    torch.cuda.synchronize()

    def work(i):
        try:
            st = torch.cuda.Stream()
            Y, Z, X = grids[i].shape
            for c in range(calls):
                fs3d.run_device(devs[i].data_ptr(), X, Y, Z, i, 3 * c, 3, st.cuda_stream)
                if c % 2:
                    st.synchronize()  # the pool gives back what it does not keep
            st.synchronize()
        except Exception as e:  # noqa: BLE001
            errs.append(e)
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errs
    for i, g in enumerate(grids):
        orc.run(g, i, 0, 3 * calls, nthreads=0)
        assert (devs[i].cpu().numpy() == g).all()


@pytest.mark.parametrize("steps", [2, 12])
def test_captured_run_replays(fs3d, orc, cuda, steps):
    import torch
    g = world(60, 9)
    Y, Z, X = g.shape
    d = to_device(torch, g)
    keep = d.clone()
    fs3d.run_device(d.data_ptr(), X, Y, Z, 4, 0, steps, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fs3d.run_device(d.data_ptr(), X, Y, Z, 4, 0, steps, torch.cuda.current_stream().cuda_stream)
    orc.run(g, 4, 0, steps, nthreads=0)
    for _ in range(3):
        d.copy_(keep)
        graph.replay()
        torch.cuda.synchronize()
        assert (d.cpu().numpy() == g).all()
