"""The drop-in byte step on rows of every length class and alignment, inside a
larger buffer whose other bytes must stay as they are: bit-exact to the oracle."""
import numpy as np
import pytest

from gpu_util import describe_diff, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X", [1, 2, 3, 15, 16, 17, 48, 63, 64, 65, 112, 127, 129, 2045, 2048])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 16])
def test_rows_of_any_length_and_alignment(fs3d, orc, cuda, X, shift):
    Y, Z, seed, n = 7, 5, 31 * X + shift, 9
    r = np.random.default_rng(seed)
    g = r.choice(np.array([0, 1, 2, 3, 4, 200], np.uint8), (Y, Z, X), p=[0.5, 0.04, 0.24, 0.18, 0.02, 0.02])
    buf = r.integers(0, 256, 64 + g.size + 64, dtype=np.uint8)
    buf[32 + shift:32 + shift + g.size] = g.reshape(-1)
    d = cuda.from_numpy(buf).cuda()
    fs3d.step_device(d.data_ptr() + 32 + shift, X, Y, Z, seed, 2, n, stream_ptr(cuda))
    ref = g.copy()
    orc.run(ref, seed, 2, n, nthreads=0)
    out = d.cpu().numpy()
    got = out[32 + shift:32 + shift + g.size].reshape(g.shape)
    assert (got == ref).all(), describe_diff(got, ref, n + 1)
    assert (out[:32 + shift] == buf[:32 + shift]).all() and (out[32 + shift + g.size:] == buf[32 + shift + g.size:]).all()


@pytest.mark.parametrize("X", [64, 75, 2064])
def test_captured_steps_replay(fs3d, orc, cuda, X):
    """The chained launches of one call in a captured graph, between copies."""
    Y, Z, n = 20, 33, 6
    r = np.random.default_rng(X)
    g = r.choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    keep = cuda.from_numpy(g).cuda()
    d, out = keep.clone(), cuda.empty_like(keep)
    fs3d.step_device(d.data_ptr(), X, Y, Z, 7, 0, n, stream_ptr(cuda))
    cuda.cuda.synchronize()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        d.copy_(keep)
        fs3d.step_device(d.data_ptr(), X, Y, Z, 7, 0, n, stream_ptr(cuda))
        out.copy_(d)
    ref = g.copy()
    orc.run(ref, 7, 0, n, nthreads=0)
    for _ in range(3):
        out.zero_()
        graph.replay()
        cuda.cuda.synchronize()
        assert (out.cpu().numpy() == ref).all()
