"""Many steps of one world in one launch over the whole GPU (a plane world's or
a drop-in run's calls of four steps or more): bit-exact to the oracle at the
sizes where the slabs' cut, their odd ends and the lane groups change."""
import numpy as np
import pytest

from gpu_util import describe_diff, stream_ptr, to_device

pytestmark = pytest.mark.gpu

SIZES = [
    (1, 1, 1), (5, 3, 4), (16, 2, 3),      # one slab, half blocks at every face
    (33, 8, 97), (64, 9, 98), (65, 40, 6),  # cut along z, odd and even ends; along y when z is thin
    (200, 301, 2), (130, 7, 305),           # more layer pairs than SMs
    (448, 150, 160), (512, 300, 64),        # row-pairs in several passes
    (2048, 12, 20), (1990, 21, 9),          # rows of 32 words
]


def level(X, Y, Z, seed):
    r = np.random.default_rng(seed)
    g = r.choice(np.array([0, 1, 2, 3, 7], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    return np.ascontiguousarray(g)


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("t0", [0, 5])
def test_world_calls_match_oracle(fs3d, orc, dims, t0):
    X, Y, Z = dims
    seed = 1000 + X + t0
    g = level(X, Y, Z, seed)
    ref, t = g.copy(), t0
    with fs3d.World(g, seed, t0, fs3d.LAYOUT_PLANES) as w:
        for n in (7, 1, 40, 2, 4):  # one launch, per-step launches, one launch on kept flags ...
            w.step(n)
            w.sync()
            orc.run(ref, seed, t, n, nthreads=0)
            t += n
            got = w.read()
            assert (got == ref).all(), describe_diff(got, ref, t - 1)


@pytest.mark.parametrize("entry", ["fs3d_run_device", "fs3d_run_device_noalloc"])
def test_drop_in_runs_match_oracle(fs3d, orc, cuda, entry):
    st = stream_ptr(cuda)
    for X, Y, Z in SIZES:
        g = level(X, Y, Z, X)
        d = to_device(cuda, g)
        assert getattr(fs3d.lib(), entry)(d.data_ptr(), X, Y, Z, 77, 3, 21, st) == 0
        fs3d.run_device_check(st)
        ref = g.copy()
        orc.run(ref, 77, 3, 21, nthreads=0)
        got = d.cpu().numpy()
        assert (got == ref).all(), ((X, Y, Z), describe_diff(got, ref, 23))
