"""A world whose multi-step launch gave up: every later launch, of many steps or
one, steps nothing until the failure is reported, so the state is the one of the
step the world is set back to."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (after 256 or 257 steps the rows' 8-bit change flags read as just changed)
@pytest.mark.parametrize("failed", [16, 256, 257])
@pytest.mark.parametrize("dims", [(64, 64, 64), (130, 120, 111)])
def test_short_calls_after_a_failed_launch_step_nothing(fs3d, orc, dims, failed):
    X, Y, Z = dims
    seed = 47
    g = np.random.default_rng(X).choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    with fs3d.World(g, seed, 0, fs3d.LAYOUT_PLANES) as w:
        w.step(9)
        w.step(1)
        w.sync()
        h10 = w.hash()
        fs3d.inject(fs3d.INJECT_COPY_STALL, 1)
        try:
            w.step(failed)  # its copies never complete
            w.step(1)  # launched after the failure, a launch a step
            w.step(3)
            w.step(5)
            with pytest.raises(fs3d.Fs3dError) as e:
                w.sync()
            assert e.value.status == fs3d.ERR_TIMEOUT
        finally:
            fs3d.inject(fs3d.INJECT_NONE, 0)
        assert w.step_counter == 10
        assert w.hash() == h10
        w.step(1)
        w.step(12)
        w.sync()
        orc.run(g, seed, 0, 23, nthreads=0)
        assert (w.read() == g).all()
