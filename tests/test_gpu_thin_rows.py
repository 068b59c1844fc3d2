"""Byte grids of a few cells a row, on both sides of the sizes where a thread takes
one block instead of a lane a row: every step equals the oracle."""
import numpy as np
import pytest

from gpu_util import describe_diff, stream_ptr, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X", [1, 2, 7, 8, 9])
@pytest.mark.parametrize("YZ", [(240, 241), (301, 330), (5, 40000)], ids=str)
def test_thin_rows_match_oracle(fs3d, orc, cuda, X, YZ):
    Y, Z = YZ
    g = np.random.default_rng(X).choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    d, st = to_device(cuda, g), stream_ptr(cuda)
    for t in range(6):
        fs3d.step_device(d.data_ptr(), X, Y, Z, 21, t, 1, st)
    fs3d.step_device(d.data_ptr(), X, Y, Z, 21, 6, 5, st)
    orc.run(g, 21, 0, 11, nthreads=0)
    got = d.cpu().numpy()
    assert (got == g).all(), describe_diff(got, g, 10)
