"""A batch segment in which one class's kernel records a failure while clusters
step worlds of another: each world of a cluster is written back whole or not at
all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cluster_worlds_are_whole_after_another_class_fails(fs3d, orc):
    n, dims = 1500, [(128 - 3 * (i % 5), 128 - 2 * (i % 4), 128 - 5 * (i % 7)) for i in range(36)]
    seeds = [900 + i for i in range(len(dims))]
    grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, dims)]
    small = fs3d.gen_batch_world(1, 32, 32, 32)
    with fs3d.Batch(4 << 30, steps_per_segment=n) as b:
        ts = b.admit_many(grids, seeds, n)
        t = b.admit(small, 1, n)
        fs3d.inject(fs3d.INJECT_COPY_STALL, 2)  # the small world's copy, 20 ms
        try:
            b.run_segment()
            with pytest.raises(fs3d.Fs3dError) as e:
                b.sync()
            assert e.value.status == fs3d.ERR_TIMEOUT
        finally:
            fs3d.inject(fs3d.INJECT_NONE, 0)
        got = [b.retire(t, g.shape) for t, g in zip(ts, grids)]
        assert (b.retire(t, small.shape) == small).all()
    stepped = 0
    for g, o, s, d in zip(grids, got, seeds, dims):
        if (o == g).all():
            continue
        orc.run(g, s, 0, n, nthreads=0)
        assert (o == g).all(), d
        stepped += 1
    print(f"{stepped} of {len(dims)} worlds stepped")
