"""Settled worlds of a batch in CTAs wider than their own class (fewer worlds
than fill the GPU): bit-exact to the oracle on each side of every level's line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# worlds of every class by itself (32, 64, 128 and 256 threads), ragged too
DIMS = [(16, 16, 16), (33, 20, 29), (64, 40, 64), (70, 24, 40), (64, 24, 128), (130, 21, 33), (128, 30, 128), (257, 18, 65)]


@pytest.mark.parametrize("copies", [1, 20, 60, 130, 250, 400])
def test_settled_worlds_match_oracle_at_every_level(fs3d, orc, copies):
    """`copies` of every world: together 0.1 to 3 times the threads that run at
    once when all are widest, so each level is taken by some count."""
    n, seeds = 150, [3 + i for i in range(len(DIMS))]
    grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, DIMS)]
    with fs3d.Batch(8 << 30, steps_per_segment=50) as b:
        ts = b.admit_many(grids * copies, seeds * copies, n, start_steps=[128] * (len(DIMS) * copies))
        for _ in range(3):
            b.run_segment()
        b.sync()
        done, hs = b.poll_many(ts)
    assert done.all()
    for g, s in zip(grids, seeds):
        orc.run(g, s, 128, n, nthreads=0)
    assert [int(h) for h in hs] == [orc.hash(g) for g in grids] * copies


def test_tall_settled_worlds_among_many(fs3d, orc):
    """Worlds of more layers than the narrow CTAs hold flags for, among so many
    mixed ones that the others are packed into those."""
    tall = [(16, 1024, 16), (16, 1025, 16), (16, 1500, 16), (20, 2048, 12), (16, 2049, 16), (70, 1100, 24)]
    n, copies, seeds = 70, 250, [3 + i for i in range(len(DIMS) + len(tall))]
    grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, DIMS + tall)]
    m = len(DIMS)
    with fs3d.Batch(8 << 30, steps_per_segment=35) as b:
        ts = b.admit_many(grids[:m] * copies + grids[m:], seeds[:m] * copies + seeds[m:], n,
                          start_steps=[128] * (m * copies + len(tall)))
        for _ in range(2):
            b.run_segment()
        b.sync()
        done, hs = b.poll_many(ts)
    assert done.all()
    for g, s in zip(grids, seeds):
        orc.run(g, s, 128, n, nthreads=0)
    want = [orc.hash(g) for g in grids]
    assert [int(h) for h in hs] == want[:m] * copies + want[m:]
