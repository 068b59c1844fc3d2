"""A batch's few large young worlds, each stepped by a cluster of CTAs: bit-exact
to the oracle at the sizes where the slabs' cuts change, over several segments
(their last ones past the age where worlds leave the clusters)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one world each: spread over 8 CTAs (or 4, or one, where 8 slabs do not fit)
SIZES = [(128, 128, 128), (96, 97, 131), (128, 512, 16), (2048, 32, 40), (130, 120, 17), (64, 200, 99), (200, 90, 63)]


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("segment,start", [(64, 0), (1, 3), (7, 120)])
def test_spread_world_matches_oracle(fs3d, orc, dims, segment, start):
    X, Y, Z = dims
    seed, n = X + Y + Z + segment, 3 * segment + 1
    r = np.random.default_rng(seed)
    g = r.choice(np.array([0, 1, 2, 3, 9], np.uint8), (Y, Z, X), p=[0.5, 0.04, 0.25, 0.19, 0.02])
    with fs3d.Batch(1 << 30, steps_per_segment=segment) as b:
        t = b.admit(g, seed, n, start_step=start)
        for _ in range(4):
            b.run_segment()
        b.sync()
        c = b.counters()
        assert 0 < c["processed_cell_steps"] <= c["dense_cell_steps"] == n * g.size
        got = b.retire(t, g.shape)
    orc.run(g, seed, start, n, nthreads=0)
    assert (got == g).all()


def test_mixed_young_batch_matches_oracle(fs3d, orc):
    """Large worlds in clusters beside small ones in their own CTAs."""
    dims = [(128, 128, 128), (16, 24, 32), (96, 128, 128), (48, 64, 64), (128, 96, 128), (64, 64, 64), (24, 16, 16)]
    grids = [fs3d.gen_batch_world(7 + i, *d) for i, d in enumerate(dims)]
    with fs3d.Batch(1 << 30) as b:
        t = b.admit_many(grids, [7 + i for i in range(len(dims))], 192)
        for _ in range(3):
            b.run_segment()
        outs = [np.empty_like(g) for g in grids]
        b.retire_many(t, [o.ctypes.data for o in outs])
    for i, (g, o) in enumerate(zip(grids, outs)):
        orc.run(g, 7 + i, 0, 192, nthreads=0)
        assert (o == g).all(), dims[i]


@pytest.mark.parametrize("small,large", [(900, [(130, 128, 131), (128, 128, 128), (257, 64, 100)]), (1500, [(64, 200, 99)])])
def test_few_largest_of_many_young_worlds(fs3d, orc, small, large):
    """More young worlds than are spread by count: only those far above an
    SM's share of a step take clusters, beside many that do not."""
    dims = large + [(16 + 8 * (i % 4), 12 + i % 9, 20 + i % 13) for i in range(small)]
    seeds = [50 + i % 40 for i in range(len(dims))]
    grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, dims)]
    with fs3d.Batch(4 << 30, steps_per_segment=40) as b:
        ts = b.admit_many(grids, seeds, 100)
        for _ in range(3):
            b.run_segment()
        b.sync()
        done, hs = b.poll_many(ts)
    assert done.all()
    for i, (g, s) in enumerate(zip(grids, seeds)):
        if i < len(large) or i % 29 == 0:
            orc.run(g, s, 0, 100, nthreads=0)
            assert int(hs[i]) == orc.hash(g), dims[i]


def test_each_cluster_runs_several_worlds(fs3d, orc):
    """More spread worlds than clusters, of different shapes: a cluster's shared
    memory, its barrier's phase and the edge words pass from world to world."""
    dims = [(128 - 7 * (i % 5), 128 - 9 * (i % 4), 128 - 5 * (i % 7)) for i in range(36)]
    seeds = [300 + i for i in range(len(dims))]
    grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, dims)]
    for mode in (3, 1):  # clusters of 8, and each world's smallest cluster
        with fs3d.Batch(4 << 30, steps_per_segment=37, use_smem=mode) as b:
            ts = b.admit_many(grids, seeds, 74)
            for _ in range(2):
                b.run_segment()
            b.sync()
            done, hs = b.poll_many(ts)
        assert done.all()
        if mode == 3:
            for g, s in zip(grids, seeds):
                orc.run(g, s, 0, 74, nthreads=0)
            want = [orc.hash(g) for g in grids]
            grids = [fs3d.gen_batch_world(s, *d) for s, d in zip(seeds, dims)]
        assert [int(h) for h in hs] == want, mode
