"""Grids through a batch and back at every kind of row and address: admitted
from pageable, page-locked and device memory, read back into each of them at
odd addresses whose neighbouring bytes must stay as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(1, 5, 3), (17, 4, 9), (64, 3, 70), (48, 20, 33), (16, 2, 300), (130, 7, 5), (200, 6, 64), (2048, 2, 3), (129, 9, 31)]


def grid(X, Y, Z, seed, statics):
    r = np.random.default_rng(seed)
    v = np.array([0, 1, 2, 3, 4, 250], np.uint8)
    return r.choice(v, (Y, Z, X), p=[0.4, 0.1, 0.25, 0.15, 0.05, 0.05] if statics else [0.5, 0.1, 0.25, 0.15, 0, 0])


@pytest.mark.parametrize("where", ["device", "pinned", "pageable", "mixed"])
@pytest.mark.parametrize("shift", [0, 1, 16])
def test_read_back_into_any_memory(fs3d, orc, cuda, where, shift):
    grids = [grid(*d, seed=i + shift, statics=i % 2 == 0) for i, d in enumerate(DIMS)]
    n = 13
    refs = []
    for i, g in enumerate(grids):
        refs.append(g.copy())
        orc.run(refs[-1], 50 + i, 4, n, nthreads=0)
    offs, at = [], 64
    for g in grids:
        offs.append(at + shift)
        at += (g.size + 15) // 16 * 16 + 32
    fill = np.random.default_rng(9).integers(0, 256, at + 64, dtype=np.uint8)
    dev = cuda.from_numpy(fill).cuda()
    pin = cuda.from_numpy(fill.copy()).pin_memory()
    page = fill.copy()
    base = {"device": dev.data_ptr(), "pinned": pin.data_ptr(), "pageable": page.ctypes.data}
    kinds = [where if where != "mixed" else ("device", "pinned", "pageable")[i % 3] for i in range(len(grids))]
    with fs3d.Batch(1 << 30, steps_per_segment=32) as b:
        t = b.admit_many(grids, [50 + i for i in range(len(grids))], n, start_steps=4)
        b.run_segment()
        b.read_many(t, [base[k] + o for k, o in zip(kinds, offs)])
        again = np.empty(sum(g.size for g in grids), np.uint8)  # back to back, on the host
        ends = np.cumsum([0] + [g.size for g in grids])
        b.retire_many(t, [again.ctypes.data + int(e) for e in ends[:-1]])
    bufs = {"device": dev.cpu().numpy(), "pinned": pin.numpy(), "pageable": page}
    want = {k: fill.copy() for k in bufs}
    for k, o, r in zip(kinds, offs, refs):
        want[k][o:o + r.size] = r.reshape(-1)
    for k in bufs:
        assert (bufs[k] == want[k]).all(), k
    assert (again == np.concatenate([r.reshape(-1) for r in refs])).all()


@pytest.mark.parametrize("shift", [0, 3])
def test_admission_from_device_memory(fs3d, cuda, shift):
    grids = [grid(*d, seed=70 + i, statics=i % 3 == 0) for i, d in enumerate(DIMS)]
    flat = np.concatenate([np.zeros(shift, np.uint8)] + [g.reshape(-1) for g in grids])
    d = cuda.from_numpy(flat).cuda()
    ends = shift + np.cumsum([0] + [g.size for g in grids])
    out = cuda.zeros_like(d)
    with fs3d.Batch(1 << 30) as b:
        t = b.admit_many(grids, [1] * len(grids), 0, ptrs=[d.data_ptr() + int(e) for e in ends[:-1]])
        b.retire_many(t, [out.data_ptr() + int(e) for e in ends[:-1]])
    assert (out.cpu().numpy() == flat).all()


@pytest.mark.parametrize("dims", [(1, 1, 1), (64, 4, 64), (130, 33, 9), (2048, 3, 5)])
def test_world_grids_with_and_without_statics(fs3d, orc, dims):
    """A world's bytes are kept exactly while some cell (here the last one, or
    any) is a static material: written grids alternate, each read back and
    hashed after a step."""
    X, Y, Z = dims
    r = np.random.default_rng(X + Y)
    plain = r.choice(np.array([0, 1, 2, 3], np.uint8), (Y, Z, X))
    last, many = plain.copy(), r.integers(0, 256, (Y, Z, X), dtype=np.uint8)
    last[-1, -1, -1] = 200
    with fs3d.World(plain, 5) as w:
        t = 0
        for g in (plain, last, many, plain, many, last):
            g = g.copy()
            w.write(g)
            assert (w.read() == g).all() and w.hash() == orc.hash(g)
            w.step(1)
            orc.run(g, 5, t, 1, nthreads=1)
            t += 1
            assert (w.read() == g).all() and w.hash() == orc.hash(g)
