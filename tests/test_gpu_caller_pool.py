"""Scratch of a call comes from the memory pool that the caller made the
device's current one, when it is not the device's default."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import stream_ptr, to_device

pytestmark = pytest.mark.gpu

_RELEASE_THRESHOLD, _USED_MEM_HIGH = 0x4, 0x8  # cudaMemPoolAttr (driver_types.h)


class _Location(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]


class _PoolProps(C.Structure):
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("location", _Location), ("security", C.c_void_p),
                ("maxSize", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


def _cudart():
    for name in ("/usr/local/cuda/lib64/libcudart.so.13", "libcudart.so.13", "libcudart.so"):
        try:
            return C.CDLL(name)
        except OSError:
            continue
    pytest.skip("the CUDA runtime library is not loadable here")


def test_scratch_follows_the_current_pool(fs3d, orc, cuda):
    rt = _cudart()
    dev = cuda.cuda.current_device()
    g = np.random.default_rng(3).choice(np.array([0, 1, 2, 3, 9], np.uint8), (60, 70, 80), p=[0.5, 0.05, 0.25, 0.18, 0.02])
    d = to_device(cuda, g)
    st = stream_ptr(cuda)
    fs3d.run_device(d.data_ptr(), 80, 60, 70, 7, 0, 5, st)  # the library's own pool exists by now
    cuda.cuda.synchronize()
    before, pool = C.c_void_p(), C.c_void_p()
    assert rt.cudaDeviceGetMemPool(C.byref(before), dev) == 0
    props = _PoolProps(allocType=1, location=_Location(1, dev))  # pinned, on this device
    assert rt.cudaMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    try:
        assert rt.cudaDeviceSetMemPool(dev, pool) == 0
        high = C.c_uint64()
        fs3d.run_device(d.data_ptr(), 80, 60, 70, 7, 5, 5, st)
        fs3d.run_device_check(st)
        assert rt.cudaMemPoolGetAttribute(pool, _USED_MEM_HIGH, C.byref(high)) == 0
        assert high.value >= g.size // 4
    finally:
        assert rt.cudaDeviceSetMemPool(dev, before) == 0
        cuda.cuda.synchronize()
        rt.cudaMemPoolDestroy(pool)
    fs3d.run_device(d.data_ptr(), 80, 60, 70, 7, 10, 5, st)
    fs3d.run_device_check(st)
    orc.run(g, 7, 0, 15, nthreads=0)
    assert (d.cpu().numpy() == g).all()
