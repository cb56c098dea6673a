"""lbm_geometry_flags where other CUDA work has left its marks: an unread error of someone else's call, and a device
pool with no room for the call's scratch."""
import ctypes as C

import numpy as np
import pytest

from pv2013_gb300 import cases

pytestmark = pytest.mark.gpu


class PoolProps(C.Structure):
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("location_type", C.c_int), ("location_id", C.c_int),
                ("security", C.c_void_p), ("maxSize", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@pytest.fixture
def cudart(engine):
    return C.CDLL("libcudart.so.13")            # the runtime the library is linked with


def test_flags_with_someone_elses_error_unread(cudart):
    geom = cases.vessel(4001).geometry()
    want = geom.flags()
    assert cudart.cudaSetDevice(4096) != 0       # leaves its error for whoever asks
    got = geom.flags()
    left = cudart.cudaGetLastError()
    assert np.array_equal(got, want) and left != 0     # answered, and the error is still its owner's


def test_flags_without_scratch(cudart):
    rt = cudart
    geom = cases.bifurcation().geometry()
    want = geom.flags()
    old, pool = C.c_void_p(), C.c_void_p()
    assert rt.cudaDeviceGetMemPool(C.byref(old), 0) == 0
    props = PoolProps(allocType=1, location_type=1, location_id=0, maxSize=1 << 20)
    assert rt.cudaMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    assert rt.cudaDeviceSetMemPool(0, pool) == 0
    try:
        held = []                                # all of it, in blocks of the call's size
        for _ in range(8):
            p = C.c_void_p()
            if rt.cudaMallocAsync(C.byref(p), C.c_size_t(32 << 20), None) != 0:
                break
            held.append(p)
        rt.cudaGetLastError()
        full = len(held) < 8
        got = geom.flags() if full else None
        for p in held:
            rt.cudaFreeAsync(p, None)
    finally:
        assert rt.cudaDeviceSetMemPool(0, old) == 0
        rt.cudaDeviceSynchronize()
        rt.cudaMemPoolDestroy(pool)
    if not full:
        pytest.skip("the pool's size limit is not enforced")
    assert np.array_equal(got, want)
