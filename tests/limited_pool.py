"""A device whose memory pool has nothing left, for the calls that then do without scratch (no other memory of the
device is touched)."""
import contextlib
import ctypes as C


class PoolProps(C.Structure):
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("location_type", C.c_int), ("location_id", C.c_int),
                ("security", C.c_void_p), ("maxSize", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


def cudart():
    return C.CDLL("libcudart.so.13")            # the runtime the library is linked with


@contextlib.contextmanager
def empty_pool(smallest):
    """Yields whether allocations of `smallest` bytes now fail (not every driver enforces a pool's size)."""
    rt = cudart()
    old, pool = C.c_void_p(), C.c_void_p()
    assert rt.cudaDeviceGetMemPool(C.byref(old), 0) == 0
    props = PoolProps(allocType=1, location_type=1, location_id=0, maxSize=1 << 20)
    assert rt.cudaMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    assert rt.cudaDeviceSetMemPool(0, pool) == 0
    held = []
    try:
        size = 32 << 20
        while size >= smallest and len(held) < 256:
            p = C.c_void_p()
            if rt.cudaMallocAsync(C.byref(p), C.c_size_t(size), None) == 0:
                held.append(p)
            else:
                rt.cudaGetLastError()
                size //= 2
        yield len(held) < 256
    finally:
        for p in held:
            rt.cudaFreeAsync(p, None)
        rt.cudaDeviceSynchronize()
        assert rt.cudaDeviceSetMemPool(0, old) == 0
        rt.cudaMemPoolDestroy(pool)
