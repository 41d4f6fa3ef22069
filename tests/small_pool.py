"""Device allocations of the block's calls come from a pool of at most `limit` bytes: running out
of scratch without filling the GPU.  Handles made in the block are freed in it.  The pool itself stays: a destroyed one
took the process down at a later allocation."""
import contextlib
import ctypes as C


class _Props(C.Structure):  # CUmemPoolProps
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("locationType", C.c_int), ("locationId", C.c_int),
                ("security", C.c_void_p), ("maxSize", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@contextlib.contextmanager
def small_pool(limit: int):
    cu = C.CDLL("libcuda.so.1")
    pool, default = C.c_void_p(), C.c_void_p()
    props = _Props(allocType=1, locationType=1, maxSize=limit)  # pinned, on device 0
    assert cu.cuMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(default), 0) == 0
    assert cu.cuDeviceSetMemPool(0, pool) == 0
    try:
        yield
    finally:
        assert cu.cuDeviceSetMemPool(0, default) == 0
