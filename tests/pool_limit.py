"""A cap on the device memory that the library can take, for tests of what it
does when an allocation fails: its buffers come from the device's current
stream-ordered pool, and within ``pool_limit`` that is one of a given size."""

import contextlib
import ctypes


class _Props(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("loc_type", ctypes.c_int),
                ("loc_id", ctypes.c_int), ("win32", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


@contextlib.contextmanager
def pool_limit(nbytes):
    cu = ctypes.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, f"CUDA driver status {rc}"

    pool, default = ctypes.c_void_p(), ctypes.c_void_p()
    props = _Props(alloc_type=1, loc_type=1, loc_id=0, max_size=nbytes)  # pinned, on device 0
    ok(cu.cuDeviceGetMemPool(ctypes.byref(default), 0))
    ok(cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)))
    ok(cu.cuDeviceSetMemPool(0, pool))
    try:
        yield
    finally:
        ok(cu.cuDeviceSetMemPool(0, default))
        cu.cuMemPoolDestroy(pool)
