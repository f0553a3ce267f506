"""A small pool for the library's stream-ordered device allocations: inside
limited_pool(bytes) every allocation that would pass the limit fails with
cudaErrorMemoryAllocation, as on a full device, with plenty of memory left."""
import contextlib
import ctypes


class Location(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int), ("id", ctypes.c_int)]


class PoolProps(ctypes.Structure):  # cudaMemPoolProps
    _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("location", Location),
                ("win32SecurityAttributes", ctypes.c_void_p), ("maxSize", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def _ok(status):
    assert status == 0, "CUDA status %d" % status


@contextlib.contextmanager
def limited_pool(limit, device=0):
    rt = ctypes.CDLL("libcudart.so.13")
    rt.cudaMemPoolCreate.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(PoolProps)]
    rt.cudaDeviceSetMemPool.argtypes = [ctypes.c_int, ctypes.c_void_p]
    rt.cudaDeviceGetMemPool.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_int]
    before, pool = ctypes.c_void_p(), ctypes.c_void_p()
    _ok(rt.cudaDeviceGetMemPool(ctypes.byref(before), device))
    props = PoolProps(1, 0, Location(1, device), None, limit)  # pinned to the device, no export handles
    _ok(rt.cudaMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)))
    _ok(rt.cudaDeviceSetMemPool(device, pool))
    try:
        yield
    finally:
        # (The pool itself stays: buffers from it are freed after this.)
        _ok(rt.cudaDeviceSetMemPool(device, before))
