"""The device's stream-ordered memory pool, through the driver API: what is in
use, and a pool of limited size in its place, so that an allocation can fail
without the device being full."""
import contextlib
import ctypes

USED_MEM_CURRENT = 7  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT


class _Location(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int), ("id", ctypes.c_int)]


class _PoolProps(ctypes.Structure):
    _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("location", _Location),
                ("win32SecurityAttributes", ctypes.c_void_p), ("maxSize", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def _cu():
    return ctypes.CDLL("libcuda.so.1")


def _current(device=0):
    pool = ctypes.c_void_p()
    assert _cu().cuDeviceGetMemPool(ctypes.byref(pool), device) == 0
    return pool


def used_bytes(ctx):
    """Bytes in use in the device's current pool, after the context's stream."""
    ctx.synchronize()
    v = ctypes.c_uint64()
    assert _cu().cuMemPoolGetAttribute(_current(), USED_MEM_CURRENT, ctypes.byref(v)) == 0
    return v.value


@contextlib.contextmanager
def limited(max_bytes, device=0):
    """The device allocates from a pool of at most max_bytes inside the block."""
    cu, old, pool = _cu(), _current(device), ctypes.c_void_p()
    props = _PoolProps(allocType=1, handleTypes=0, location=_Location(1, device), maxSize=max_bytes)  # pinned, device
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    try:
        assert cu.cuDeviceSetMemPool(device, pool) == 0
        yield
    finally:
        assert cu.cuDeviceSetMemPool(device, old) == 0
        cu.cuMemPoolDestroy(pool)
