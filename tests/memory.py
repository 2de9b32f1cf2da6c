"""Device memory in the GPU tests: what the stream-ordered pool holds, and a
pool with almost nothing left in it."""
import ctypes
import gc

USED_CURRENT = 7  # cudaMemPoolAttrUsedMemCurrent


class _Location(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int), ("id", ctypes.c_int)]


class _PoolProps(ctypes.Structure):
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location", _Location),
                ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t), ("usage", ctypes.c_ushort),
                ("reserved", ctypes.c_ubyte * 54)]


def _runtime():
    for name in ("libcudart.so.13", "libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            pass
    import pytest
    pytest.skip("no CUDA runtime library to ask about the memory pool")


def pool_used(device=0):
    """Bytes that the device's default pool has handed out."""
    gc.collect()
    rt = _runtime()
    pool, v = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), device) == 0
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaMemPoolGetAttribute(pool, USED_CURRENT, ctypes.byref(v)) == 0
    return v.value


_short_pool = {}


def _pool_of_64mb(rt, device):
    """One for the process: library buffers may outlive the test in it."""
    if device not in _short_pool:
        p = _PoolProps()
        p.alloc_type = 1  # pinned
        p.location = _Location(1, device)
        p.max_size = 64 << 20
        pool, keep = ctypes.c_void_p(), ctypes.c_uint64(1 << 62)  # released bytes stay in the pool
        assert rt.cudaMemPoolCreate(ctypes.byref(pool), ctypes.byref(p)) == 0
        assert rt.cudaMemPoolSetAttribute(pool, 4, ctypes.byref(keep)) == 0
        _short_pool[device] = pool
    return _short_pool[device]


class ShortMemory:
    """While entered, stream-ordered allocations come from a pool of 64 MB of
    which `left` bytes are free; what was allocated before stays valid."""

    def __init__(self, left=1 << 20, device=0):
        self.left, self.device = left, device

    def __enter__(self):
        gc.collect()
        rt = self.rt = _runtime()
        self.fill, self.default = [], ctypes.c_void_p()
        assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(self.default), self.device) == 0
        self.pool = _pool_of_64mb(rt, self.device)
        room = self._take(self.left)
        n = 64 << 20
        while n >= 1 << 12:
            q = self._take(n)
            if q:
                self.fill.append(q)
            else:
                n //= 2
        if room:
            assert rt.cudaFreeAsync(room, None) == 0
        assert rt.cudaDeviceSynchronize() == 0
        assert rt.cudaDeviceSetMemPool(self.device, self.pool) == 0
        return self

    def _take(self, n):
        q = ctypes.c_void_p()
        if self.rt.cudaMallocFromPoolAsync(ctypes.byref(q), ctypes.c_size_t(n), self.pool, None) == 0:
            return q
        self.rt.cudaGetLastError()
        return None

    def __exit__(self, *exc):
        assert self.rt.cudaDeviceSetMemPool(self.device, self.default) == 0
        for q in self.fill:
            assert self.rt.cudaFreeAsync(q, None) == 0
        assert self.rt.cudaDeviceSynchronize() == 0
        return False
