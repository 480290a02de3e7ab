"""A shortage of device memory made on the host: inside the context the
process's stream-ordered allocations come from a pool of a bounded size that
is already used up, so each is refused with an out-of-memory error.  The
device's own memory is not touched, and the former pool is put back."""
import contextlib
import ctypes as C


class _Props(C.Structure):              # CUmemPoolProps
    _fields_ = [('allocType', C.c_int), ('handleTypes', C.c_int), ('locType', C.c_int), ('locId', C.c_int),
                ('security', C.c_void_p), ('maxSize', C.c_size_t), ('usage', C.c_ushort), ('reserved', C.c_ubyte * 54)]


def _cu(name, *args):
    return getattr(C.CDLL('libcuda.so.1'), name)(*args)


@contextlib.contextmanager
def no_device_memory(device=0, room=0):
    """`room`: bytes left in the pool"""
    props = _Props(allocType=1, locType=1, locId=device, maxSize=32 << 20)    # pinned memory of the device
    pool, old, held, spare = C.c_void_p(), C.c_void_p(), [], C.c_uint64()
    assert _cu('cuDeviceGetMemPool', C.byref(old), device) == 0
    assert _cu('cuMemPoolCreate', C.byref(pool), C.byref(props)) == 0

    def take(n):
        p = C.c_uint64()
        ok = _cu('cuMemAllocFromPoolAsync', C.byref(p), C.c_size_t(n), pool, None) == 0
        return p if ok else None

    try:
        if room:
            spare = take(room)
            assert spare is not None
        n = 64 << 20
        while n >= 256:
            p = take(n)
            if p is None:
                n //= 2
            else:
                held.append(p)
                assert len(held) < 4096
        if room:
            _cu('cuMemFreeAsync', spare, None)
        _cu('cuCtxSynchronize')
        assert _cu('cuDeviceSetMemPool', device, pool) == 0
        yield
    finally:
        _cu('cuDeviceSetMemPool', device, old)
        for p in held:
            _cu('cuMemFreeAsync', p, None)
        _cu('cuCtxSynchronize')
        _cu('cuMemPoolDestroy', pool)
