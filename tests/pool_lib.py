"""Device memory taken from the library's allocator: the default pool's high-water mark (cudaMemPoolAttrUsedMemHigh)."""
import ctypes as C

ATTR_USED, ATTR_USED_HIGH = 7, 8


class PoolMark:
    """bytes(): the most the pool held since the mark was made, less what it held then."""

    def __init__(self):
        import torch  # loads the CUDA runtime

        torch.cuda.init()
        self.rt = C.CDLL("libcudart.so.12")
        self.pool = C.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(C.byref(self.pool), torch.cuda.current_device()) == 0
        zero = C.c_uint64(0)
        assert self.rt.cudaMemPoolSetAttribute(self.pool, ATTR_USED_HIGH, C.byref(zero)) == 0
        self.base = self._get(ATTR_USED)

    def _get(self, attr):
        v = C.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def bytes(self):
        return self._get(ATTR_USED_HIGH) - self.base
