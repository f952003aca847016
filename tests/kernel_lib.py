"""The kernel library (libpolyb200.so) by itself, for tests of its C entry points: no polygrad
library is needed, so these tests run wherever the kernels are built."""
import ctypes

import numpy as np
import pytest

from polygrad_b200 import ffi

P, I, LL = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
_SIGNATURES = {
    'poly_cuda_init': (I, []),
    'poly_cuda_alloc': (ctypes.c_ulonglong, [ctypes.c_size_t]),
    'poly_cuda_free': (None, [ctypes.c_ulonglong]),
    'poly_cuda_copy_htod': (I, [ctypes.c_ulonglong, P, ctypes.c_size_t]),
    'poly_cuda_copy_dtoh': (I, [P, ctypes.c_ulonglong, ctypes.c_size_t]),
    'poly_b200_set_gemm_policy': (None, [I]),
    'poly_b200_gemm': (I, [LL, LL, LL, P, LL, LL, P, LL, LL, P, LL, P, I, I]),
    'poly_b200_gemm_ex': (I, [LL, LL, LL, P, LL, LL, P, LL, LL, P, LL, P, I, I]),
    'poly_b200_attention': (I, [P, P, P, P, ctypes.c_float, P, I, I, I]),
    'poly_compile_cuda': (P, [ctypes.c_char_p, ctypes.c_char_p]),
    'poly_cuda_program_destroy': (None, [P]),
    'poly_cuda_launch': (I, [P, P, I] + [I] * 6),
    'poly_b200_last_error': (ctypes.c_char_p, []),
}


class Kernels:
    def __init__(self):
        self.c = ctypes.CDLL(ffi.KERNEL_LIB, mode=ctypes.RTLD_LOCAL)
        for name, (restype, args) in _SIGNATURES.items():
            fn = getattr(self.c, name)
            fn.restype, fn.argtypes = restype, args
        assert self.c.poly_cuda_init() == 0, 'no usable B200: ' + self.error()
        self.live = []

    def error(self):
        return self.c.poly_b200_last_error().decode(errors='replace')

    def put(self, a, offset=0):
        """A device copy of `a`, `offset` bytes into its allocation."""
        a = np.ascontiguousarray(a)
        d = self.c.poly_cuda_alloc(a.nbytes + offset)
        assert d
        self.live.append(d)
        assert self.c.poly_cuda_copy_htod(d + offset, a.ctypes.data, a.nbytes) == 0, self.error()
        return d + offset

    def get(self, ptr, shape, dtype=np.float32):
        out = np.empty(shape, dtype)
        assert self.c.poly_cuda_copy_dtoh(out.ctypes.data, ptr, out.nbytes) == 0, self.error()
        return out

    def launch(self, text, name, ptrs):
        prog = self.c.poly_compile_cuda(text.encode(), name.encode())
        assert prog, self.error()
        arr = (ctypes.c_ulonglong * len(ptrs))(*ptrs)
        argv = (P * len(ptrs))(*[ctypes.addressof(arr) + 8 * i for i in range(len(ptrs))])
        rc = self.c.poly_cuda_launch(prog, argv, len(ptrs), 1, 1, 1, 1, 1, 1)
        assert rc == 0, self.error()
        self.c.poly_cuda_program_destroy(prog)

    def release(self):
        for d in self.live:
            self.c.poly_cuda_free(d)
        self.live.clear()


_one = None


@pytest.fixture
def kernels():
    global _one
    if _one is None:
        _one = Kernels()
    yield _one
    _one.c.poly_b200_set_gemm_policy(0)
    _one.release()
