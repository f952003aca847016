"""What a launch that fails on the host leaves behind: one with too many threads, and any without a device."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which('nvcc') or '/usr/local/cuda/bin/nvcc'

ONE_LAUNCH = r'''
#include "pb_gemm.h"
#include <cstdio>
__global__ void nothing(int) {}
int main() {
  const cudaError_t e = pb_launch_chained(nothing, dim3(1), 2048, 0, (cudaStream_t)0, 1, 0);
  printf("%d %d\n", (int)(e == cudaErrorInvalidValue || e == cudaErrorInvalidConfiguration), (int)cudaPeekAtLastError());
}
'''


@pytest.mark.gpu
def test_chained_launch_that_fails_is_reported_once(tmp_path):
    (tmp_path / 'one.cu').write_text(ONE_LAUNCH)
    csrc = os.path.join(ROOT, 'polygrad_b200', 'csrc')
    subprocess.run([NVCC, '-gencode', 'arch=compute_100a,code=sm_100a', '-std=c++17', '-I', os.path.join(csrc, 'kernels'), '-I', os.path.join(csrc, 'runtime'),
                    '-o', 'one', 'one.cu'], cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / 'one')], stdout=subprocess.PIPE, text=True, check=True).stdout
    assert out.split() == ['1', '0']


CALLS = r'''
import sys
import numpy as np
import ctypes
from polygrad_b200 import ffi
c = ctypes.CDLL(ffi.KERNEL_LIB)
LL, P, I = ctypes.c_longlong, ctypes.c_void_p, ctypes.c_int
c.poly_b200_gemm.argtypes = [LL, LL, LL, P, LL, LL, P, LL, LL, P, LL, P, I, I]
c.poly_b200_last_error.restype = ctypes.c_char_p
assert c.poly_cuda_init() == 0
n, k = 1024, int(sys.argv[1])
a, b, o = np.zeros((n, k), np.float32), np.zeros((k, n), np.float32), np.zeros((n, n), np.float32)
print(c.poly_b200_gemm(n, n, k, a.ctypes.data, k, 1, b.ctypes.data, n, 1, o.ctypes.data, n, None, 0, 0), c.poly_b200_last_error().decode())
'''


@pytest.mark.parametrize('k', [512, 1024])
def test_operand_split_that_fails_is_not_taken_for_a_full_pool(k):
    """Either range of the float32 tensor-core route: the call fails with that launch's error and goes no other way."""
    from polygrad_b200 import ffi
    if not os.path.isfile(ffi.KERNEL_LIB):
        pytest.skip('kernel library not built')
    out = subprocess.run([sys.executable, '-c', CALLS, str(k)], cwd=ROOT, env=dict(os.environ, CUDA_VISIBLE_DEVICES='', POLY_B200_DRYRUN='1', PYTHONPATH=ROOT),
                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True, check=True).stdout
    assert out.startswith('-1 gemm: operand split launch: ')
