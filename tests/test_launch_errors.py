"""What a launch that fails on the host leaves behind."""
import os
import shutil
import subprocess

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
