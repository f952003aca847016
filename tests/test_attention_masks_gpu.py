"""The attention entry point with every kind of mask tile (one value, a step, values of its own) in every
arrangement a row of tiles can have, operands on and off the 16-byte grid, against float64 on bfloat16-rounded
operands: what is left is the probabilities' rounding to bfloat16 (2^-9), below 5e-3 of the result's rms."""
import numpy as np
import pytest

from kernel_lib import kernels  # noqa: F401
from test_gemm_layouts_gpu import bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scale', [0.125, -0.1])
@pytest.mark.parametrize('mask', ['none', 'causal', 'bias', 'mixed'])
@pytest.mark.parametrize('b,h,t,offset', [(1, 1, 128, 0), (2, 3, 256, 0), (1, 2, 640, 0), (2, 1, 384, 4)], ids=str)
def test_attention(kernels, b, h, t, offset, mask, scale):  # noqa: F811
    rng = np.random.default_rng([b, h, t])
    q, k, v = (rng.standard_normal((b, t, h, 64)).astype(np.float32) for _ in range(3))
    upper = np.triu(np.ones((t, t), bool), 1)
    bias = rng.standard_normal((t, t)).astype(np.float32)
    m = {'none': np.zeros((t, t), np.float32), 'causal': np.where(upper, np.float32(-1e9), np.float32(0)), 'bias': bias,
         'mixed': np.where(upper, np.float32(-1e9), bias)}[mask].astype(np.float32)
    out = kernels.put(np.zeros((b, h, t, 64), np.float32))
    assert kernels.c.poly_b200_attention(kernels.put(q, offset), kernels.put(k, offset), kernels.put(v, offset), kernels.put(m), scale, out, b, h, t) == 0, \
        kernels.error()
    q, k, v = (bf16(x).astype(np.float64).transpose(0, 2, 1, 3) for x in (q, k, v))
    x = q @ k.transpose(0, 1, 3, 2) * scale + m
    p = np.exp(x - x.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True)) @ v
    err, rms = kernels.get(out, (b, h, t, 64)) - want, np.sqrt(np.mean(want ** 2))
    assert np.sqrt(np.mean(err ** 2)) <= 5e-3 * rms
    # one probability's rounding error is at most 2^-9 of it, and the probabilities of a row add up to one
    assert np.abs(err).max() <= 2.0 ** -8 * np.abs(v).max()
