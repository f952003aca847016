"""The lookup kernel and its gradient's at the sizes where their splitting can go wrong: rows of one
float4, of more than a warp takes at once and of no whole float4; fewer tokens than a warp has lanes, one
more than a chunk holds, every token the same; tables of one row, of less than a block, with a ragged
last block; numberings that are consecutive, distinct, repeated.  Both kernels add in the reference's
order (ascending row, token order, from +0), so numpy's sequential float32 sums are met bit for bit."""
import numpy as np
import pytest

from kernel_lib import kernels  # noqa: F401

pytestmark = pytest.mark.gpu


def numbering(kind, vocab, rng):
    a = np.arange(vocab, dtype=np.float32)
    if kind == 'shifted':
        return a * 3 - 20
    if kind == 'permuted':
        return rng.permutation(vocab).astype(np.float32)
    if kind == 'runs':
        return a // 3
    if kind == 'repeated':
        a[vocab // 2:] = a[:vocab - vocab // 2]
        if vocab > 4:
            a[2] = np.nan
    return a


SIZES = [(1, 4, 1, 1), (5, 7, 1, 3), (64, 64, 2, 33), (65, 96, 1, 4097), (130, 768, 3, 50), (1000, 1604, 1, 17), (257, 1028, 2, 100),
         (40, 128, 1, 9000), (33, 20, 1, 700), (70, 36, 1, 1500), (20000, 12, 1, 300)]


@pytest.mark.parametrize('kind', ['plain', 'shifted', 'permuted', 'repeated', 'runs'])
@pytest.mark.parametrize('vocab,dim,batch,tokens', SIZES, ids=str)
def test_lookup_and_gradient(kernels, vocab, dim, batch, tokens, kind):  # noqa: F811
    rng = np.random.default_rng([vocab, dim, tokens])
    ar = numbering(kind, vocab, rng)
    n = batch * tokens
    ids = ar[rng.integers(0, vocab, n)] if kind != 'permuted' else rng.integers(0, vocab, n).astype(np.float32)
    if n > 2:
        ids[1] = np.nan
        ids[n // 2] = -1e9
    table = rng.standard_normal((vocab, dim)).astype(np.float32)
    table[0, 0] = -0.0
    g = rng.standard_normal((n, dim)).astype(np.float32)
    rows = [np.flatnonzero(ar == x) for x in ids]
    want = np.zeros((n, dim), np.float32)
    want_g = np.zeros((vocab, dim), np.float32)
    for t, match in enumerate(rows):
        for v in match:
            want[t] = want[t] + table[v]
            want_g[v] = want_g[v] + g[t]
    d_ids, d_ar = kernels.put(ids), kernels.put(ar)
    out = kernels.put(np.full((n, dim), 7, np.float32))
    kernels.launch(f'//PB200 1\n//kind gather\n//nparams 4\n//params 0 1 2 3\n//vocab {vocab} {dim}\n//offsets 0 0 0\n'
                   f'//tok {n} {dim} 1\n//feat {dim} 1 1\n', 'lookup', [out, d_ids, d_ar, kernels.put(table)])
    assert np.array_equal(kernels.get(out, (n, dim)).view(np.uint32), want.view(np.uint32))
    out = kernels.put(np.full((vocab, dim), 7, np.float32))
    kernels.launch(f'//PB200 1\n//kind scatter\n//nparams 4\n//params 0 1 2 3\n//vocab {vocab} {dim}\n//offsets 0 0 0\n'
                   f'//tok {tokens} 1 {dim} {batch} {tokens} {tokens * dim}\n//feat {dim} 1 1\n', 'gradient', [out, d_ids, d_ar, kernels.put(g)])
    assert np.array_equal(kernels.get(out, (vocab, dim)).view(np.uint32), want_g.view(np.uint32))


@pytest.mark.parametrize('shift', [0, 1])
def test_axes_that_do_not_merge(kernels, shift):  # noqa: F811
    """Token axes of a transposed id buffer, a feature axis split in two with a gap, rows off the 16-byte grid."""
    rng = np.random.default_rng(shift)
    vocab, b, t, h, e = 70, 3, 41, 2, 8
    ids = rng.integers(0, vocab, (t, b)).astype(np.float32)                 # read as [b][t]
    ar = np.arange(vocab, dtype=np.float32)
    pitch = 2 * (e + 4)
    table = rng.standard_normal((vocab, h, e + 4)).astype(np.float32)
    g = rng.standard_normal((b, t, h, e + 4)).astype(np.float32)
    tok = ids.T.astype(np.int64)
    want = table[tok][..., :e] + np.float32(0)
    want_g = np.zeros((vocab, h, e), np.float32)
    for i in range(b):
        for j in range(t):
            want_g[tok[i, j]] += g[i, j, :, :e]
    d_ids, d_ar = kernels.put(ids), kernels.put(ar)
    out = kernels.put(np.zeros(b * t * h * e, np.float32), 4 * shift)
    kernels.launch(f'//PB200 1\n//kind gather\n//nparams 4\n//params 0 1 2 3\n//vocab {vocab} {pitch}\n//offsets 0 0 0\n'
                   f'//tok {t} {h * e} {b} {b} {t * h * e} 1\n//feat {h} {e} {e + 4} {e} 1 1\n', 'lookup',
                   [out, d_ids, d_ar, kernels.put(table, 4 * shift)])
    assert np.array_equal(kernels.get(out, (b, t, h, e)), want)
    out = kernels.put(np.zeros(vocab * h * e, np.float32), 4 * shift)
    kernels.launch(f'//PB200 1\n//kind scatter\n//nparams 4\n//params 0 1 2 3\n//vocab {vocab} {h * e}\n//offsets 0 0 0\n'
                   f'//tok {t} {b} {pitch} {b} 1 {t * pitch}\n//feat {h} {e} {e + 4} {e} 1 1\n', 'gradient',
                   [out, d_ids, d_ar, kernels.put(g, 4 * shift)])
    assert np.array_equal(kernels.get(out, (vocab, h, e)), want_g)
