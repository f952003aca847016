"""Contractions through the C entry points with each operand stored either way round, at the edges of
tiles, of 64-row boxes and of k blocks, with row pitches TMA can and cannot address, against float64.

16-bit products are exact and summed in float32: the error of a sum of K terms is below K 2^-24 of the
sum of their magnitudes, for these sizes and random signs far below 1e-5 of the result's rms times ten."""
import numpy as np
import pytest

from conftest import assert_close
from kernel_lib import kernels  # noqa: F401

pytestmark = pytest.mark.gpu


def bf16(x):
    """Rounded to nearest even, as float32."""
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    return ((u + 0x7fff + ((u >> 16) & 1)) & np.uint32(0xffff0000)).view(np.float32)


def bits(x):
    return (np.ascontiguousarray(x, np.float32).view(np.uint32) >> 16).astype(np.uint16)


def stored(x, kfast, pad, rng, conv):
    """The matrix x [rows][k] in memory: k fastest, or rows fastest; `pad` unused elements after each line."""
    m = x if kfast else x.T
    buf = np.full((m.shape[0], m.shape[1] + pad), np.nan, np.float32)
    buf[:, :m.shape[1]] = m
    ld = buf.shape[1]
    return conv(buf), ((ld, 1) if kfast else (1, ld))


SIZES = [(128, 64, 64), (1, 8, 16), (40, 72, 24), (197, 200, 768), (130, 257, 100), (64, 264, 1032), (300, 136, 17)]


@pytest.mark.parametrize('pad', [0, 8, 3])
@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize('m,n,k', SIZES, ids=str)
def test_bf16_operands(kernels, m, n, k, a_kfast, b_kfast, pad):  # noqa: F811
    run_bf16(kernels, m, n, k, a_kfast, b_kfast, pad)


@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (False, False), (False, True)])
def test_bf16_operands_of_cta_pairs(kernels, monkeypatch, a_kfast, b_kfast):  # noqa: F811
    """CTA pairs, forced: by estimated time sizes this small take single CTAs.  A remainder on every axis."""
    monkeypatch.setenv('POLY_B200_TC_CTAS', '2')
    run_bf16(kernels, 2312, 2184, 1048, a_kfast, b_kfast, 0)


def run_bf16(kernels, m, n, k, a_kfast, b_kfast, pad):  # noqa: F811
    rng = np.random.default_rng([m, n, k, pad])
    a, b = bf16(rng.standard_normal((m, k))), bf16(rng.standard_normal((n, k)))
    bias = rng.standard_normal(n).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, a_kfast, pad, rng, bits)
    mb, (b_sn, b_sk) = stored(b, b_kfast, pad, rng, bits)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(ma), a_sm, a_sk, kernels.put(mb), b_sk, b_sn, c, n, kernels.put(bias), 0, 1) == 0, kernels.error()
    want = a.astype(np.float64) @ b.T.astype(np.float64) + bias
    assert_close(kernels.get(c, (m, n)), want, 1e-4, f'bf16 {m} {n} {k}')


F32_SIZES = [(128, 64, 64), (197, 200, 768), (130, 257, 100), (64, 264, 1032), (300, 136, 17), (520, 1030, 333), (2312, 2184, 200)]


@pytest.mark.parametrize('pad', [0, 3])
@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize('m,n,k', F32_SIZES, ids=str)
def test_f32_operands_on_the_tensor_cores(kernels, monkeypatch, m, n, k, a_kfast, b_kfast, pad):  # noqa: F811
    """Every form of the three-product route (single CTAs, pairs, both orders of each operand): float32 accuracy."""
    monkeypatch.setenv('POLY_B200_FP32', 'tcp')
    rng = np.random.default_rng([m, n, k, pad])
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, a_kfast, pad, rng, lambda x: x)
    mb, (b_sn, b_sk) = stored(b, b_kfast, pad, rng, lambda x: x)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(ma), a_sm, a_sk, kernels.put(mb), b_sk, b_sn, c, n, kernels.put(bias), 0, 0) == 0, kernels.error()
    want = a.astype(np.float64) @ b.T.astype(np.float64) + bias
    assert_close(kernels.get(c, (m, n)), want, 1e-5, f'f32 {m} {n} {k}')


def test_f32_infinities_on_the_tensor_cores(kernels, monkeypatch):  # noqa: F811
    """An infinity meets finite values of either sign, zeros (NaN), another infinity, a NaN."""
    monkeypatch.setenv('POLY_B200_FP32', 'tcp')
    m, n, k = 128, 64, 32
    rng = np.random.default_rng(1)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a[3, 5], a[7, 1], a[9, 2], a[11, 30] = np.inf, -np.inf, np.nan, 3.4e38
    b[5, 4], b[5, 6], b[1, 8], b[8, 9] = 0.0, np.inf, -np.inf, -np.inf
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(a), k, 1, kernels.put(b), n, 1, c, n, None, 0, 0) == 0, kernels.error()
    with np.errstate(all='ignore'):
        want = (a[:, :, None].astype(np.float64) * b.astype(np.float64)).sum(1)
    got, rows = kernels.get(c, (m, n)), np.arange(m) != 11         # a product near the largest float32 may round to infinity or not
    assert_close(got[rows], want[rows], 1e-5, 'infinities')


@pytest.mark.parametrize('relu', [0, 1])
@pytest.mark.parametrize('m,n,k', [(160, 257, 64), (31, 1001, 128), (2620, 51237, 16)], ids=str)
def test_rows_of_float32_off_the_16_byte_grid(kernels, m, n, k, relu):  # noqa: F811
    """Whole and ragged groups of 32 rows; the largest result (537 MB) is written with streaming stores."""
    rng = np.random.default_rng([m, n])
    a, b = bf16(rng.standard_normal((m, k))), bf16(rng.standard_normal((n, k)))
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(bits(a)), k, 1, kernels.put(bits(b)), 1, k, c, n, None, relu, 1) == 0, kernels.error()
    got, want = kernels.get(c, (m, n)), a @ b.T
    for r in range(0, m, 500):
        assert_close(got[r:r + 500], np.maximum(want[r:r + 500], 0) if relu else want[r:r + 500], 1e-4, f'{m} {n} {k} from row {r}')


SMALL = [(1, 1, 1), (256, 10, 512), (64, 64, 32), (65, 63, 33), (3, 200, 5000), (100, 1, 77), (1, 100, 64), (256, 512, 784), (500, 900, 100), (640, 420, 288)]


@pytest.mark.parametrize('pad', [0, 4, 3])
@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize('m,n,k', SMALL, ids=str)
def test_small_f32(kernels, m, n, k, a_kfast, b_kfast, pad):  # noqa: F811
    """Tiles of 32 and of 64, one to eight CTAs per tile, slabs of k that are missing, partial or past the end, every operand order and
    alignment; the sums are float32 ones in another order than float64's, far inside 1e-5 at these K."""
    rng = np.random.default_rng([m, n, k, pad])
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, a_kfast, pad, rng, lambda x: x)
    mb, (b_sn, b_sk) = stored(b, b_kfast, pad, rng, lambda x: x)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(ma), a_sm, a_sk, kernels.put(mb), b_sk, b_sn, c, n, kernels.put(bias), 1, 0) == 0, kernels.error()
    want = np.maximum(a.astype(np.float64) @ b.T.astype(np.float64) + bias, 0)
    assert_close(kernels.get(c, (m, n)), want, 1e-5, f'f32 {m} {n} {k}')


@pytest.mark.parametrize('pad', [0, 4, 3])
@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize('m,n,k', SIZES, ids=str)
def test_f32_operands_rounded_to_bf16(kernels, m, n, k, a_kfast, b_kfast, pad):  # noqa: F811
    kernels.c.poly_b200_set_gemm_policy(1)
    rng = np.random.default_rng([m, n, k, pad])
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, a_kfast, pad, rng, lambda x: x)
    mb, (b_sn, b_sk) = stored(b, b_kfast, pad, rng, lambda x: x)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(ma), a_sm, a_sk, kernels.put(mb), b_sk, b_sn, c, n, None, 0, 0) == 0, kernels.error()
    want = bf16(a).astype(np.float64) @ bf16(b).T.astype(np.float64)
    assert_close(kernels.get(c, (m, n)), want, 1e-4, f'policy {m} {n} {k}')


@pytest.mark.parametrize('relu', [0, 1])
@pytest.mark.parametrize('m,n,k,pitch,offset,b_kfast', [(2312, 2185, 72, 2185, 0, True), (129, 18945, 64, 18950, 4, True), (2561, 1799, 1048, 1803, 12, True),
                                                        (2312, 2185, 72, 2185, 0, False), (2620, 51237, 16, 51237, 8, True)], ids=str)
def test_rows_written_line_by_line(kernels, monkeypatch, m, n, k, pitch, offset, b_kfast, relu):  # noqa: F811
    """CTA pairs (forced, with the 74 tiles that this way of writing asks for) whose result rows start anywhere: every offset of
    a row in its 128-byte line, parts of a tile with one column and none, ragged rows; what lies between the rows stays as
    it was.  The largest result (537 MB) is written with streaming stores."""
    monkeypatch.setenv('POLY_B200_TC_CTAS', '2')
    rng = np.random.default_rng([m, n, k])
    a, b = bf16(rng.standard_normal((m, k))), bf16(rng.standard_normal((n, k)))
    mb, (b_sn, b_sk) = stored(b, b_kfast, 0, rng, bits)
    c = kernels.put(np.full((m, pitch), 7, np.float32), offset)
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(bits(a)), k, 1, kernels.put(mb), b_sk, b_sn, c, pitch, None, relu, 1) == 0, kernels.error()
    got = kernels.get(c, (m, pitch))
    assert np.all(got[:, n:] == 7)
    for r in range(0, m, 500):
        want = a[r:r + 500].astype(np.float64) @ b.T.astype(np.float64)
        assert_close(got[r:r + 500, :n], np.maximum(want, 0) if relu else want, 1e-4, f'{m} {n} {k} from row {r}')


@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (False, True)])
@pytest.mark.parametrize('m,n,k', [(1024, 1024, 512), (1023, 1025, 513), (100, 12321, 438), (4096, 4100, 33), (512, 512, 2050)], ids=str)
def test_f32_default_route_around_half_a_giga(kernels, m, n, k, a_kfast, b_kfast):  # noqa: F811
    """2^29 multiply-adds, a little more and a little less, many and few tiles, both routes."""
    rng = np.random.default_rng([m, n, k])
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, a_kfast, 0, rng, lambda x: x)
    mb, (b_sn, b_sk) = stored(b, b_kfast, 0, rng, lambda x: x)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(ma), a_sm, a_sk, kernels.put(mb), b_sk, b_sn, c, n, None, 0, 0) == 0, kernels.error()
    got, want = kernels.get(c, (m, n)), a.astype(np.float64) @ b.T.astype(np.float64)
    assert_close(got, want, 1e-5, f'f32 {m} {n} {k}')
    assert np.sqrt(np.mean((got - want) ** 2)) <= 6e-7 * np.sqrt(np.mean(want ** 2))      # sequential float32 sums: 6e-7 at these K


@pytest.mark.parametrize('first', [0, 1])
@pytest.mark.parametrize('m,n,k', [(128, 2, 64), (2, 128, 64)], ids=str)
def test_policy_switched_on_the_same_operands(kernels, monkeypatch, m, n, k, first):  # noqa: F811
    """One call's operands under either policy in turn, unwritten in between: with two rows stored rows fastest, the kept
    copies for the two policies are equally large."""
    monkeypatch.setenv('POLY_B200_FP32', 'tcp')
    rng = np.random.default_rng([m, n, k])
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    ma, (a_sm, a_sk) = stored(a, m > 2, 0, rng, lambda x: x)
    mb, (b_sn, b_sk) = stored(b, n > 2, 0, rng, lambda x: x)
    d_a, d_b, c = kernels.put(ma), kernels.put(mb), kernels.put(np.zeros((m, n), np.float32))
    exact = [x.astype(np.float64) @ y.T.astype(np.float64) for x, y in ((a, b), (bf16(a), bf16(b)))]
    for policy in (first, 1 - first, first, 1 - first):
        kernels.c.poly_b200_set_gemm_policy(policy)
        assert kernels.c.poly_b200_gemm(m, n, k, d_a, a_sm, a_sk, d_b, b_sk, b_sn, c, n, None, 0, 0) == 0, kernels.error()
        assert_close(kernels.get(c, (m, n)), exact[policy], 1e-5, f'policy {policy}')


@pytest.mark.parametrize('values', ['normal', 'relu', 'positive', 'probabilities'])
@pytest.mark.parametrize('m,n,k', [(4096, 4100, 33), (3000, 2900, 64), (2300, 2300, 112), (2048, 1600, 191), (1700, 1700, 192), (1024, 1024, 768)], ids=str)
def test_f32_default_route_errs_no_more_than_sums_in_k_order(kernels, m, n, k, values):  # noqa: F811
    """Around 2^29 multiply-adds, operands of either and of one sign: on a sample of the result the error is that of one
    rounded multiply-add after the other, or less (the tenth is the sample's own scatter)."""
    rng = np.random.default_rng([m, k])
    a, b = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    if values == 'relu':
        a = np.maximum(a, 0)
    elif values == 'positive':
        a, b = rng.random((m, k)), rng.random((n, k))
    elif values == 'probabilities':
        a = np.exp(2 * a)
        a, b = a / a.sum(1, keepdims=True), rng.random((n, k)) + 0.5
    a, b = a.astype(np.float32), b.astype(np.float32)
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(a), k, 1, kernels.put(b.T), n, 1, c, n, None, 0, 0) == 0, kernels.error()
    rows, cols = rng.permutation(m)[:96], rng.permutation(n)[:96]
    x, y = a[rows].astype(np.float64), b[cols].astype(np.float64)
    acc = np.zeros((96, 96), np.float32)
    for i in range(k):
        acc = (acc + np.outer(x[:, i], y[:, i])).astype(np.float32)
    err = [np.sqrt(np.mean((v - x @ y.T) ** 2)) for v in (kernels.get(c, (m, n))[np.ix_(rows, cols)], acc)]
    assert err[0] <= 1.1 * err[1]


def test_f32_nan_of_any_payload(kernels):  # noqa: F811
    """A NaN that differs from an infinity only in bits that tf32 does not hold stays a NaN (2^29 multiply-adds, default route)."""
    m, n, k = 1024, 1024, 512
    rng = np.random.default_rng(6)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a.view(np.uint32)[3, 5], a.view(np.uint32)[700, 500], b.view(np.uint32)[9, 77] = 0x7f800001, 0xff801fff, 0x7f801000
    c = kernels.put(np.zeros((m, n), np.float32))
    assert kernels.c.poly_b200_gemm(m, n, k, kernels.put(a), k, 1, kernels.put(b), n, 1, c, n, None, 0, 0) == 0, kernels.error()
    want = np.zeros((m, n), bool)
    want[[3, 700], :] = want[:, 77] = True
    assert np.array_equal(np.isnan(kernels.get(c, (m, n))), want)


@pytest.mark.parametrize('arith', ['f32', 'policy', 'bf16'])
@pytest.mark.parametrize('shared_b', [False, True])
@pytest.mark.parametrize('a_kfast,b_kfast', [(True, False), (True, True), (False, False), (False, True)])
def test_batches(kernels, monkeypatch, a_kfast, b_kfast, shared_b, arith):  # noqa: F811
    """Two batch axes, the second operand the same for one of them or not: the parts, copies and views of every batch entry."""
    if arith == 'f32':
        monkeypatch.setenv('POLY_B200_FP32', 'tcp')
    kernels.c.poly_b200_set_gemm_policy(int(arith == 'policy'))
    rng = np.random.default_rng([a_kfast, b_kfast, shared_b])
    h, t, m, n, k = 2, 3, 136, 72, 40
    a, b = rng.standard_normal((t, h, m, k)).astype(np.float32), rng.standard_normal((t, 1 if shared_b else h, n, k)).astype(np.float32)
    if arith != 'f32':
        a, b = bf16(a), bf16(b)
    want = a.astype(np.float64) @ b.astype(np.float64).transpose(0, 1, 3, 2)
    conv = bits if arith == 'bf16' else (lambda x: x)
    ma, mb = (conv(x if kfast else x.transpose(0, 1, 3, 2)) for x, kfast in ((a, a_kfast), (b, b_kfast)))
    a_sm, a_sk = (k, 1) if a_kfast else (1, m)
    b_sn, b_sk = (k, 1) if b_kfast else (1, n)
    b_h, b_t = (0, n * k) if shared_b else (n * k, h * n * k)
    c = kernels.put(np.zeros((t, h, m, n), np.float32))
    kernels.launch(f'//PB200 1\n//kind gemm\n//nparams 3\n//params 0 1 2 -1\n//offsets 0 0 0 0\n//relu 0\n//dtype {"bf16" if arith == "bf16" else "f32"}\n'
                   f'//naxes 5\n//axis0 b {h} {m * n} {m * k} {b_h} 0\n//axis1 b {t} {h * m * n} {h * m * k} {b_t} 0\n//axis2 m {m} {n} {a_sm} 0 0\n'
                   f'//axis3 n {n} 1 0 {b_sn} 0\n//axis4 k {k} 0 {a_sk} {b_sk} 0\n//numel {h * t * m * n}\n', 'batches', [c, kernels.put(ma), kernels.put(mb)])
    assert_close(kernels.get(c, (t, h, m, n)), want, 1e-5 if arith == 'f32' else 1e-4, arith)
