"""Launches that may start while their predecessors drain, captured into a graph between work of other kinds:
the replays give what the calls gave."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close
from kernel_lib import kernels  # noqa: F401

pytestmark = pytest.mark.gpu


def declare(c):
    P = ctypes.c_void_p
    c.poly_b200_capture_end.restype, c.poly_b200_capture_end.argtypes = P, [ctypes.c_int]
    c.poly_b200_graph_launch.argtypes = [P, ctypes.c_ulonglong, ctypes.c_ulonglong]
    c.poly_b200_graph_destroy.restype, c.poly_b200_graph_destroy.argtypes = None, [P]
    c.poly_cuda_memset.argtypes = [ctypes.c_ulonglong, ctypes.c_ubyte, ctypes.c_size_t]
    c.poly_b200_trim.restype, c.poly_b200_stream.restype = None, P
    return c


def test_captured_chain(kernels):  # noqa: F811
    c = declare(kernels.c)
    rng = np.random.default_rng(3)
    n = 256
    x = [rng.standard_normal((n, n)).astype(np.float32) / 16 for _ in range(3)]
    a, b, d = (kernels.put(v) for v in x)
    t, u, w = (kernels.put(np.zeros((n, n), np.float32)) for _ in range(3))
    q = kernels.put(rng.standard_normal((1, 128, 2, 64)).astype(np.float32))
    mask, o = kernels.put(np.zeros((128, 128), np.float32)), kernels.put(np.zeros((1, 2, 128, 64), np.float32))

    def chain():
        # every call reads what the one before it wrote
        c.poly_b200_set_gemm_policy(0)
        rc = [c.poly_b200_gemm(n, n, n, a, n, 1, b, n, 1, t, n, None, 0, 0), c.poly_b200_gemm(n, n, n, t, n, 1, d, n, 1, u, n, None, 0, 0)]
        c.poly_b200_set_gemm_policy(1)
        rc.append(c.poly_b200_gemm(n, n, n, u, n, 1, d, n, 1, w, n, None, 0, 0))
        rc.append(c.poly_cuda_memset(t, 1, n * n * 4))
        rc.append(c.poly_b200_gemm(n, n, n, w, 1, n, t, n, 1, u, n, None, 0, 0))
        rc.append(c.poly_b200_attention(q, u, w, mask, 0.125, o, 1, 2, 128))
        assert not any(rc), kernels.error()

    def results():
        return [kernels.get(p, s).copy() for p, s in ((t, (n, n)), (u, (n, n)), (w, (n, n)), (o, (1, 2, 128, 64)))]

    for _ in range(3):
        chain()
    want = results()
    assert c.poly_b200_capture_begin() == 0
    chain()
    graph = c.poly_b200_capture_end(0)
    assert graph, kernels.error()
    for p in (u, w):
        c.poly_cuda_memset(p, 2, n * n * 4)
    for _ in range(3):
        assert c.poly_b200_graph_launch(graph, 0, 0) == 0, kernels.error()
    got = results()
    c.poly_b200_graph_destroy(graph)
    for g, v in zip(got, want):
        assert np.array_equal(g.view(np.uint32), v.view(np.uint32))


@pytest.mark.parametrize('whose', ['library', 'caller'])
def test_float32_contraction_captured_before_any_call(kernels, whose):  # noqa: F811
    """2^29 multiply-adds with nothing in the pool, in a capture of the library's or of a program that captures the
    library's stream itself: it is recorded, and a replay reads the operands as they are then."""
    c = declare(kernels.c)
    rng = np.random.default_rng(4)
    m, n, k = 1024, 1024, 516
    a, b, d = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (k, n)))
    p_a, p_b, p_c = kernels.put(a), kernels.put(b), kernels.put(np.zeros((m, n), np.float32))

    def call():
        return c.poly_b200_gemm(m, n, k, p_a, k, 1, p_b, n, 1, p_c, n, None, 0, 0)

    c.poly_b200_trim()
    if whose == 'library':
        assert c.poly_b200_capture_begin() == 0
        rc = call()
        graph = c.poly_b200_capture_end(0)
        assert rc == 0 and graph, kernels.error()
    else:
        torch = pytest.importorskip('torch')
        graph, status = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(c.poly_b200_stream()), capture_error_mode='thread_local'):
            status.append(call())
        assert status == [0], kernels.error()
    assert c.poly_cuda_copy_htod(p_b, d.ctypes.data, d.nbytes) == 0 and c.poly_b200_synchronize() == 0
    if whose == 'library':
        assert c.poly_b200_graph_launch(graph, 0, 0) == 0, kernels.error()
    else:
        graph.replay()
        torch.cuda.synchronize()
    got = kernels.get(p_c, (m, n))
    if whose == 'library':
        c.poly_b200_graph_destroy(graph)
    assert_close(got, a.astype(np.float64) @ d.astype(np.float64), 1e-5, whose)


@pytest.mark.parametrize('policy,m,n,k', [(1, 136, 64, 64), (0, 1096, 1024, 512), (0, 1096, 1024, 1024)], ids=str)
@pytest.mark.parametrize('discard', [0, 1])
def test_call_after_a_capture_that_never_ran(kernels, policy, m, n, k, discard):  # noqa: F811
    """Operand copies that a capture recorded and nothing replayed are not taken for the operands'."""
    c = declare(kernels.c)
    c.poly_b200_set_gemm_policy(policy)
    m += 64 * discard                         # a program of its own each time
    rng = np.random.default_rng(5)
    # small whole numbers: every route gives the same result
    x = [rng.integers(-4, 5, s).astype(np.float32) for s in ((m, k), (k, n), (m, k), (k, n))]
    p_x, p_c = [kernels.put(v) for v in x], kernels.put(np.zeros((m, n), np.float32))

    def call(i):
        assert c.poly_b200_gemm(m, n, k, p_x[i], k, 1, p_x[i + 1], n, 1, p_c, n, None, 0, 0) == 0, kernels.error()

    call(0)                                   # the program and its memory exist
    assert c.poly_b200_capture_begin() == 0
    call(2)
    graph = c.poly_b200_capture_end(discard)
    assert bool(graph) != bool(discard)
    c.poly_b200_graph_destroy(graph)
    call(2)
    assert np.array_equal(kernels.get(p_c, (m, n)), x[2] @ x[3])
