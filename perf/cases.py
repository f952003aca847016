"""The work whose time matters here: the calls a program makes through the C interface of
include/poly_b200.h, over the sizes, layouts and element types it makes them with.

Three families, each through its public entry points:

* contractions -- poly_b200_gemm and poly_b200_gemm_ex: float32 operands in float32 arithmetic (the
  default), float32 operands under the bfloat16 policy, bfloat16 operands; row-major weights as a
  matmul has them, weights stored by output row as tied embeddings are, the transposed activations
  of a weight gradient; bias, ReLU, GELU; float32 and bfloat16 results;
* attention -- poly_b200_attention with a causal mask and with an additive position bias;
* the embedding lookup and its gradient -- poly_compile_cuda / poly_cuda_launch on the program text
  that poly_render_cuda gives for them.

Sizes come from the benchmark's workloads: the 784-512-10 MLP at batch 256, square matmuls, GPT-2 124M
at 8 x 1024 tokens (width 768, 12 heads, MLP 3072, vocabulary 50257), GPT-2 1.5B's 25 heads.
"""
import ctypes
import math

import torch

from polygrad_b200 import ffi

HEAD = 64           # the attention kernel's head size
GELU, C_BF16 = 2, 1

_c = None


def _lib():
    """The kernel library, with the signatures of the calls made here; initialised on the GPU."""
    global _c
    if _c is None:
        c = ctypes.CDLL(ffi.KERNEL_LIB, mode=ctypes.RTLD_LOCAL)
        p, i, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
        for name, restype, args in [
                ('poly_cuda_init', i, []),
                ('poly_b200_last_error', ctypes.c_char_p, []),
                ('poly_b200_set_gemm_policy', None, [i]),
                ('poly_b200_gemm', i, [ll, ll, ll, p, ll, ll, p, ll, ll, p, ll, p, i, i]),
                ('poly_b200_gemm_ex', i, [ll, ll, ll, p, ll, ll, p, ll, ll, p, ll, p, i, i]),
                ('poly_b200_attention', i, [p, p, p, p, ctypes.c_float, p, i, i, i]),
                ('poly_compile_cuda', p, [ctypes.c_char_p, ctypes.c_char_p]),
                ('poly_cuda_program_destroy', None, [p]),
                ('poly_cuda_launch', i, [p, p, i] + [i] * 6)]:
            fn = getattr(c, name)
            fn.restype, fn.argtypes = restype, args
        if c.poly_cuda_init() != 0:
            raise RuntimeError('no usable B200: ' + c.poly_b200_last_error().decode())
        _c = c
    return _c


def _gemm(name, m, n, k, operands='f32', policy='f32', layout='nn', bias=True, act='none', out='f32'):
    """C[m, n] = A[m, k] B[k, n].  layout: 'nn' both row-major; 'nt' B stored by output column ([n][k]);
    'tn' A stored [k][m].  operands: the element type in memory; policy: the arithmetic of float32 ones."""
    c = dict(kind='gemm', m=m, n=n, k=k, operands=operands, policy=policy, layout=layout, bias=bias, act=act, out=out)
    return dict(c, name=name) if name else c


def _attention(name, batch, heads, tokens, mask):
    c = dict(kind='attention', batch=batch, heads=heads, tokens=tokens, mask=mask)
    return dict(c, name=name) if name else c


def _lookup(name, kind, vocab, dim, batch, tokens, ids):
    c = dict(kind=kind, vocab=vocab, dim=dim, batch=batch, tokens=tokens, ids=ids)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the MLP's output layer: ten columns, the smallest call a model makes
        _gemm('mlp_head_f32', 256, 10, 512),
        # its hidden layer with bias and ReLU: an ordinary small float32 layer
        _gemm('mlp_hidden_f32', 256, 512, 784, act='relu'),
        # GPT-2 124M's fused q/k/v projection in float32, the default arithmetic of large contractions
        _gemm('qkv_f32', 8192, 2304, 768),
        # the weight gradient x^T dy of its MLP over 8 x 512 tokens: training is float32
        _gemm('wgrad_f32', 768, 3072, 4096, layout='tn', bias=False),
        # a square matmul of the bfloat16 sweep, both operands row-major as a matmul gives them
        _gemm('square_bf16', 4096, 4096, 4096, operands='bf16', bias=False),
        # the MLP's first projection as an inference pass runs it: bias, GELU, bfloat16 result
        _gemm('fc_gelu_bf16', 8192, 3072, 768, operands='bf16', act='gelu', out='bf16'),
        # the logits: tied embedding ([vocabulary][width]), rows of 50257 floats; the largest call
        _gemm('logits_bf16', 8192, 50257, 768, operands='bf16', layout='nt', bias=False),
        # one short prompt (197 tokens) through the q/k/v projection under the bfloat16 policy
        _gemm('prompt_policy', 197, 2304, 768, policy='bf16'),
        # GPT-2 124M's attention: 8 sequences, 12 heads, causal
        _attention('attention_causal', 8, 12, 1024, 'causal'),
        # long sequences of a 25-head model with an additive position bias: no tile of the mask is constant
        _attention('attention_bias', 1, 25, 2048, 'bias'),
        # token embedding of a batch, ids as the benchmark draws them
        _lookup('lookup', 'lookup', 50257, 768, 8, 1024, 'uniform'),
        # its gradient for every table row in a training step; ids as frequent as words in text are
        _lookup('lookup_grad', 'lookup_grad', 50257, 768, 8, 1024, 'text'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['gemm'] * 6 + ['attention'] * 2 + ['lookup', 'lookup_grad'])
    if kind == 'gemm':
        arith = rng.choice(['f32', 'f32', 'policy', 'bf16', 'bf16', 'bf16'])
        # multiply-adds a call may take: float32 arithmetic costs more of them than bfloat16 does
        most = {'f32': 1.6e10, 'policy': 6e10, 'bf16': 1.5e11}[arith]
        while True:
            m, n, k = _log(rng, 16, 8192), _log(rng, 10, 16384), _log(rng, 32, 4096)
            if rng.random() < 0.5:         # model widths are round, token counts and vocabularies are not
                n, k = max(16, n // 16 * 16), max(32, k // 16 * 16)
            if 1e6 <= m * n * k <= most:
                break
        act, out = rng.choice(['none', 'none', 'relu']), 'f32'
        if arith == 'bf16' and rng.random() < 0.5:
            out, act, n = 'bf16', rng.choice(['none', 'gelu']), max(8, n // 4 * 4)      # such results need n to be a multiple of 4
        return _gemm(None, m, n, k, operands='bf16' if arith == 'bf16' else 'f32', policy='bf16' if arith == 'policy' else 'f32',
                     layout=rng.choice(['nn', 'nn', 'nt', 'tn']), bias=act != 'none' or rng.random() < 0.5, act=act, out=out)
    if kind == 'attention':
        while True:
            b, h, t = _log(rng, 1, 16), rng.randint(1, 25), 128 * _log(rng, 1, 32)
            if b * h * t * t <= 4e8:
                return _attention(None, b, h, t, rng.choice(['causal', 'causal', 'bias']))
    while True:
        v, d, b, t = _log(rng, 64, 50257), _log(rng, 16, 1600), _log(rng, 1, 16), _log(rng, 16, 1024)
        if v * d <= 50257 * 768 and b * t * d <= 16384 * 1024:
            return _lookup(None, kind, v, d, b, t, rng.choice(['uniform', 'text']))


def _normal(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device='cuda') * std


def _prepare_gemm(c, g):
    m, n, k = c['m'], c['n'], c['k']
    dt = torch.bfloat16 if c['operands'] == 'bf16' else torch.float32
    # activations ~ N(0, 1); weights scaled so that the result is of order one, as initialised layers are;
    # a weight gradient multiplies activations by the small gradients of a mean loss
    a = _normal(g, *((k, m) if c['layout'] == 'tn' else (m, k))).to(dt)
    b = _normal(g, *((n, k) if c['layout'] == 'nt' else (k, n)), std=k ** -0.5).to(dt)
    x = _normal(g, n, std=0.02) if c['bias'] else None
    o = torch.empty(m, n, device='cuda', dtype=torch.bfloat16 if c['out'] == 'bf16' else torch.float32)
    sa = (1, m) if c['layout'] == 'tn' else (k, 1)
    sb = (1, k) if c['layout'] == 'nt' else (n, 1)
    bf16 = int(c['operands'] == 'bf16')
    args = [m, n, k, a.data_ptr(), *sa, b.data_ptr(), *sb, o.data_ptr(), n, x.data_ptr() if c['bias'] else None]
    if c['out'] == 'bf16':
        fn, args = _lib().poly_b200_gemm_ex, args + [bf16, C_BF16 | (GELU if c['act'] == 'gelu' else 0)]
    else:
        fn, args = _lib().poly_b200_gemm, args + [int(c['act'] == 'relu'), bf16]
    # the arguments as the C call takes them, converted once
    args = [t(v) for t, v in zip(fn.argtypes, args)]
    return dict(call=fn, args=args, policy=int(c['policy'] == 'bf16'), out=o, keep=(a, b, x))


def _prepare_attention(c, g):
    b, h, t = c['batch'], c['heads'], c['tokens']
    q, k, v = (_normal(g, b, t, h, HEAD) for _ in range(3))
    pos = torch.arange(t, device='cuda')
    if c['mask'] == 'causal':
        mask = torch.zeros(t, t, device='cuda').masked_fill_(pos[None, :] > pos[:, None], -1e9)
    else:
        mask = _normal(g, 2 * t, std=0.5)[pos[None, :] - pos[:, None] + t].contiguous()      # one value per distance
    o = torch.empty(b, h, t, HEAD, device='cuda')
    fn = _lib().poly_b200_attention
    args = [ty(x) for ty, x in zip(fn.argtypes, [q.data_ptr(), k.data_ptr(), v.data_ptr(), mask.data_ptr(), HEAD ** -0.5, o.data_ptr(), b, h, t])]
    return dict(call=fn, args=args, policy=1, out=o, keep=(q, k, v, mask))


class _Program:
    """A compiled program, destroyed with its last state."""

    def __init__(self, text, name):
        self.h = _lib().poly_compile_cuda(text.encode(), name.encode())
        if not self.h:
            raise RuntimeError(_lib().poly_b200_last_error().decode())

    def __del__(self):
        _lib().poly_cuda_program_destroy(self.h)


def _prepare_lookup(c, g):
    v, d, n = c['vocab'], c['dim'], c['batch'] * c['tokens']
    # ids and the table's numbering are float32 buffers, as the model builder has them
    if c['ids'] == 'uniform':
        ids = torch.randint(0, v, (n,), generator=g, device='cuda')
    else:
        # the r-th most frequent word has frequency ~ 1 / (r + 2.7)
        u = torch.rand(n, generator=g, device='cuda', dtype=torch.float64)
        rank = (2.7 * ((v + 2.7) / 2.7) ** u - 2.7).long().clamp_(0, v - 1)
        ids = torch.randperm(v, generator=g, device='cuda')[rank]
    ids, arange = ids.float(), torch.arange(v, device='cuda').float()
    grad = c['kind'] == 'lookup_grad'
    src = _normal(g, n if grad else v, d, std=0.02)
    o = torch.empty(v if grad else n, d, device='cuda')
    # parameters: result, ids, numbering, source; axes of the tokens (extent, strides) and of the features
    head = f'//PB200 1\n//kind {"scatter" if grad else "gather"}\n//nparams 4\n//params 0 1 2 3\n//vocab {v} {d}\n//offsets 0 0 0\n'
    if grad:
        tok = f' {c["tokens"]} 1 {d} {c["batch"]} {c["tokens"]} {c["tokens"] * d}'
    else:
        tok = f' {n} {d} 1'
    prog = _Program(head + f'//tok{tok}\n//feat {d} 1 1\n', c['kind'])
    ptrs = (ctypes.c_ulonglong * 4)(o.data_ptr(), ids.data_ptr(), arange.data_ptr(), src.data_ptr())
    argv = (ctypes.c_void_p * 4)(*[ctypes.addressof(ptrs) + 8 * j for j in range(4)])
    fn = _lib().poly_cuda_launch
    args = [ctypes.c_void_p(prog.h), ctypes.cast(argv, ctypes.c_void_p), 4] + [1] * 6
    return dict(call=fn, args=args, policy=0, out=o, keep=(ids, arange, src, prog, ptrs, argv))


def prepare(case, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed))
    _lib()
    s = {'gemm': _prepare_gemm, 'attention': _prepare_attention}.get(case['kind'], _prepare_lookup)(case, g)
    torch.cuda.synchronize()        # the library works on a stream of its own
    return s


def run(state):
    lib = _lib()
    lib.poly_b200_set_gemm_policy(state['policy'])
    if state['call'](*state['args']) != 0:
        raise RuntimeError(lib.poly_b200_last_error().decode())
    return state['out']


def work(case):
    c = case
    if c['kind'] == 'gemm':
        m, n, k = c['m'], c['n'], c['k']
        e = 2 if c['operands'] == 'bf16' else 4
        return dict(bytes=e * (m * k + k * n) + (2 if c['out'] == 'bf16' else 4) * m * n + (4 * n if c['bias'] else 0), flops=2 * m * n * k)
    if c['kind'] == 'attention':
        bh, t = c['batch'] * c['heads'], c['tokens']
        pairs = t * (t + 1) // 2 if c['mask'] == 'causal' else t * t
        return dict(bytes=4 * (4 * bh * t * HEAD + t * t), flops=4 * bh * pairs * HEAD)
    v, d, n = c['vocab'], c['dim'], c['batch'] * c['tokens']
    if c['kind'] == 'lookup':
        return dict(bytes=4 * (n + v + min(n, v) * d + n * d), flops=0)
    return dict(bytes=4 * (n + v + n * d + v * d), flops=n * d)


def tolerance(case):
    if case['kind'] == 'lookup':
        return 'exact'
    if case['kind'] == 'lookup_grad':
        return {'rel': 1e-5}                # float32 sums
    if case['kind'] == 'attention' or case.get('out') == 'bf16':
        return {'rel': 1e-2}                # probabilities, or the result, rounded to bfloat16
    if case['operands'] == 'bf16' or case['policy'] == 'bf16':
        return {'rel': 1e-4}                # exact products of bfloat16 values, summed in float32 by the tensor cores
    return {'rel': 1e-5}                    # float32
