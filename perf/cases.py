"""Measured workloads of the framework: what its users have it do, through its public entry points.

Two jobs make up nearly all the GPU time of a program that uses this library.  Quantizing a model: calibration
activations and weights go in, packed int4 matrices come out (`accumulate_H`, `gptq`, `pack_matrix`, `gptq_many`).
Running the quantized model: `quantized_matmul` at the token counts of decoding, of batched decoding, of a prompt
and of a fine-tuning step, where the gradient of the activations needs the transposed product as well.

`listed()` holds the fixed cases, `draw(rng)` more of the same ranges; `prepare` makes what a program has in hand
before the call, `run` is one pass, `exact` the same outputs from plain torch in 64 bits.
"""
from __future__ import annotations

import importlib
import math

import torch

_gptq = importlib.import_module('jax_gptq_b200.gptq')
_op = importlib.import_module('jax_gptq_b200.op')

_DTYPES = {'f32': torch.float32, 'f16': torch.float16, 'bf16': torch.bfloat16}
_BYTES = {'f32': 4, 'f16': 2, 'bf16': 2}

# the four linears of a GPT-2-small block (K, N), in execution order
_BLOCK = ((768, 2304), (768, 768), (768, 3072), (3072, 768))
_BLOCK_SIZE, _DAMPING = 128, 0.01


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # One token through one linear of a 7B-sized model: the smallest call there is, launches and latency count.
        dict(name='decode_m1_4096x4096_f16', kind='matmul', M=1, K=4096, N=4096, x='f16', zs='f16'),
        # One token through the widest linear of a 70B-sized block: the packed weights stream once from HBM.
        dict(name='decode_m1_8192x28672_f16', kind='matmul', M=1, K=8192, N=28672, x='f16', zs='f16'),
        # Eight concurrent sequences with bf16 activations and the fp32 scales that pack_matrix returns.
        dict(name='decode_m8_4096x11008_bf16', kind='matmul', M=8, K=4096, N=11008, x='bf16', zs='f32'),
        # A decode step of a GPT-2-small-shaped model, batch 32: 48 small products one after another.
        dict(name='decode_step_gpt2_m32_f16', kind='step', M=32, layers=12, x='f16', zs='f32'),
        # A short prompt, or one chunk of a long one.
        dict(name='chunk_m128_8192x28672_f16', kind='matmul', M=128, K=8192, N=28672, x='f16', zs='f16'),
        # A prompt of 2048 tokens.
        dict(name='prefill_m2048_4096x11008_bf16', kind='matmul', M=2048, K=4096, N=11008, x='bf16', zs='f32'),
        # Fine-tuning around a frozen quantized linear: the product and the gradient of its input.
        dict(name='tune_m2048_11008x4096_bf16', kind='grad', M=2048, K=11008, N=4096, x='bf16', zs='f32'),
        # Odd channel count, ragged token count, fp32 activations, with the gradient: a small adapter layer.
        dict(name='ragged_m137_256x909_f32', kind='grad', M=137, K=256, N=909, x='f32', zs='f32'),
        # The Hessian alone, sixteen calibration batches that the program captured one by one.
        dict(name='hessian_3072_n65536_f32', kind='hessian', K=3072, n=65536, batches=16, x='f32'),
        # One dense layer from calibration data to packed weights.
        dict(name='layer_768x3072_n4096_f32', kind='layer', K=768, N=3072, n=4096, batches=4, x='f32', bits=4,
             actorder=False),
        # A linear of a 7B-sized model, bf16 weights and activations, in activation order.
        dict(name='layer_4096x4096_n16384_bf16', kind='layer', K=4096, N=4096, n=16384, batches=8, x='bf16', bits=4,
             actorder=True),
        # Every linear of a GPT-2-small-shaped model, 128 sequences of 512 tokens: the headline workload.
        dict(name='model_gpt2_n65536_f32', kind='model', layers=12, n=65536, batches=16, x='f32'),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(value, m):
    return max(m, value // m * m)


def draw(rng):
    kind = rng.choice(['matmul', 'matmul', 'matmul', 'grad', 'step', 'hessian', 'layer', 'layer', 'model'])
    if kind in ('matmul', 'grad'):
        M = _log_int(rng, 1, 2048)
        K, N = _log_int(rng, 256, 11008), _log_int(rng, 256, 32000)
        align = rng.choice([1, 16, 128])          # a third of the shapes as they fall, K even because two codes share a byte
        K, N = _multiple(K, max(2, align)), _multiple(N, align)
        return dict(kind=kind, M=M, K=K, N=N, x=rng.choice(['f16', 'bf16', 'f32']), zs=rng.choice(['f16', 'f32']))
    if kind == 'step':
        return dict(kind=kind, M=_log_int(rng, 1, 64), layers=rng.randint(2, 12), x=rng.choice(['f16', 'bf16']), zs='f32')
    if kind == 'hessian':
        K = _multiple(_log_int(rng, 256, 4096), rng.choice([4, 64]))
        batches = rng.choice([1, 4, 16])
        return dict(kind=kind, K=K, n=batches * _log_int(rng, 512, 65536 // batches), batches=batches,
                    x=rng.choice(['f32', 'bf16', 'f16']))
    if kind == 'layer':
        K = _multiple(_log_int(rng, 256, 4096), _BLOCK_SIZE)
        batches = rng.choice([1, 4, 8])
        return dict(kind=kind, K=K, N=_log_int(rng, 256, 8192), n=batches * _log_int(rng, 1024, 16384 // batches + 1024),
                    batches=batches, x=rng.choice(['f32', 'bf16']), bits=rng.choice([4, 4, 3]),
                    actorder=rng.random() < 0.25)
    return dict(kind=kind, layers=rng.randint(1, 4), n=16 * _log_int(rng, 256, 4096), batches=16, x='f32')


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def _quantized(gen, K, N, zs):
    """Uniform codes, scales ~ U(0.001, 0.02), whole zeros in [0, 15] (a layer's packed weights as loaded)."""
    packed = torch.randint(0, 256, (K // 2, N), generator=gen, dtype=torch.uint8, device='cuda')
    scale = (0.001 + 0.019 * torch.rand(N, generator=gen, device='cuda')).to(_DTYPES[zs])
    zero = torch.randint(0, 16, (N,), generator=gen, device='cuda').to(_DTYPES[zs])
    return _gptq.QuantizedMatrix(packed, zero, scale)


def _randn(gen, shape, dtype):
    return torch.randn(shape, generator=gen, device='cuda').to(_DTYPES[dtype])


def _activations(gen, n, K, dtype):
    """Calibration activations: features mixed by a random matrix with a decaying spectrum, plus a mean (inputs of
    attention and MLP layers are correlated); wide ones have been through the MLP's GELU."""
    spectrum = torch.exp(-4.0 * torch.arange(K, device='cuda') / K)
    mix = torch.randn((K, K), generator=gen, device='cuda') / math.sqrt(K) * spectrum[:, None]
    x = torch.randn((n, K), generator=gen, device='cuda') @ mix
    x += 0.2
    if K >= 3072:
        x = torch.nn.functional.gelu(x)
    return x.to(_DTYPES[dtype])


def _batches(x, count):
    return [b.clone() for b in x.chunk(count)]


def _layer_inputs(case, gen):
    W = 0.02 * torch.randn((case['K'], case['N']), generator=gen, device='cuda')
    return W.to(_DTYPES[case['x']]), _activations(gen, case['n'], case['K'], case['x'])


def _model_inputs(case, gen):
    jobs = []
    for _ in range(case['layers']):
        for K, N in _BLOCK:
            W = 0.02 * torch.randn((K, N), generator=gen, device='cuda')
            jobs.append((W, list(_activations(gen, case['n'], K, case['x']).chunk(case['batches']))))
    return jobs


def _matmul_inputs(case, gen):
    qm = _quantized(gen, case['K'], case['N'], case['zs'])
    return qm, _randn(gen, (case['M'], case['K']), case['x'])


def _step_inputs(case, gen):
    out = []
    for _ in range(case['layers']):
        for K, N in _BLOCK:
            out.append((_quantized(gen, K, N, case['zs']), _randn(gen, (case['M'], K), case['x'])))
    return out


def prepare(case, seed):
    gen = _generator(seed)
    kind = case['kind']
    if kind == 'matmul':
        qm, x = _matmul_inputs(case, gen)
        return dict(kind=kind, qm=qm, x=x)
    if kind == 'grad':
        qm, x = _matmul_inputs(case, gen)
        return dict(kind=kind, qm=qm, x=x.requires_grad_(), dy=_randn(gen, (case['M'], case['N']), case['x']))
    if kind == 'step':
        return dict(kind=kind, linears=_step_inputs(case, gen))
    if kind == 'hessian':
        return dict(kind=kind, xs=_batches(_activations(gen, case['n'], case['K'], case['x']), case['batches']))
    if kind == 'layer':
        W, x = _layer_inputs(case, gen)
        return dict(kind=kind, W=W, xs=_batches(x, case['batches']), bits=case['bits'], actorder=case['actorder'])
    return dict(kind=kind, jobs=_model_inputs(case, gen))


def _checkpoint(linears):
    """The linears' packed bytes, scales and zeros as three flat tensors, the form in which a program saves them."""
    return [torch.cat([t.reshape(-1) for t in column]) for column in zip(*linears)]


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    kind = state['kind']
    if kind == 'matmul':
        return _op.quantized_matmul(state['x'], state['qm'])
    if kind == 'grad':
        y = _op.quantized_matmul(state['x'], state['qm'])
        dx, = torch.autograd.grad(y, state['x'], state['dy'])
        return y.detach(), dx
    if kind == 'step':
        return [_op.quantized_matmul(x, qm) for qm, x in state['linears']]
    if kind == 'hessian':
        return _gptq.accumulate_H(state['xs'])
    if kind == 'layer':
        Q, params = _gptq.gptq(state['W'], state['xs'], block_size=_BLOCK_SIZE, damping=_DAMPING,
                               actorder=state['actorder'], bits=state['bits'])
        qm = _gptq.pack_matrix(Q, params)
        return Q, qm.scale, qm.zero, qm.int_weight
    res = _gptq.gptq_many(state['jobs'], block_size=_BLOCK_SIZE, damping=_DAMPING, streams=12)
    return _checkpoint([(q.int_weight, q.scale, q.zero) for q in res])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _matmul_work(case):
    M, K, N, b = case['M'], case['K'], case['N'], _BYTES[case['x']]
    return K * N / 2 + 2 * N * _BYTES[case['zs']] + M * (K + N) * b, 2.0 * M * K * N


def _hessian_work(n, K, b):
    return n * K * b, 1.0 * n * K * (K + 1)                       # the products on and below the diagonal


def _layer_work(n, K, N, b):
    xb, hf = _hessian_work(n, K, b)
    return xb + K * N * b + K * N / 2 + 8 * N, hf + 2.0 / 3.0 * K ** 3 + 1.0 * N * K * (K + 1)


def work(case):
    kind = case['kind']
    if kind == 'matmul':
        by, fl = _matmul_work(case)
    elif kind == 'grad':
        by, fl = _matmul_work(case)
        by, fl = by + case['M'] * (case['K'] + case['N']) * _BYTES[case['x']], 2 * fl
    elif kind == 'step':
        by, fl = 0.0, 0.0
        for K, N in _BLOCK * case['layers']:
            b, f = _matmul_work(dict(case, K=K, N=N))
            by, fl = by + b, fl + f
    elif kind == 'hessian':
        by, fl = _hessian_work(case['n'], case['K'], _BYTES[case['x']])
        by += 4 * case['K'] ** 2
    elif kind == 'layer':
        by, fl = _layer_work(case['n'], case['K'], case['N'], _BYTES[case['x']])
        by += case['K'] * case['N'] * _BYTES[case['x']]             # Q
    else:
        by, fl = 0.0, 0.0
        for K, N in _BLOCK * case['layers']:
            b, f = _layer_work(case['n'], K, N, _BYTES[case['x']])
            by, fl = by + b, fl + f
    return {'bytes': by, 'flops': fl}


# --------------------------------------------------------------------------
# how far another correct implementation may be off
# --------------------------------------------------------------------------
def tolerance(case):
    kind = case['kind']
    if kind in ('matmul', 'grad', 'step'):
        # 16-bit results: their rounding, 2.2e-4 and 1.8e-3.  fp32 activations enter the products as two 16-bit planes:
        # up to 3.1e-5 with the planes' own rounding and sums over 15000 channels.
        return {'rel': {'f32': 1.2e-4, 'f16': 1e-3, 'bf16': 8e-3}[case['x']]}
    if kind == 'hessian':
        return {'rel': 3e-6}
    # One code that falls the other way changes every later one of its channel, so that fp32 against fp64 differs in up
    # to 0.01 of the bytes with fp32 weights, 0.027 with bf16 ones at K = 2816 from 2215 rows.
    if kind == 'layer':
        return {'rel': 0.15, 'differ': 0.04} if case['x'] == 'f32' else {'rel': 0.2, 'differ': 0.1}
    return {'rel': 1e-6, 'differ': 0.018}


# --------------------------------------------------------------------------
# the same outputs in 64 bits
# --------------------------------------------------------------------------
def _dense(qm):
    w = qm.int_weight
    codes = torch.empty((2 * w.shape[0], w.shape[1]), dtype=torch.float64, device=w.device)
    codes[0::2] = (w & 15).double()
    codes[1::2] = (w >> 4).double()
    return codes.sub_(qm.zero.double()).mul_(qm.scale.double())


def _hessian64(x):
    K = x.shape[1]
    H = torch.zeros((K, K), dtype=torch.float64, device=x.device)
    for b in x.split(8192):
        b = b.double()
        H += b.T @ b
    return H / x.shape[0]


def _layer64(W, x, bits, actorder):
    """GPTQ of one layer: (Q, scale, zero, packed).  Scale and zero are part of the format: fp32 of an fp32 weight,
    where -lo / scale is often exactly half way between two whole numbers (bf16 weights with hi = -lo)."""
    W = W.float()
    K, N = W.shape
    maxq = 2 ** bits - 1
    lo, hi = W.amin(0).clamp(max=0.0), W.amax(0).clamp(min=0.0)
    lo, hi = torch.where(lo == 0, -torch.ones_like(lo), lo), torch.where(hi == 0, torch.ones_like(hi), hi)
    scale = (hi - lo) / torch.full_like(lo, maxq)               # a scalar divisor would become a multiplication
    zero = torch.round(-lo / scale).double()
    scale, W = scale.double(), W.double()
    H = _hessian64(x)
    perm = None
    if actorder:
        perm = torch.argsort(torch.diagonal(H), stable=True).flip(0)
        W, H = W[perm], H[perm][:, perm]
    d = torch.diagonal(H)
    dead = d == 0
    W[dead] = 0
    d[dead] = 1
    d += d.mean() * _DAMPING
    inv = torch.cholesky_inverse(torch.linalg.cholesky(H))
    L = torch.linalg.cholesky((inv + inv.T) / 2)
    codes = torch.empty_like(W)
    for s in range(0, K, _BLOCK_SIZE):
        e = s + _BLOCK_SIZE
        block, Lb, err = W[s:e], L[s:e, s:e], torch.empty_like(W[s:e])
        inv_d = 1.0 / torch.diagonal(Lb)
        for i in range(_BLOCK_SIZE):
            c = torch.clamp(torch.round(block[i] / scale) + zero, 0, maxq)
            codes[s + i] = c
            err[i] = (block[i] - (c - zero) * scale) * inv_d[i]
            block[i + 1:] -= Lb[i + 1:, i:i + 1] * err[i]
        W[e:] -= L[e:, s:e] @ err
    if perm is not None:
        codes = codes[torch.argsort(perm)]
    c8 = codes.to(torch.uint8)
    return (codes - zero) * scale, scale, zero, c8[0::2] | (c8[1::2] << 4)


def exact(case, seed):
    gen = _generator(seed)
    kind = case['kind']
    if kind in ('matmul', 'grad'):
        qm, x = _matmul_inputs(case, gen)
        w = _dense(qm)
        y = x.double() @ w
        if kind == 'matmul':
            return y
        return y, _randn(gen, (case['M'], case['N']), case['x']).double() @ w.T
    if kind == 'step':
        return [x.double() @ _dense(qm) for qm, x in _step_inputs(case, gen)]
    if kind == 'hessian':
        return _hessian64(_activations(gen, case['n'], case['K'], case['x']))
    if kind == 'layer':
        W, x = _layer_inputs(case, gen)
        return _layer64(W, x, case['bits'], case['actorder'])
    out = []
    for W, xs in _model_inputs(case, gen):
        _, scale, zero, packed = _layer64(W, torch.cat(xs), 4, False)
        out.append((packed, scale, zero))
    return _checkpoint(out)
