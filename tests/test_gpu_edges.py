"""Sizes and values at the edges of the kernels' tiles, ranges and dispatch rules, against the oracle or against
the general path."""
import importlib

import numpy as np
import pytest
import torch

from oracle import ref_gptq as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def gg():
    return importlib.import_module('jax_gptq_b200.gptq')


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def second_moment(rng, K):
    A = rng.standard_normal((K, K)).astype(np.float32) / np.sqrt(K)
    return R.accumulate_H([(rng.standard_normal((4 * K, K)).astype(np.float32) @ A).astype(np.float32)])


@pytest.mark.parametrize('K', [1, 15, 16, 17, 63, 65, 130, 198, 257, 322])     # rows of 4 floats and not, one panel to two outer blocks
def test_damp_invert_partial_panels_and_unaligned_rows(gg, K):
    rng = np.random.default_rng(500 + K)
    H = second_moment(rng, K)
    W = dev(np.ones((K, 3), np.float32))
    L, status = gg._damp_and_invert(W, dev(H), 0.01)
    assert int(status.item()) == 0
    L = L.cpu().numpy().astype(np.float64)
    Hdamp = H.astype(np.float64) + np.eye(K) * float(np.mean(np.diag(H)) * np.float32(0.01))
    _, L_ref, _ = R.damp_and_invert(np.ones((K, 3), np.float32), H, 0.01)
    ref = np.abs(L_ref.astype(np.float64) @ L_ref.astype(np.float64).T @ Hdamp - np.eye(K)).max()
    assert np.abs(L @ L.T @ Hdamp - np.eye(K)).max() <= max(4 * ref, 1e-5)
    assert np.all(np.triu(L, 1) == 0)


@pytest.mark.parametrize('K', [16, 100, 320])
def test_damp_invert_scaled_by_powers_of_four(gg, K):
    """Every operation of the factorization commutes with a scaling of H by a power of four, so the results are the
    same bits times a power of two; 2^-104 and 2^100 put the pivots outside the range of the fast root and quotients."""
    H = dev(second_moment(np.random.default_rng(600 + K), K))
    W = torch.ones((K, 3), device='cuda')
    L, _ = gg._damp_and_invert(W, H.clone(), 0.01)
    for e in (-104, 100):
        Ls, status = gg._damp_and_invert(W, H * 2.0 ** e, 0.01)
        assert int(status.item()) == 0
        assert torch.equal(Ls * 2.0 ** (e // 2), L)


@pytest.mark.parametrize('K,N,bs', [(256, 33, 128), (384, 96, 96), (300, 70, 100), (256, 130, 64), (96, 5, 48), (120, 64, 20),
                                    (640, 31, 128)])
def test_quantize_loop_several_blocks_any_width(gg, K, N, bs):
    """Ragged channel counts, blocks that are no multiple of a sub-block, rows of W that are not 16-byte aligned: codes
    against the oracle's loop run with the same factor.  Codes differ only where the lazy update's last bits decide a
    rounding (its products carry 22 bits, sums of 128 of them): at most 0.1 % of them, the bar of the layer tests."""
    rng = np.random.default_rng(700 + K + N)
    W = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
    _, L, _ = R.damp_and_invert(W, second_moment(rng, K), 0.01)
    L = L.astype(np.float32)
    params = R.get_col_quantize_params(W)
    Wr, blocks = W.copy(), []
    for s in range(0, K, bs):
        q, err = R.process_block(Wr, L, s, params, bs)
        Wr[s + bs:] -= (L[s + bs:, s:s + bs] @ err).astype(np.float32)
        blocks.append(q)
    Q = np.concatenate(blocks)
    want = np.round(Q / params['scale'] + params['zero']).astype(np.uint8)
    dp = {'scale': dev(params['scale']), 'zero': dev(params['zero']), 'maxq': 15}
    Qd, codes = gg._quantize(dev(W), dev(L), dp, bs, torch.float32, want_codes=True)
    codes = codes.cpu().numpy()
    assert (codes != want).mean() <= 1e-3
    assert np.array_equal(codes[:bs], want[:bs])                       # the first block has no lazy update
    assert np.array_equal(Qd.cpu().numpy(), (params['scale'] * (codes.astype(np.float32) - params['zero'])).astype(np.float32))


def test_quantize_loop_values_outside_the_fast_quotients(gg):
    """Scales, pivots and weights outside the range of the corrected quotients take the plain divisions: one block,
    bit-identical to the oracle (tiny, huge and zero scales of weights, an infinite weight, a large zero point)."""
    K = N = 64
    rng = np.random.default_rng(800)
    W = (0.02 * rng.standard_normal((K, N))).astype(np.float32)
    W[:, 3] *= np.float32(1e-38)
    W[:, 4] *= np.float32(1e30)
    W[:, 5] = 0
    W[7, 6] = np.inf
    L = np.tril(0.05 * rng.standard_normal((K, K))).astype(np.float32)
    L[np.arange(K), np.arange(K)] = np.linspace(0.5, 2.0, K, dtype=np.float32)
    scale = np.full(N, 0.004, np.float32)
    zero = np.full(N, 8, np.float32)
    scale[1], scale[2], zero[8] = 1e-30, 1e30, 3e6
    params = {'scale': scale, 'zero': zero, 'maxq': 15}
    with np.errstate(all='ignore'):
        Q, _ = R.process_block(W, L, 0, params, K)
    Qd, _ = gg._quantize(dev(W), dev(L), {'scale': dev(scale), 'zero': dev(zero), 'maxq': 15}, K, torch.float32)
    got = Qd.cpu().numpy()
    ok = np.isfinite(Q) & (np.arange(N) != 6)[None, :]                  # behind the infinite weight clip(NaN) is the host's choice
    assert np.array_equal(got[ok], Q[ok])


@pytest.mark.parametrize('K,ns,dtype', [(512, (600, 1333, 2048, 777), torch.float32), (768, (1024,) * 4, torch.float32),
                                        (1800, (1500, 4096, 5000), torch.bfloat16), (1024, (512, 100, 700), torch.float32),
                                        (1032, (2048,) * 5, torch.float16), (2048, (1024,) * 17, torch.bfloat16),
                                        (3072, (4096,) * 3, torch.float32), (256, (1000, 600), torch.float32),
                                        (300, (700, 40), torch.float16)])
def test_hessian_of_separate_batches_equals_one_by_one(gg, K, ns, dtype):
    """Batches that share a launch (tile by tile, batch by batch or slice by slice, whichever the plan takes), batches too
    small or too odd for it, and more than fit one call: the bits of one call per batch."""
    g = torch.Generator(device='cuda').manual_seed(K + len(ns))
    xs = [(torch.randn((n, K), generator=g, device='cuda') + 0.3).to(dtype) for n in ns]
    together, n = gg._accumulate_raw(xs)
    assert n == sum(ns)
    H = torch.zeros((K, K), device='cuda')
    for x in xs:
        gg._accumulate_raw([x], H=H)
    assert torch.equal(together.tril(), H.tril())
    ref = sum(x.double().T @ x.double() for x in xs)
    assert ((together.double() - ref).tril().norm() / ref.tril().norm()).item() < 3e-6


@pytest.mark.parametrize('M', [1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('K,N', [(8, 16), (136, 48), (3080, 144), (768, 2304)])
def test_matmul_decode_rows_types_and_ragged_edges(gg, M, dtype, K, N):
    """Token counts around the groups of eight, channel groups that are not full, contraction ranges that end inside a
    box.  Against the dequantized product in fp64: the output's rounding (2^-11, 2^-8, or the two bf16 planes' 2^-17 with
    fp32 sums over at most 3080 terms), in the 2-norm."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(1000 * M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    zs = torch.float32 if M % 2 else torch.float16
    scale = (0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')).to(zs)
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').to(zs)
    x = torch.randn((M, K), generator=g, device='cuda').to(dtype)
    dense = (torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - zero.double()) * scale.double()
    want = x.double() @ dense
    bound = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]
    first = None
    for _ in range(3):                                  # the later calls fetch weights early
        got = quantized_matmul(x, QuantizedMatrix(packed, zero, scale))
        assert ((got.double() - want).norm() / want.norm()).item() <= bound
        assert first is None or torch.equal(got, first)
        first = got


@pytest.mark.parametrize('M,dtype,passes', [(24, torch.float16, 2), (32, torch.bfloat16, 2), (12, torch.float32, 1), (20, torch.float32, 2)])
def test_matmul_with_the_smallest_workspace_it_accepts(gg, M, dtype, passes):
    """The slices of 32 rows are larger than what a call is refused without; with the least workspace 16-bit activations
    take the decode kernel in passes of 16 rows: the bits of separate calls for those rows."""
    from jax_gptq_b200 import _lib
    lib = _lib.lib
    N, K = 2048, 8192
    g = torch.Generator(device='cuda').manual_seed(M)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale, zero = torch.rand(N, generator=g, device='cuda') * 0.01, torch.full((N,), 8.0, device='cuda')
    x = torch.randn((M, K), generator=g, device='cuda').to(dtype)
    full = lib.jgq_w4_matmul_workspace_bytes(M, N, K, 0)
    ws = torch.zeros(full, dtype=torch.uint8, device='cuda')

    def call(rows, nbytes):
        out = torch.full((rows.shape[0], N), float('nan'), dtype=dtype, device='cuda')
        before = lib.jgq_launch_count()
        rc = lib.jgq_w4_matmul(rows.data_ptr(), gg._DT[dtype], packed.data_ptr(), zero.data_ptr(), scale.data_ptr(), _lib.F32,
                               out.data_ptr(), rows.shape[0], N, K, 0, ws.data_ptr(), nbytes, gg._stream())
        assert rc in (0, -3)
        return (out, lib.jgq_launch_count() - before) if rc == 0 else None
    refused, least = 0, full
    while least - refused > 1:
        mid = (least + refused) // 2
        if call(x, mid) is None:
            refused = mid
        else:
            least = mid
    want = x.double() @ ((torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - 8) * scale.double())
    bound = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]
    for nbytes in (least, least + 256, full):
        out, launches = call(x, nbytes)
        assert ((out.double() - want).norm() / want.norm()).item() <= bound
        if nbytes <= least + 256:
            assert launches == passes
            if dtype != torch.float32:
                assert least < full
                assert torch.equal(out, torch.cat([call(x[:16], full)[0], call(x[16:], full)[0]]))
        elif dtype != torch.float32:
            assert launches == 1
    assert call(x, least - 1) is None
    assert int(ws[:16384].sum()) == 0                    # the tickets are back at zero


def _some_matrix(K=256, N=128):
    from jax_gptq_b200 import QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(5)
    return QuantizedMatrix(torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8),
                           torch.full((N,), 8.0, device='cuda'), torch.rand(N, generator=g, device='cuda') * 0.01)


def test_matmul_outside_and_inside_autograd(gg):
    """A product that nothing differentiates is launched directly; with gradients (of the input, or recorded for the
    scales), under forward mode and under a functorch transform it still goes through the autograd function."""
    from jax_gptq_b200 import quantized_matmul
    qm = _some_matrix()
    x = torch.randn((2, 3, 256), device='cuda')
    plain = quantized_matmul(x, qm)
    assert plain.shape == (2, 3, 128) and not plain.requires_grad
    xg = x.clone().requires_grad_()
    y = quantized_matmul(xg, qm)
    assert y.requires_grad and torch.equal(y.detach(), plain)
    y.sum().backward()
    assert torch.equal(xg.grad, quantized_matmul(torch.ones_like(y), qm, transpose_b=True))
    with torch.no_grad():
        assert not quantized_matmul(xg, qm).requires_grad
    qm.scale.requires_grad_()
    assert quantized_matmul(x, qm).requires_grad
    qm.scale.requires_grad_(False)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        with pytest.raises(RuntimeError):
            quantized_matmul(dual, qm)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda r: quantized_matmul(r, qm))(x)
    assert torch.equal(quantized_matmul(x.transpose(0, 1), qm), plain.transpose(0, 1))
    assert torch.equal(quantized_matmul(torch.nn.Parameter(x, requires_grad=False), qm), plain)
    with pytest.raises(ValueError):
        quantized_matmul(x[0, 0], qm)
    traced = torch.jit.trace(lambda t: quantized_matmul(t, qm), (x,), check_trace=False)
    other = torch.randn_like(x)
    assert torch.equal(traced(other), quantized_matmul(other, qm))


@pytest.mark.parametrize('M,K,N', [(33, 64, 256), (1, 136, 16), (20, 4104, 400), (256, 520, 272), (257, 1032, 528), (300, 128, 272),
                                   (513, 4104, 400), (700, 3080, 1040), (1025, 72, 2064)])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('transpose', [False, True])
def test_matmul_many_rows_edges_of_tiles(gg, M, K, N, dtype, transpose):
    """Tiles of 256 weight rows by 256 or 512 tokens that are not full, contractions that end inside a stage, both
    directions.  Against the dequantized product in fp64: the output's rounding, or for fp32 the planes' 2^-17 and
    fp32 sums."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    x = torch.randn((M, N if transpose else K), generator=g, device='cuda').to(dtype)
    dense = (torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - zero.double()) * scale.double()
    want = x.double() @ (dense.T if transpose else dense)
    qm = QuantizedMatrix(packed, zero, scale)
    got = quantized_matmul(x, qm, transpose_b=transpose)
    bound = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]
    assert ((got.double() - want).norm() / want.norm()).item() <= bound
    assert torch.equal(got, quantized_matmul(x, qm, transpose_b=transpose))


@pytest.mark.parametrize('M,K,N', [(65, 256, 4096), (97, 136, 272), (150, 72, 640), (200, 512, 4800), (512, 136, 8208),
                                   (768, 136, 8208), (1300, 200, 10256), (2300, 72, 10256)])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('transpose', [False, True])
def test_matmul_many_rows_blocks_and_rounds(gg, M, K, N, dtype, transpose):
    """Blocks of fewer than 256 tokens, and work lists of several items per pair of SMs (whole rounds, halved
    items, a last odd column), in both directions: the weights' sides are exchanged for the transposed product.
    Against the dequantized product in fp64, the whole and each element."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    if transpose:
        K, N = N, K // 16 * 16
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    x = torch.randn((M, N if transpose else K), generator=g, device='cuda').to(dtype)
    dense = (torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - zero.double()) * scale.double()
    want = x.double() @ (dense.T if transpose else dense)
    got = quantized_matmul(x, QuantizedMatrix(packed, zero, scale), transpose_b=transpose)
    bound = {torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]
    assert ((got.double() - want).norm() / want.norm()).item() <= bound
    # no element is missing or misplaced: 16 x the bound, of the element and its row together (a missing stage or tile is of order one)
    row = want.norm(dim=1, keepdim=True) / want.shape[1] ** 0.5
    assert ((got.double() - want).abs() / (row + want.abs())).max().item() <= 16 * bound


@pytest.mark.parametrize('M', [1, 2, 8, 16, 17, 24, 32, 33, 64])
@pytest.mark.parametrize('K,N', [(768, 2304), (136, 48), (270, 37)])
def test_matmul_small_f16_activations(gg, M, K, N):
    """f16 activations far below one, rows of different magnitudes: every one enters the product as it is, so all that is
    lost is the output's rounding, 2^-11 of the value or half a step of the subnormals (2^-25), row by row."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(M + K)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    dense = (torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - zero.double()) * scale.double()
    for s in (1e-3, 1e-4, 1e-5):
        x = (torch.randn((M, K), generator=g, device='cuda') * s * 2.0 ** -(torch.arange(M, device='cuda') % 3)[:, None]).half()
        want = x.double() @ dense
        err = (quantized_matmul(x, QuantizedMatrix(packed, zero, scale)).double() - want).norm(dim=1)
        assert torch.all(err <= 2.0 ** -11 * want.norm(dim=1) + 2.0 ** -25 * N ** 0.5)


@pytest.mark.parametrize('M,K,N', [(1, 256, 1024), (137, 768, 1024), (300, 272, 4112), (1, 256, 909), (64, 768, 909), (137, 256, 909)])
@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
def test_transposed_matmul_of_any_magnitude(gg, M, K, N, dtype):
    """Gradients of a mean over many tokens are far below one, scaled losses far above: both kernels of the transposed
    product, rows of different magnitudes and rows of zeros in one call.  Row by row against fp64: the output's rounding,
    and the planes' 2^-22 with fp32 sums over up to 4112 channels, which are of the codes and of the zero points apart:
    2e-5 of either one's norm, also where their difference is smaller."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    dense = (torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - zero.double()) * scale.double()
    qm = QuantizedMatrix(packed, zero, scale)
    offset = zero.double() * scale.double()
    bound = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 0.0}[dtype]
    floor = 2.0 ** -25 * K ** 0.5 if dtype == torch.float16 else 0.0         # half a step of f16's subnormals
    for s in (1.0, 1e-3, 1e-4) if dtype == torch.float16 else (1.0, 1e-3, 1e-4, 1e-5, 1e-6, 1e-8, 1e-30, 1e6, 1e20):
        row = torch.tensor([1.0, 2.0 ** -6, 3.0, 0.0])[torch.arange(M) % 4].cuda()[:, None]
        x = (torch.randn((M, N), generator=g, device='cuda') * s * row).to(dtype)
        want = x.double() @ dense.T
        got = quantized_matmul(x, qm, transpose_b=True)
        parts = (want + (x.double() @ offset)[:, None]).norm(dim=1) + (x.double() @ offset).abs() * K ** 0.5
        assert torch.all((got.double() - want).norm(dim=1) <= bound * want.norm(dim=1) + 2e-5 * parts + floor)
    # beside an infinity and a NaN the other rows keep their values
    if M > 4:
        x[1, 5], x[2, 7] = float('inf'), float('nan')
        again = quantized_matmul(x, qm, transpose_b=True)
        keep = torch.ones(M, dtype=torch.bool, device='cuda')
        keep[1] = keep[2] = False
        assert torch.equal(again[keep], got[keep]) and not torch.isfinite(again[1]).any() and torch.isnan(again[2]).all()


@pytest.mark.parametrize('M', [1, 64, 128, 200])
def test_transposed_matmul_in_the_least_workspace(gg, M):
    """The least a call is accepted with: whole tiles of 64 rows and four bytes a row, too little for all rows in one
    pass where M is a multiple of the tile."""
    from jax_gptq_b200 import _lib
    lib = _lib.lib
    K, N = 128, 200
    g = torch.Generator(device='cuda').manual_seed(M)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale, zero = torch.rand(N, generator=g, device='cuda') * 0.01, torch.full((N,), 8.0, device='cuda')
    x = torch.randn((M, N), generator=g, device='cuda')
    up = lambda v: (v + 255) // 256 * 256
    least = 16384 + 2 * up((M + 63) // 64 * 64 * 256 * 2) + up(4 * M)
    ws = torch.zeros(lib.jgq_w4_matmul_workspace_bytes(M, N, K, 1), dtype=torch.uint8, device='cuda')
    want = x.double() @ ((torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double() - 8) * scale.double()).T
    for nbytes, rc in ((least - 1, -3), (least, 0), (ws.numel(), 0)):
        out = torch.full((M, K), float('nan'), device='cuda')
        assert lib.jgq_w4_matmul(x.data_ptr(), _lib.F32, packed.data_ptr(), zero.data_ptr(), scale.data_ptr(), _lib.F32,
                                 out.data_ptr(), M, N, K, _lib.W4_TRANSPOSE_B, ws.data_ptr(), nbytes, gg._stream()) == rc
        if rc == 0:
            assert ((out.double() - want).norm() / want.norm()).item() <= 2e-5
    assert int(ws[:16384].sum()) == 0


@pytest.mark.parametrize('dtype', [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize('M', [1, 8, 16])
def test_matmul_products_that_feed_one_another(gg, M, dtype):
    """Each product starts while the one that writes its activations is finishing, and the allocator hands the same few
    buffers around: the bits of the same chain with a synchronisation after every product."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    K = 1024
    g = torch.Generator(device='cuda').manual_seed(M)
    qms = [QuantizedMatrix(torch.randint(0, 256, (K // 2, K), generator=g, device='cuda', dtype=torch.uint8),
                           torch.full((K,), 7.5, device='cuda'), 0.0065 * (0.9 + 0.2 * torch.rand(K, generator=g, device='cuda'))) for _ in range(4)]
    x = torch.randn((M, K), generator=g, device='cuda').to(dtype)

    def chain(sync):
        y = x
        for i in range(48):
            y = quantized_matmul(y, qms[i % 4])
            if sync:
                torch.cuda.synchronize()
        return y
    want = chain(True)
    assert torch.isfinite(want).all() and want.abs().max() > 0
    for _ in range(5):
        assert torch.equal(chain(False), want)


@pytest.mark.parametrize('widths', [(64, 128), (128, 64), (512, 512, 520)])
@pytest.mark.parametrize('use_fp64', [False, True])
def test_hessian_refuses_batches_of_another_width(gg, widths, use_fp64):
    """A wider batch would be added beyond the matrix that the first one was given."""
    xs = [torch.randn((600, K), device='cuda') for K in widths]
    with pytest.raises(ValueError, match='features'):
        gg.accumulate_H(xs, use_fp64=use_fp64)
    assert torch.isfinite(gg.accumulate_H(xs[:1], use_fp64=use_fp64)).all()


@pytest.mark.parametrize('K,ns', [(512, (600, 1333, 2048, 777)), (4096, (1024,) * 3)])      # sums by way of buffers, and added to H tile by tile
def test_hessian_bounded_wait_of_several_batches(gg, K, ns, monkeypatch):
    """Waits that run out while several batches share a launch: the call raises, H is then undefined, and the next call with
    a fresh one is correct again."""
    g = torch.Generator(device='cuda').manual_seed(K)
    xs = [torch.randn((n, K), generator=g, device='cuda') for n in ns]
    before = gg.accumulate_H(xs)
    monkeypatch.setenv('JGQ_TEST_WITHHOLD_COMMIT', '1')
    with pytest.raises(RuntimeError, match='timed out'):
        gg.accumulate_H(xs)
    monkeypatch.delenv('JGQ_TEST_WITHHOLD_COMMIT')
    assert torch.equal(gg.accumulate_H(xs), before)


@pytest.mark.parametrize('parity', [0, 1])
def test_damp_invert_roots_and_reciprocals_of_many_mantissas(gg, parity):
    """A diagonal matrix is factored pivot by pivot: the factor of its inverse is 1 / sqrt, both operations IEEE's, bit for
    bit; every 32nd mantissa, the neighbours of the powers of two, and pivots whose root has the largest mantissa, in both
    exponent parities, and the values at which the fast form hands over to the plain one."""
    K = 4096
    m = np.concatenate([np.arange(parity, 1 << 23, 32), np.arange(64), (1 << 23) - 1 - np.arange(64)]).astype(np.uint32)
    a = (m | np.uint32((127 + parity) << 23)).view(np.float32)
    edge = np.float32([2.0 ** -96, 2.0 ** 96, np.nextafter(np.float32(2.0 ** -96), np.float32(0)), np.nextafter(np.float32(2.0 ** 96), np.float32(np.inf)), 1e-37, 1e37])
    a = np.concatenate([a, edge, np.ones(-(len(a) + len(edge)) % K, np.float32)])
    want = np.float32(1) / np.sqrt(a)
    W = torch.zeros((K, 1), device='cuda')
    for s in range(0, len(a), K):
        L, status = gg._damp_and_invert(W, torch.diag(dev(a[s:s + K])), 0.0)
        assert int(status.item()) == 0
        assert np.array_equal(torch.diagonal(L).cpu().numpy(), want[s:s + K])
    assert torch.count_nonzero(L) == K


def test_matmul_tensor_path_on_the_single_cta_kernel():
    """Which tensor-core kernel a product takes depends on its sizes.  With JGQ_W4_PATH=stream, read once per process, more
    than 32 rows all take the single-CTA kernel: the ring depths, split contractions, two planes and launches of hundreds of
    CTAs that `test_matmul_tensor_path_every_channel_group` and `test_matmul_many_ctas_repeatable` list, in a process of its own."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, '-m', 'pytest', '-q', '-x', '-p', 'no:cacheprovider', os.path.join(here, 'test_gpu_parity.py'),
                        '-k', 'every_channel_group or many_ctas_repeatable'], env=dict(os.environ, JGQ_W4_PATH='stream'),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:]
    assert '11 passed' in r.stdout


@pytest.mark.parametrize('M,K,N,dtype', [(9, 5120, 8192, torch.float32), (9, 5112, 8192, torch.float32), (16, 5128, 8208, torch.float32),
                                         (5, 7680, 8192, torch.float32), (4, 7680, 8192, torch.float32), (32, 24576, 4096, torch.float32),
                                         (8, 24584, 4096, torch.float32), (17, 8192, 12288, torch.float16), (16, 8192, 12288, torch.float16),
                                         (24, 8200, 12304, torch.bfloat16), (25, 8192, 12288, torch.bfloat16), (1, 8192, 20480, torch.bfloat16),
                                         (32, 20488, 8192, torch.float16)])
def test_matmul_decode_rows_of_large_weights(gg, M, K, N, dtype):
    """Both sides of the lines between the decode kernel and the streaming kernel, against the dequantized product in fp64:
    the output's rounding, or the planes' 2^-17 and fp32 sums.  f16 activations of 1e-4 among them."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    x = (torch.randn((M, K), generator=g, device='cuda') * torch.tensor([1.0, 1e-4], device='cuda')[torch.arange(M, device='cuda') % 2][:, None]).to(dtype)
    got = quantized_matmul(x, QuantizedMatrix(packed, zero, scale))
    assert torch.equal(got, quantized_matmul(x, QuantizedMatrix(packed, zero, scale)))
    bound = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2e-5}[dtype]
    for c in range(0, N, 2048):
        w = packed[:, c:c + 2048]
        want = x.double() @ ((torch.stack([w & 15, w >> 4], 1).reshape(K, -1).double() - zero[c:c + 2048].double()) * scale[c:c + 2048].double())
        assert torch.all((got[:, c:c + 2048].double() - want).norm(dim=1) <= bound * want.norm(dim=1))


@pytest.mark.parametrize('M,N', [(150, 1024), (150, 1040), (300, 2048), (300, 2064), (149, 4096), (148, 4096), (149, 4112), (2, 8192), (3, 8208), (150, 16400), (150, 1025)])
@pytest.mark.parametrize('dtype,zs', [(torch.bfloat16, torch.float32), (torch.float32, torch.float16)])
@pytest.mark.parametrize('shift', [0, 1])
def test_transposed_matmul_rows_of_any_length_and_alignment(gg, M, N, dtype, zs, shift):
    """Row lengths and counts at which the kernel in front changes its block, rows that it keeps in registers and longer ones;
    activations, scales and zero points that do not start on 16 bytes (or on 8)."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    K = 64
    g = torch.Generator(device='cuda').manual_seed(M + N)

    def moved(t):
        flat = torch.zeros(t.numel() + 16, dtype=t.dtype, device='cuda')
        flat[shift:shift + t.numel()] = t.reshape(-1)
        return flat[shift:shift + t.numel()].view(t.shape)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = moved((0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')).to(zs))
    zero = moved(torch.randint(0, 16, (N,), generator=g, device='cuda').to(zs))
    x = moved((torch.randn((M, N), generator=g, device='cuda') * 1e-5).to(dtype))
    codes = torch.stack([packed & 15, packed >> 4], 1).reshape(K, N).double()
    want = x.double() @ ((codes - zero.double()) * scale.double()).T
    parts = x.double() @ (codes * scale.double()).T                        # sums of the codes and of the zero points, apart
    got = quantized_matmul(x, QuantizedMatrix(packed, zero, scale), transpose_b=True).double()
    # fp32 sums in one chain over N: a tensor core drops what lies below the accumulator's last bit at each of N / 16 steps
    # (two planes: N / 8), at most 2^-23 of it, half of that on average; the accumulator grows with the steps: N / 8 x 2^-25 of its end
    bound = {torch.bfloat16: 2.0 ** -8, torch.float32: 0.0}[dtype]
    sums = max(2e-5, N / 8 * 2.0 ** -25)
    assert torch.all((got - want).norm(dim=1) <= bound * want.norm(dim=1) + sums * (parts.norm(dim=1) + (parts - want).norm(dim=1)))


@pytest.mark.parametrize('M,K,N', [(33, 8192, 256), (64, 8192, 256), (64, 4096, 4096), (150, 4096, 256), (8, 8192, 20480), (17, 8192, 20480), (16, 5120, 8192)])
def test_matmul_fp32_keeps_its_precision_on_long_contractions(gg, M, K, N):
    """fp32 activations: the planes' 2^-17 (2.2e-6 in the 2-norm) and sums whose chains are cut.  One chain over 8192 indices loses
    1.5e-5, codes with an offset of 128 4e-6 to 5e-6."""
    from jax_gptq_b200 import quantized_matmul, QuantizedMatrix
    g = torch.Generator(device='cuda').manual_seed(M + K + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device='cuda', dtype=torch.uint8)
    scale = 0.001 + 0.019 * torch.rand(N, generator=g, device='cuda')
    zero = torch.randint(0, 16, (N,), generator=g, device='cuda').float()
    x = torch.randn((M, K), generator=g, device='cuda')
    got = quantized_matmul(x, QuantizedMatrix(packed, zero, scale))
    err = ref = 0.0
    for c in range(0, N, 2048):
        w = packed[:, c:c + 2048]
        want = x.double() @ ((torch.stack([w & 15, w >> 4], 1).reshape(K, -1).double() - zero[c:c + 2048].double()) * scale[c:c + 2048].double())
        err += (got[:, c:c + 2048].double() - want).square().sum().item()
        ref += want.square().sum().item()
    assert (err / ref) ** 0.5 <= 3.6e-6
