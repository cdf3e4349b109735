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
