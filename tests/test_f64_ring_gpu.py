"""The FP64 ring kernel (uniform FP64 batches up to 128^3 with the N x K B
layout, and FP64 plans) at the edges of its cut: parts of 16 tiles and the
next size, parts copied whole and in chunks of K, several problems to a part,
rows a multiple of 128 bytes apart (exchanged k-steps) and not, strided rows,
partial k-steps, one chunk and many laps of the ring, alpha / beta.  Integer
inputs against the oracle: exact."""
import numpy as np
import pytest
import torch

import oracle
from kami_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,batch", [
    (64, 64, 64, 700), (65, 64, 64, 300), (33, 64, 34, 5), (1, 33, 2, 900), (40, 24, 32, 900),  # 16 tiles, cut, tiny
    (120, 32, 64, 200), (128, 32, 128, 200), (128, 128, 128, 160), (121, 91, 110, 160),         # chunks of K
    (96, 96, 96, 300), (48, 48, 96, 300), (8, 64, 64, 1200), (34, 18, 6, 700), (20, 100, 10, 1),  # whole parts
    (24, 24, 24, 3000), (32, 32, 32, 2000), (17, 31, 30, 4001), (18, 20, 22, 5003),              # shared parts
])
@pytest.mark.parametrize("pad", [0, 2, 8])
def test_uniform_exact(cuda, M, N, K, batch, pad):
    rng = np.random.default_rng(M * 1000 + N * 10 + K + pad)
    A = rng.integers(-9, 10, (batch, M, K + pad)).astype(np.float64)
    B = rng.integers(-9, 10, (batch, N, K + pad)).astype(np.float64)
    if pad:  # what lies between the rows must not matter
        A[:, :, K:] = np.nan
        B[:, :, K:] = np.inf
    C = api.gemm_batched(torch.tensor(A, device="cuda")[:, :, :K], torch.tensor(B, device="cuda")[:, :, :K])
    assert np.array_equal(C.cpu().numpy(), oracle.gemm(np.ascontiguousarray(A[:, :, :K]),
                                                       np.ascontiguousarray(B[:, :, :K])))


@pytest.mark.parametrize("M,N,K", [(64, 64, 64), (33, 47, 18), (121, 91, 110), (24, 32, 32)])
def test_alpha_beta_repeats_and_unaligned_c(cuda, M, N, K):
    rng = np.random.default_rng(M)
    batch = 1500
    A = rng.integers(-4, 5, (batch, M, K)).astype(np.float64)
    B = rng.integers(-4, 5, (batch, N, K)).astype(np.float64)
    C0 = rng.integers(-4, 5, (batch, M, N + 1)).astype(np.float64)
    C = torch.tensor(C0, device="cuda")
    api.gemm_batched(torch.tensor(A, device="cuda"), torch.tensor(B, device="cuda"), C[:, :, :N], alpha=2.0,
                     beta=-3.0, num_iter=2)
    want = C0.copy()
    want[:, :, :N] = 4.0 * oracle.gemm(A, B) - 3.0 * C0[:, :, :N]
    assert np.array_equal(C.cpu().numpy(), want)


def test_shared_operands(cuda):
    """Problem stride 0: every problem reads the same A and B."""
    rng = np.random.default_rng(3)
    A, B = (rng.integers(-9, 10, (1, 48, 40)).astype(np.float64) for _ in range(2))
    dA, dB = (torch.tensor(x, device="cuda").expand(400, 48, 40) for x in (A, B))
    C = api.gemm_batched(dA, dB)
    assert np.array_equal(C.cpu().numpy(), np.broadcast_to(oracle.gemm(A, B), (400, 48, 48)))
