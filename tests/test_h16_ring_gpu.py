"""The 16-bit ring kernel (uniform FP16 / BF16 batches of small or ragged
blocks, and their plans) at the edges of its rules: accumulators of 64 columns
and of 128, rows in each of the four lane groups (M up to 32, 64, 96, 128), K in
one chunk and two with partial k-steps, rows stored whole and in pieces, every
output type, alpha / beta, strided and shared operands, one problem and more
than the ring holds.  Integer inputs against the oracle: exact in FP32."""
import numpy as np
import pytest
import torch

import oracle
from kami_b200 import api

pytestmark = pytest.mark.gpu

SHAPES = [(100, 16, 40, 900), (16, 104, 40, 5000), (24, 100, 72, 2000), (20, 20, 128, 900), (31, 33, 8, 9000),
          (32, 64, 64, 900), (33, 40, 128, 700), (64, 56, 64, 800), (40, 120, 24, 900), (64, 8, 72, 900),
          (97, 24, 56, 1), (128, 24, 128, 900), (65, 9, 16, 9000), (9, 128, 120, 3000), (1, 40, 40, 200),
          (32, 32, 32, 5000), (17, 31, 24, 11000)]


def _ints(rng, shape, dtype):
    x = rng.integers(-3, 4, shape).astype(np.float64)
    return x, torch.tensor(x, dtype=dtype, device="cuda")


@pytest.mark.parametrize("M,N,K,batch", SHAPES)
@pytest.mark.parametrize("dtype,out", [(torch.float16, torch.float32), (torch.bfloat16, torch.float32),
                                       (torch.float16, torch.float16)])
def test_uniform_exact(cuda, M, N, K, batch, dtype, out):
    rng = np.random.default_rng(M * 1000 + N * 10 + K)
    A, dA = _ints(rng, (batch, M, K), dtype)
    B, dB = _ints(rng, (batch, N, K), dtype)
    C = api.gemm_batched(dA, dB, out_dtype=out)
    want = torch.tensor(oracle.gemm(A, B), dtype=torch.float32).to(out)
    assert torch.equal(C.cpu(), want)


@pytest.mark.parametrize("M,N,K", [(100, 16, 40), (24, 100, 72), (40, 56, 64), (33, 41, 128)])
def test_alpha_beta_and_strides(cuda, M, N, K):
    """Strided rows and problems (what lies between must not matter), C with
    its own row stride, alpha and beta, repeats."""
    rng = np.random.default_rng(N)
    batch, pad = 1500, 8
    A, dA = _ints(rng, (batch, M, K + pad), torch.float16)
    B, dB = _ints(rng, (batch, N, K + pad), torch.float16)
    dA[:, :, K:] = float("nan")
    dB[:, :, K:] = float("inf")
    C0, C = _ints(rng, (batch, M, N + 3), torch.float32)
    api.gemm_batched(dA[:, :, :K], dB[:, :, :K], C[:, :, :N], alpha=2.0, beta=-3.0, num_iter=3)
    C0[:, :, :N] = 6.0 * oracle.gemm(np.ascontiguousarray(A[:, :, :K]), np.ascontiguousarray(B[:, :, :K])) \
        - 3.0 * C0[:, :, :N]
    assert np.array_equal(C.double().cpu().numpy(), C0)


def test_shared_operand(cuda):
    rng = np.random.default_rng(5)
    A, dA = _ints(rng, (1, 100, 40), torch.float16)
    B, dB = _ints(rng, (700, 16, 40), torch.float16)
    C = api.gemm_batched(dA.expand(700, 100, 40), dB)
    assert np.array_equal(C.double().cpu().numpy(), oracle.gemm(np.repeat(A, 700, 0), B))
