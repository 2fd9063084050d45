"""C of the 16-bit ring kernel that does not leave in whole aligned rows: one
column and more than a patch of 32, odd and even widths and row strides, C on a
boundary of 4, 8 and 16 bytes and on none, every output type, with and without
alpha and beta, NaN in a C that is not read.  Integer inputs against the
oracle, exact; what lies around C stays as it was."""
import numpy as np
import pytest
import torch

import oracle
from kami_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 40), (24, 33), (32, 1), (96, 24), (120, 31), (31, 104), (16, 127), (40, 48), (64, 56)])
@pytest.mark.parametrize("shift,extra", [(0, 0), (1, 0), (0, 1), (2, 2), (4, 4), (3, 5)])
@pytest.mark.parametrize("out", [torch.float32, torch.float16, torch.bfloat16])
def test_stores(cuda, M, N, shift, extra, out):
    K, ldc = 40, N + extra
    batch = 16_100_000 // ((M + N) * K * 2 + M * N * (4 if out == torch.float32 else 2)) + 1  # past the rule's 16 MB
    rng = np.random.default_rng(M + N + shift)
    A = rng.integers(-2, 3, (batch, M, K)).astype(np.float64)
    B = rng.integers(-2, 3, (batch, N, K)).astype(np.float64)
    AB = torch.from_numpy(oracle.gemm(A, B)).cuda()
    dA, dB = (torch.tensor(x, dtype=torch.float16, device="cuda") for x in (A, B))
    room = batch * M * ldc + shift + 8
    for alpha, beta in ((1.0, 0.0), (2.0, -3.0), (-1.0, 0.0)):
        flat = torch.randint(-3, 4, (room,), device="cuda").to(out)
        if beta == 0.0:
            flat[shift:].fill_(float("nan"))
        C = flat[shift:shift + batch * M * ldc].view(batch, M, ldc)[:, :, :N]
        want = flat.clone()
        w = want[shift:shift + batch * M * ldc].view(batch, M, ldc)[:, :, :N]
        w.copy_((alpha * AB + (beta * w.double() if beta else 0.0)).float().to(out))
        api.gemm_batched(dA, dB, C, alpha=alpha, beta=beta)
        assert torch.equal(torch.nan_to_num(flat, nan=77.0), torch.nan_to_num(want, nan=77.0))
