"""16-bit plans whose bytes lie mostly in large problems (two groups of warps per
CTA with larger rings) and just not (four): one problem, fewer than the lists and
many per list, sizes on both sides of the line in one plan.  Integer inputs
against the oracle, exact."""
import numpy as np
import pytest
import torch

import oracle
from kami_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [(1, 0), (200, 0), (1500, 300), (300, 3000), (40, 700)])
@pytest.mark.parametrize("dtype,out", [(torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_plan(cuda, large, small, dtype, out):
    rng = np.random.default_rng(large + small)
    big = np.stack([rng.integers(90, 129, large), rng.integers(96, 129, large), 8 * rng.integers(1, 17, large)], 1)
    few = np.stack([rng.integers(1, 60, small), rng.integers(1, 60, small), 8 * rng.integers(1, 17, small)], 1)
    shapes = rng.permutation(np.concatenate([big, few]))
    plan = api.GroupedPlan(shapes, dtype, out, kernel="tcgen05")
    A = rng.integers(-2, 3, plan.sizes[0]).astype(np.float64)
    B = rng.integers(-2, 3, plan.sizes[1]).astype(np.float64)
    C = torch.full((plan.sizes[2],), float("nan"), dtype=out, device="cuda")
    dA, dB = (torch.tensor(x, dtype=dtype, device="cuda") for x in (A, B))
    plan.run(dA, dB, C)
    got, (ao, bo, co) = C.double().cpu().numpy(), plan.offsets
    for (M, N, K), a, b, c in zip(shapes.tolist(), ao, bo, co):
        want = oracle.gemm(A[a:a + M * K].reshape(1, M, K), B[b:b + N * K].reshape(1, N, K)).reshape(-1)
        want = torch.tensor(want, dtype=torch.float32).to(out).double().numpy()
        assert np.array_equal(got[c:c + M * N], want)
