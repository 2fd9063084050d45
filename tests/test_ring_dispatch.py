"""Which uniform batches the library's own choice gives to the ring kernels, as
kami_gemm_describe reports it (host only), and the ring kernels' results at
odd sizes that take them (GPU): integer inputs against the oracle, exact."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from kami_b200 import _lib, api


def _describe(dtype, M, N, K, batch, variant=_lib.VARIANT_AUTO, partition=_lib.PARTITION_AUTO, P=0,
              b_layout=_lib.B_REF_NK):
    out = (ctypes.c_int * 8)()
    _lib.check(_lib.load().kami_gemm_describe(dtype, _lib.F64 if dtype == _lib.F64 else _lib.F32, partition, variant,
                                              M, N, K, P, 0, batch, _lib.A_ROW_MK, b_layout, out))
    return list(out)


RING = [(_lib.F16, 40, 40, 40, 100), (_lib.BF16, 100, 16, 40, 10), (_lib.F16, 20, 20, 128, 1600),
        (_lib.F16, 33, 128, 40, 1), (_lib.F16, 32, 64, 64, 300), (_lib.F64, 64, 64, 64, 5),
        (_lib.F64, 40, 24, 32, 1), (_lib.F64, 32, 32, 32, 2000)]
OTHER = [(_lib.F16, 128, 128, 128, 592), (_lib.F16, 16, 16, 16, 10 ** 6), (_lib.F16, 20, 20, 128, 900),
         (_lib.F16, 32, 64, 64, 296), (_lib.BF16, 8, 40, 40, 1),
         (_lib.F16, 33, 41, 128, 1500), (_lib.F64, 16, 16, 16, 10 ** 5), (_lib.F64, 32, 32, 32, 1000)]


@pytest.mark.parametrize("request_", RING)
def test_ring_is_described(request_):
    dtype, M, N, K, batch = request_
    d = _describe(dtype, M, N, K, batch)
    assert d[7] == 1 and d[0] == (_lib.VARIANT_MMA_SYNC if dtype == _lib.F64 else _lib.VARIANT_TCGEN05)
    assert d[3] == (640 if dtype == _lib.F64 else 896) and 200 * 1024 < d[4] <= 227 * 1024
    assert 1 <= d[6] <= 148 or d[6] <= batch  # CTAs: one per SM at most
    assert d[5] * d[6] >= batch
    # asked for by name or layout, the block kernels
    assert _describe(dtype, M, N, K, batch, b_layout=_lib.B_ROW_KN)[7] == 0
    if dtype == _lib.F64:
        assert _describe(dtype, M, N, K, batch, variant=_lib.VARIANT_MMA_SYNC)[7] == 0


@pytest.mark.parametrize("request_", OTHER)
def test_others_are_described(request_):
    assert _describe(*request_)[7] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,batch,pad,alpha,beta", [
    (20, 20, 128, 1700, 0, 1.0, 0.0), (31, 33, 72, 2000, 0, 1.0, 0.0), (31, 33, 72, 2000, 8, 2.0, -3.0),
    (120, 31, 40, 1500, 8, 2.0, -3.0), (32, 127, 128, 700, 8, -1.0, 1.0)])
@pytest.mark.parametrize("out", [torch.float32, torch.float16])
def test_odd_sizes_on_the_ring(cuda, M, N, K, batch, pad, alpha, beta, out):
    if out == torch.float16:
        batch *= 2  # the rule counts bytes
    d = (ctypes.c_int * 8)()
    _lib.check(_lib.load().kami_gemm_describe(_lib.F16, api._DT[out], 0, 0, M, N, K, 0, 0, batch, _lib.A_ROW_MK,
                                              _lib.B_REF_NK, d))
    assert d[7] == 1
    rng = np.random.default_rng(M + N)
    A = rng.integers(-3, 4, (batch, M, K + pad)).astype(np.float64)
    B = rng.integers(-3, 4, (batch, N, K + pad)).astype(np.float64)
    C0 = rng.integers(-3, 4, (batch, M, N + pad)).astype(np.float64)
    dA, dB = (torch.tensor(x, dtype=torch.float16, device="cuda") for x in (A, B))
    if pad:  # what lies between the rows must not matter
        dA[:, :, K:] = float("nan")
        dB[:, :, K:] = float("inf")
    C = torch.tensor(C0, dtype=out, device="cuda")
    api.gemm_batched(dA[:, :, :K], dB[:, :, :K], C[:, :, :N], alpha=alpha, beta=beta)
    C0[:, :, :N] = alpha * oracle.gemm(np.ascontiguousarray(A[:, :, :K]), np.ascontiguousarray(B[:, :, :K])) \
        + beta * C0[:, :, :N]
    assert torch.equal(C.cpu(), torch.tensor(C0, dtype=torch.float32).to(out))
