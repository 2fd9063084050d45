"""The block-row SpGEMM kernel with and without the column fill, four and eight
warps per row: the row that fits the staging capacities and those that do not
(A entries, C tiles, products), columns at the ends of the bitmap's words, more
columns than the bitmap takes, and every output type.  Integer inputs against
the dense product in FP64: exact in FP32."""
import ctypes

import numpy as np
import pytest
import torch

from kami_b200 import _lib, api

pytestmark = pytest.mark.gpu


def _bsr(rng, rows, cols, pick, dtype):
    """rows x cols blocks; pick(row): the row's columns"""
    per = [np.unique(np.asarray(pick(r), dtype=np.int32)) for r in range(rows)]
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum([len(c) for c in per], out=rp[1:])
    ci = np.concatenate(per).astype(np.int32)
    v = rng.integers(-3, 4, (len(ci), 16, 16)).astype(np.float64)
    m = api.BSR(torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda(), torch.tensor(v, dtype=dtype, device="cuda"), cols)
    return m, rp, ci, v


def _product(rows, A, B):
    """row pointers, columns and tiles of A * B"""
    (_, rpa, cia, va), (_, rpb, cib, vb) = A, B
    rp, ci, tiles = [0], [], []
    for i in range(rows):
        acc = {}
        for e in range(rpa[i], rpa[i + 1]):
            for b in range(rpb[cia[e]], rpb[cia[e] + 1]):
                acc[cib[b]] = acc.get(cib[b], 0.0) + va[e] @ vb[b]
        ci += sorted(acc)
        tiles += [acc[c] for c in sorted(acc)]
        rp.append(len(ci))
    return np.array(rp), np.array(ci, dtype=np.int64), np.array(tiles).reshape(-1, 16, 16)


CASES = {  # block-rows, inner, block columns, entries of A's and B's rows
    "few": (40, 30, 70, 4, 5), "many rows": (1200, 20, 33, 2, 3), "one column": (9, 9, 1, 3, 1),
    "A entries": (6, 40, 64, 30, 4), "C tiles": (3, 8, 1100, 6, 200), "products": (5, 24, 100, 20, 60),
    "bitmap full": (12, 10, 16384, 4, 9), "past the bitmap": (12, 10, 16385, 4, 9), "empty rows": (700, 50, 60, 0, 3),
    "32 A entries": (6, 32, 64, 400, 4), "more A entries": (6, 70, 64, 90, 4), "more C tiles": (3, 8, 2000, 6, 400),
    "a few long rows": (1200, 90, 60, -1, 4), "long rows": (1200, 40, 200, 9, 30),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("dtype,out", [(torch.float16, torch.float32), (torch.bfloat16, torch.float32),
                                       (torch.float16, torch.float16)])
def test_fill_and_numeric(cuda, name, dtype, out):
    rows, inner, cols, na, nb = CASES[name]
    rng = np.random.default_rng(len(name))
    A = _bsr(rng, rows, inner, lambda r: rng.integers(0, inner, na if na > 0 else (r % 4 == 0) * 3 if na == 0 else 1 + (r % 50 == 0) * 60), dtype)
    ends = [0, 31, 32, 63, cols - 1]
    B = _bsr(rng, inner, cols, lambda r: [c for c in ends[:1 + r % 5] if c < cols] + list(rng.integers(0, cols, nb)), dtype)
    rp, ci, tiles = _product(rows, A, B)
    want = torch.tensor(tiles, dtype=torch.float32).to(out)
    got = api.spgemm(A[0], B[0], out)
    assert np.array_equal(got.row_ptr.cpu().numpy(), rp) and np.array_equal(got.col_idx.cpu().numpy(), ci)
    assert torch.equal(got.values.cpu(), want)
    # without the fill: the numeric pass alone, twice into the same tiles with alpha and beta
    C = api.spgemm_numeric(A[0], B[0], got.row_ptr, got.col_idx, torch.float32)
    assert torch.equal(C.cpu().double(), torch.from_numpy(tiles))
    api.spgemm_numeric(A[0], B[0], got.row_ptr, got.col_idx, torch.float32, C, alpha=2.0, beta=-1.0, num_iter=2)
    assert torch.equal(C.cpu().double(), torch.from_numpy(3 * tiles))
    # the call that does both, for the kernel chosen by name as well
    for variant in (_lib.VARIANT_AUTO, _lib.VARIANT_MMA_SYNC, _lib.VARIANT_TCGEN05):
        cic = torch.full_like(got.col_idx, -1)
        C2 = torch.empty_like(got.values)
        st = _lib.load().kami_spgemm_bsr_fill_numeric(
            variant, api._DT[dtype], api._DT[out], 16, rows, inner, cols, A[0].row_ptr.data_ptr(), A[0].col_idx.data_ptr(),
            A[0].values.data_ptr(), B[0].row_ptr.data_ptr(), B[0].col_idx.data_ptr(), B[0].values.data_ptr(),
            got.row_ptr.data_ptr(), cic.data_ptr(), C2.data_ptr(), cic.numel(), 1.0, 0.0, 1,
            ctypes.c_void_p(api._stream_ptr(None)))
        _lib.check(st)
        assert torch.equal(cic, got.col_idx) and torch.equal(C2.cpu(), want)


def test_more_columns_than_products(cuda):
    """A wider structure of C than the products need: those tiles are zeros."""
    rng = np.random.default_rng(3)
    A = _bsr(rng, 30, 20, lambda r: rng.integers(0, 20, 3), torch.float16)
    B = _bsr(rng, 20, 40, lambda r: rng.integers(0, 40, 3), torch.float16)
    rp, ci, tiles = _product(30, A, B)
    wide = torch.arange(0, 31 * 40, 40, dtype=torch.int32, device="cuda")
    cols = torch.arange(40, dtype=torch.int32, device="cuda").repeat(30)
    C = torch.full((1200, 16, 16), float("nan"), device="cuda")
    api.spgemm_numeric(A[0], B[0], wide, cols, torch.float32, C)
    want = np.zeros((1200, 16, 16))
    for i in range(30):
        want[i * 40 + ci[rp[i]:rp[i + 1]]] = tiles[rp[i]:rp[i + 1]]
    assert np.array_equal(C.cpu().double().numpy(), want)
