"""kami_spgemm_bsr_fill_numeric with nnz_c below the number of C tiles: the
columns and tiles below the bound are those of the whole product, what lies at
or past it is untouched -- for bounds that cut a row, cut between rows and
leave one tile, rows that fit the staging capacities and those that do not,
four and eight warps, the separate column fill, and the kernels by name."""
import ctypes

import numpy as np
import pytest
import torch

from kami_b200 import _lib, api

pytestmark = pytest.mark.gpu


def _bsr(rng, rows, cols, per):
    cnt = np.minimum(rng.integers(0, 2 * per + 1, rows), cols)
    cnt[0] = per
    ci = np.concatenate([np.sort(rng.choice(cols, c, replace=False)) for c in cnt]).astype(np.int32)
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(cnt, out=rp[1:])
    v = torch.tensor(rng.integers(-3, 4, (len(ci), 16, 16)), dtype=torch.float16, device="cuda")
    return api.BSR(torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda(), v, cols)


@pytest.mark.parametrize("rows,inner,cols,a,b", [
    (40, 30, 70, 4, 5),        # eight warps
    (1200, 20, 33, 2, 3),      # four warps
    (6, 70, 64, 50, 4),        # more A entries than are staged
    (3, 8, 2000, 6, 600),      # more C tiles
    (12, 10, 16385, 4, 9),     # columns by a launch of their own
])
@pytest.mark.parametrize("variant", [_lib.VARIANT_AUTO, _lib.VARIANT_MMA_SYNC, _lib.VARIANT_TCGEN05])
def test_bound(cuda, rows, inner, cols, a, b, variant):
    rng = np.random.default_rng(rows)
    A, B = _bsr(rng, rows, inner, a), _bsr(rng, inner, cols, b)
    rpc, total = api.spgemm_symbolic(A, B)
    cic = api.spgemm_fill_colidx(A, B, rpc, total)
    want = api.spgemm_numeric(A, B, rpc, cic)
    rp = rpc.cpu().numpy()
    mid = int(np.argmax(np.diff(rp)))
    for bound in {1, int(rp[mid]), int(rp[mid] + rp[mid + 1]) // 2, total - 1} - {0}:
        got_c = torch.full((total + 64,), -7, dtype=torch.int32, device="cuda")
        got_v = torch.full((total + 2, 16, 16), -7.0, device="cuda")
        st = _lib.load().kami_spgemm_bsr_fill_numeric(
            variant, _lib.F16, _lib.F32, 16, rows, inner, cols, A.row_ptr.data_ptr(), A.col_idx.data_ptr(),
            A.values.data_ptr(), B.row_ptr.data_ptr(), B.col_idx.data_ptr(), B.values.data_ptr(), rpc.data_ptr(),
            got_c.data_ptr(), got_v.data_ptr(), bound, 1.0, 0.0, 1, ctypes.c_void_p(api._stream_ptr(None)))
        _lib.check(st)
        assert torch.equal(got_c[:bound], cic[:bound]) and bool((got_c[bound:] == -7).all())
        assert torch.equal(got_v[:bound], want[:bound]) and bool((got_v[bound:] == -7).all())
