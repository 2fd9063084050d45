"""api.gemm_batched, api.spmm and api.spgemm through the C++ module and through
the Python code: the same results, the same returned object, the same errors,
for every form that the two could take differently."""
import numpy as np
import pytest
import torch

from kami_b200 import api

pytestmark = pytest.mark.gpu

F16 = torch.float16


def _both(monkeypatch, f):
    """f()'s outcome through the C++ module, then through Python alone."""
    out = []
    assert api._native()
    for calls in (api._calls, False):
        with monkeypatch.context() as m:
            m.setattr(api, "_calls", calls)
            try:
                out.append(f())
            except Exception as e:
                out.append((type(e), str(e)))
    return out


def _t(seed, *shape, dtype=F16):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(-3, 4, shape, generator=g).to(dtype).cuda()


GEMM = {
    "2-D": lambda: api.gemm_batched(_t(1, 16, 32), _t(2, 24, 32)),
    "3-D": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32)),
    "layouts": lambda: api.gemm_batched(_t(1, 5, 32, 16), _t(2, 5, 32, 24), a_layout="col_mk", b_layout="row_kn"),
    "out": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32), out_dtype=F16, alpha=2, num_iter=3),
    "strided": lambda: api.gemm_batched(_t(1, 5, 16, 64)[:, :, 8:40], _t(2, 9, 24, 32)[::2], alpha=0.5),
    "shared": lambda: api.gemm_batched(_t(1, 1, 16, 32).expand(5, 16, 32), _t(2, 5, 24, 32)),
    "one row": lambda: api.gemm_batched(_t(1, 5, 1, 32), _t(2, 5, 1, 32)),
    "f64": lambda: api.gemm_batched(_t(1, 5, 16, 32, dtype=torch.float64), _t(2, 5, 24, 32, dtype=torch.float64)),
    "no problems": lambda: api.gemm_batched(_t(1, 0, 16, 32), _t(2, 0, 24, 32)),
    "requires grad": lambda: api.gemm_batched(_t(1, 5, 16, 32).requires_grad_(), _t(2, 5, 24, 32)),
    "types differ": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32, dtype=torch.bfloat16)),
    "no such type": lambda: api.gemm_batched(_t(1, 5, 16, 32, dtype=torch.int32), _t(2, 5, 24, 32, dtype=torch.int32)),
    "on the CPU": lambda: api.gemm_batched(_t(1, 5, 16, 32).cpu(), _t(2, 5, 24, 32)),
    "inner stride": lambda: api.gemm_batched(_t(1, 5, 32, 16).mT, _t(2, 5, 24, 32)),
    "no such layout": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32), b_layout="kn"),
    "refused": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32), num_iter=0),
    "refused type": lambda: api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32), out_dtype=torch.float64),
}


@pytest.mark.parametrize("form", GEMM)
def test_gemm(cuda, monkeypatch, form):
    a, b = _both(monkeypatch, GEMM[form])
    if isinstance(b, tuple):
        assert a == b
    else:
        assert a.dtype == b.dtype and a.shape == b.shape and a.requires_grad == b.requires_grad and torch.equal(a, b)


def test_gemm_into(cuda, monkeypatch):
    def f():
        C = _t(3, 5, 16, 40, dtype=torch.float32)
        view = C[:, :, 4:28]
        assert api.gemm_batched(_t(1, 5, 16, 32), _t(2, 5, 24, 32), view, beta=2.0) is view
        return C
    a, b = _both(monkeypatch, f)
    assert torch.equal(a, b)


def _bsr(seed, rows, cols, density, dtype=F16):
    rng = np.random.default_rng(seed)
    r, c = np.nonzero(rng.random((rows, cols)) < density)
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=rows), out=rp[1:])
    return api.BSR(torch.from_numpy(rp).cuda(), torch.from_numpy(c.astype(np.int32)).cuda(),
                   _t(seed, len(c), 16, 16, dtype=dtype), cols)


@pytest.mark.parametrize("rows,inner,cols,density", [(9, 7, 11, 0.4), (3, 2, 1, 1.0), (5, 4, 6, 0.0), (0, 4, 6, 0.5)])
def test_spgemm(cuda, monkeypatch, rows, inner, cols, density):
    A, B = _bsr(1, rows, inner, density), _bsr(2, inner, cols, density)
    a, b = _both(monkeypatch, lambda: api.spgemm(A, B))
    for x, y in ((a.row_ptr, b.row_ptr), (a.col_idx, b.col_idx), (a.values, b.values)):
        assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x, y)
    assert (a.block_rows, a.block_cols) == (b.block_rows, b.block_cols)


@pytest.mark.parametrize("form", ["inner", "type", "variant", "iter"])
def test_spgemm_errors(cuda, monkeypatch, form):
    A, B = _bsr(1, 4, 5, 0.5), _bsr(2, 6 if form == "inner" else 5, 4, 0.5)
    f = {"inner": lambda: api.spgemm(A, B), "type": lambda: api.spgemm(A, B, torch.int32),
         "variant": lambda: api.spgemm(A, B, variant="x"), "iter": lambda: api.spgemm(A, B, num_iter=0)}[form]
    a, b = _both(monkeypatch, f)
    assert isinstance(b, tuple) and a == b


@pytest.mark.parametrize("layout", ["row_kn", "ref_nk"])
@pytest.mark.parametrize("n", [1, 24])
def test_spmm(cuda, monkeypatch, layout, n):
    A = _bsr(1, 6, 5, 0.5)
    B = _t(2, 80, n) if layout == "row_kn" else _t(2, n, 80)
    a, b = _both(monkeypatch, lambda: api.spmm(A, B, b_layout=layout, alpha=2.0))
    assert a.dtype == b.dtype and torch.equal(a, b)
    C = _t(3, 96, n, dtype=torch.float32)
    assert api.spmm(A, B, C, b_layout=layout, beta=1.0) is C
    for bad in (lambda: api.spmm(A, B[:-1], b_layout="row_kn"), lambda: api.spmm(A, B.cpu(), b_layout=layout)):
        a, b = _both(monkeypatch, bad)
        assert isinstance(b, tuple) and a == b
