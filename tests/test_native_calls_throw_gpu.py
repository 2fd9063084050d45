"""A C++ exception out of the library's entry point: the C++ form of a call holds
the interpreter lock again and leaves the call to the Python code."""
import ctypes
import shutil
import subprocess

import pytest
import torch

from kami_b200 import _lib, api

pytestmark = pytest.mark.gpu


def test_exception(cuda, tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    (tmp_path / "throws.cpp").write_text(
        "#include <new>\nstatic int n;\nextern \"C\" int calls() { return n; }\n"
        "extern \"C\" int throws() { ++n; throw std::bad_alloc(); }\n")
    so = tmp_path / "throws.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-o", str(so), str(tmp_path / "throws.cpp")], check=True)
    fake = ctypes.CDLL(str(so))
    calls, L = api._native(), _lib.load()

    def bind(gemm):
        calls.bind(*(ctypes.cast(f, ctypes.c_void_p).value for f in (
            gemm, L.kami_spmm_bsr, L.kami_spgemm_bsr_symbolic, L.kami_spgemm_bsr_fill_numeric)))
    A, B = torch.ones(3, 16, 32, device="cuda").half(), torch.ones(3, 24, 32, device="cuda").half()
    try:
        bind(fake.throws)
        C = api.gemm_batched(A, B)
    finally:
        bind(L.kami_gemm_batched)
    assert fake.calls() == 1 and ctypes.pythonapi.PyGILState_Check() == 1
    assert torch.equal(C, torch.full((3, 16, 24), 32.0, device="cuda"))
