"""Matrices of 2^31 - 1 nonzeros, the most that 32-bit indices take, and of 128
fewer, the most that the vector kernel takes: every kernel's element index ends
within a step of the type's largest value.  Ones times ones, so that a row's sum
is its length exactly."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

NNZ, ROW = 2**31 - 1, 32768


@pytest.fixture(scope="module")
def arrays():
    import torch
    m = -(-NNZ // ROW)
    rp = torch.arange(m + 1, dtype=torch.int64, device="cuda").mul_(ROW).clamp_(max=NNZ).to(torch.int32)
    yield rp, torch.zeros(NNZ, dtype=torch.int32, device="cuda"), torch.ones(NNZ, device="cuda")


@pytest.mark.parametrize("nnz", [NNZ, NNZ - 128])
@pytest.mark.parametrize("k", [1, 8])
@pytest.mark.parametrize("flag", [0, 1, 2], ids=["stream", "vector", "merge"])
def test_csr_of_int_max_nonzeros(arrays, flag, k, nnz):
    import torch
    from sspmv_gb300 import _lib
    from sspmv_gb300 import lespmv as L
    rp, col, val = arrays
    rp = rp.clamp(max=nnz)
    m = rp.numel() - 1
    s = _lib.Csr()
    _lib.call("sspmv_csr_wrap", C.byref(s), _lib.F32, m, 1, nnz, *(C.c_void_p(t.data_ptr()) for t in (rp, col, val)))
    A = L.CSR_Matrix(s)
    A.set_kernel(flag, 0)
    y = torch.zeros((m, k), device="cuda")
    L.spmm(1.0, A, torch.ones((1, k), device="cuda"), 0.0, y)
    want = (rp[1:].long() - rp[:-1].long()).float().unsqueeze(1).expand(m, k)
    assert torch.equal(y, want)
    A.delete()
