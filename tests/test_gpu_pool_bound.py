"""What the library's memory pool keeps: no more than its bound beside the live
matrices, something even where these alone are larger than the bound, and
nothing once a request server that held all of them is gone.  Each in a process
of its own."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import ctypes as C
import numpy as np, torch
from sspmv_gb300 import _lib
from sspmv_gb300 import lespmv as L
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
GB = 1 << 30
def wrapped(n, per):
    keep = (torch.arange(n + 1, dtype=torch.int32, device="cuda") * per,
            torch.randint(n, (n * per,), dtype=torch.int32, device="cuda"),
            torch.rand(n * per, dtype=torch.float64, device="cuda"))
    s = _lib.Csr()
    _lib.call("sspmv_csr_wrap", C.byref(s), _lib.F64, n, n, n * per, *(C.c_void_p(t.data_ptr()) for t in keep))
    M = L.CSR_Matrix(s)
    M.keep = keep
    return M
"""

BOUND = HEAD + """
A = wrapped(1 << 20, 32)                       # 0.4 GB converted
B = wrapped(1 << 22, 40)                       # 2 GB converted
L.csr_to_sell_c_sigma(A).delete()              # modules loaded
start = free()
small = L.csr_to_sell_c_sigma(A)
own = start - free()
L.csr_to_sell_c_sigma(B).delete()
kept = start - free() - own
assert 0 < kept <= GB + (128 << 20), kept      # 2 GB freed beside 0.4 GB live
big = L.csr_to_sell_c_sigma(B)
L.csr_to_sell_c_sigma(A).delete()
kept = start - free() - own
assert start - free() > 2.2 * GB, start - free()   # 2.4 GB live and what is kept beside it
big.delete()
kept = start - free() - own
assert kept <= GB + (128 << 20), kept
small.delete()
assert start - free() <= 0, start - free()
print("ok")
"""

KEEPS = HEAD + """
A = wrapped(1 << 20, 32)
B = wrapped(1 << 22, 40)
L.csr_to_sell_c_sigma(A).delete()
big = L.csr_to_sell_c_sigma(B)                 # 2 GB live: more than is kept
before = free()
L.csr_to_sell_c_sigma(A).delete()
assert before - free() > 300 << 20, before - free()
print("ok")
"""

SERVER = HEAD + """
from sspmv_gb300 import synth
from sspmv_gb300.serving import Server
A = synth.generate(synth.banded(1 << 20), 1, np.float64)
x, y = np.ones(A.num_cols), np.empty(A.num_rows)
def serve():
    with Server() as s:
        s.add_matrix(0, A)
        s.add_matrix(1, A, "sell_c_sigma")
        for m in (0, 1):
            assert s.wait(s.submit(m, x, y), 60.0)["status"] == 0
serve()                                        # modules loaded
start = free()
serve()
assert start - free() <= 0, start - free()
M = L.csr_from_host(A)
M.delete()
assert start - free() <= 0, start - free()
print("ok")
"""


@pytest.mark.parametrize("program", [BOUND, KEEPS, SERVER], ids=["bound", "keeps", "server"])
def test_pool(program):
    r = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
