"""The library's memory pool: freed blocks are kept for the next matrix up to
the pool's bound, and everything goes back to the device with the last one."""
import pytest

pytestmark = pytest.mark.gpu


PROGRAM = """
import numpy as np, torch
from sspmv_gb300 import lespmv as L, synth
A = synth.generate(synth.banded(1 << 20), 1, np.float64)
x = torch.ones(A.num_cols, dtype=torch.float64, device="cuda")
y = torch.empty(A.num_rows, dtype=torch.float64, device="cuda")
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
def use(M):
    for convert in (L.csr_to_sell_c_sigma, L.csr_to_csr5, L.csr_to_dia, L.csr_to_ell):
        B = convert(M)
        L.LeSpMV(1.0, B, x, 0.0, y)
        B.delete()
M = L.csr_from_host(A)
use(M)                      # modules loaded
M.delete()
start = free()
M = L.csr_from_host(A)
own = start - free()
use(M)
kept = start - free() - own
assert kept <= 1 << 30, kept
M.delete()
assert start - free() <= 0, start - free()
print("ok", own >> 20, kept >> 20)
"""


def test_pool_gives_memory_back_with_the_last_matrix():
    """In a process of its own (no other live matrices): what is kept beside a
    live matrix is bounded, and nothing stays mapped after the last one."""
    import subprocess
    import sys
    from pathlib import Path
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
