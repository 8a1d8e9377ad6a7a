"""The bytes that the request server counts against its budget are those that the
matrices and their plans hold: for every format, once its first product has
built the plan, within a tenth of what the device has lost; and the budget holds
when plans are counted."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
from sspmv_gb300 import synth
from sspmv_gb300.serving import Server
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
A = synth.generate(synth.powerlaw(3_000_000, 1.8, 16.0, 30_000, 0.05), 3, np.float64)
x = torch.ones(A.num_cols, dtype=torch.float64, device="cuda")
y = torch.ones(A.num_rows, dtype=torch.float64, device="cuda")
def serve(s, m):
    assert s.wait(s.submit(m, x, y, device=True), 120.0)["status"] == 0
for fmt, params in [("csr", None), ("coo", None), ("csr5", None), ("sell_c_sigma", (4096, 32, 0)), ("sell_c_R", (32, 1)),
                    ("bsr", (1, 4))]:
    with Server(arena_bytes=1 << 20) as s:
        s.add_matrix(1, synth.generate(synth.banded(1000), 1, np.float64), fmt, params)
        serve_small = s.wait(s.submit(1, x, y, device=True), 120.0)   # kernels loaded
        before, counted0 = free(), s.stats()["resident_bytes"]
        s.add_matrix(0, A, fmt, params)
        serve(s, 0)
        counted = s.stats()["resident_bytes"] - counted0
        held = before - free()
    # the pool keeps up to 1 GiB of conversion scratch beside the matrix
    assert counted <= held * 1.02 + (64 << 20), (fmt, counted, held)
    assert counted >= held - (1 << 30) - (192 << 20), (fmt, counted, held)
    assert counted >= A.nnz * 12 * (1.05 if fmt != "bsr" else 1.0), (fmt, counted / A.nnz)
    print(fmt, counted >> 20, held >> 20)
print("ok")
"""


def test_counted_bytes_match_held_bytes():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=600,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout.rstrip().endswith("ok"), r.stdout + r.stderr
    print(r.stdout)


def test_budget_holds_with_plans():
    """Sliced matrices whose plans copy their long rows: what is resident stays
    within the budget after each first product, by evicting idle ones."""
    import numpy as np
    from sspmv_gb300 import synth
    from sspmv_gb300.serving import Server
    mats = [synth.generate(synth.powerlaw(60_000, 1.8, 16.0, 20_000), 3 + i, np.float64) for i in range(6)]
    need = 3 * (mats[0].nnz * 12 + 60_001 * 4)
    with Server(hbm_budget_bytes=2 * need) as s:
        for i, A in enumerate(mats):
            s.add_matrix(i, A, "sell_c_sigma", (4096, 8, 0))
        for i in [0, 1, 2, 3, 4, 5, 0, 1, 2, 3]:
            x, y = np.ones(60_000), np.empty(60_000)
            assert s.wait(s.submit(i, x, y), 60.0)["status"] == 0
            st = s.stats()
            assert st["resident_bytes"] <= 2 * need, st
            assert np.allclose(y, np.add.reduceat(np.append(mats[i].values, 0.0), mats[i].row_offset[:-1])
                               * (np.diff(mats[i].row_offset) > 0), rtol=1e-9, atol=1e-9)
