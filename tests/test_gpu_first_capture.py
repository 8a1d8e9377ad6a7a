"""The process's first call of the library that allocates, made under a stream
capture: the 2-D PyTorch operator, whose scratch then belongs to the graph."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
import sspmv_gb300.torch_ops
n, per, k = 5000, 7, 3
rp = torch.arange(n + 1, dtype=torch.int32, device="cuda") * per
col = torch.randint(n, (n * per,), dtype=torch.int32, device="cuda")
val = torch.rand(n * per, dtype=torch.float64, device="cuda")
x = torch.rand(n, k, dtype=torch.float64, device="cuda")
want = torch.zeros(n, k, dtype=torch.float64, device="cuda")
want.index_add_(0, torch.arange(n, device="cuda").repeat_interleave(per), val.unsqueeze(1) * x[col.long()])
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = torch.ops.sspmv.spmv_csr(rp, col, val, n, x)
for _ in range(3):
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert (y - want).abs().max() < 1e-13
assert torch.equal(torch.ops.sspmv.spmv_csr(rp, col, val, n, x), y)  # and outside a capture
torch.cuda.synchronize()
print("ok")
"""


def test_first_allocation_under_capture():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
