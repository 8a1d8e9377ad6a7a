"""The BSR block-stream kernel at the edges of its windows and loads: every
block shape it takes, matrices of one block, of steps that are exactly full,
runs of empty block rows, a ragged last block column and row, and an x
that is not aligned for vector loads."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu

LENS = {"one": [0, 1], "full": [4] * 1024, "gaps": ([0] * 70 + [9, 1, 30]) * 40, "long": [5, 4000, 0, 3, 900, 1],
        "ragged": list(np.random.default_rng(4).integers(0, 20, 2777))}


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", [(1, 1), (1, 2), (2, 1), (2, 2), (4, 4), (8, 8), (16, 16), (32, 4), (4, 8), (8, 1)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("case", list(LENS))
def test_bsr_stream_edges(case, shape, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(7)
    lens, n = np.minimum(LENS[case], 901), 901
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.permutation(n)[:l]) for l in lens]).astype(np.int32)
    A = HostCSR(len(lens), n, rp, ci, rng.uniform(-1, 1, rp[-1]).astype(dt))
    B = L.csr_to_bsr(L.csr_from_host(A), *shape)
    B.set_kernel(2, 0)
    for alpha, beta, shift in [(1.0, 0.0, 0), (0.8, 0.7, 0), (0.8, 0.7, 1)]:
        x = rng.uniform(-1, 1, n).astype(dt)
        y0 = rng.uniform(-1, 1, A.num_rows).astype(dt)
        xd = torch.zeros(n + shift, dtype=to_dev(x).dtype, device="cuda")[shift:]
        xd.copy_(to_dev(x))
        y = to_dev(y0)
        L.LeSpMV(alpha, B, xd, beta, y)
        y64, absum = oracle_lib.spmm_ref(A, x.reshape(-1, 1), alpha, beta, y0.reshape(-1, 1))
        ok, mx, _ = tolerance_ok(to_host(y).reshape(-1, 1), y64, absum, lens, dt, alpha, beta, y0.reshape(-1, 1))
        assert ok, f"{case} {shape} shift={shift}: max normalised error {mx}"
