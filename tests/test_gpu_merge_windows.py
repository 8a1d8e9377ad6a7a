"""The merge-path kernel at the edges of its windows: windows of row ends only,
of nonzeros only, rows that end on a window's last item, runs of empty rows,
one item, unaligned arrays, every K."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu

LENS = {"one": [1], "one_empty": [0], "empty": [0] * 3000, "edge": [503] * 40, "past": [504, 0] * 40,
        "gaps": ([0] * 1100 + [9, 700]) * 6, "long": [5, 40_000, 0, 3, 9000, 1], "short": [1, 2, 3, 0] * 3000,
        "ragged": list(np.random.default_rng(4).integers(0, 60, 2777))}


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("case", list(LENS))
def test_merge_windows(case, dt, oracle_lib):
    import sspmv_gb300.torch_ops  # noqa: F401  (registers the operator)
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(7)
    rp = np.concatenate([[0], np.cumsum(LENS[case])]).astype(np.int32)
    A = HostCSR(len(LENS[case]), 901, rp, rng.integers(0, 901, rp[-1]).astype(np.int32),
                rng.uniform(-1, 1, rp[-1]).astype(dt))
    M = L.csr_from_host(A)
    M.set_kernel(2, 0)
    X = rng.uniform(-1, 1, (901, 8)).astype(dt)
    Y0 = rng.uniform(-1, 1, (A.num_rows, 8)).astype(dt)
    for k, alpha, beta in [(1, 1.0, 0.0), (1, 0.8, 0.7), (2, 1.0, 0.0), (4, 0.8, 0.7), (7, 0.8, 0.7), (8, 1.0, 0.0)]:
        x, y0 = np.ascontiguousarray(X[:, :k]), np.ascontiguousarray(Y0[:, :k])
        Y = to_dev(y0)
        L.spmm(alpha, M, to_dev(x), beta, Y)
        y64, absum = oracle_lib.spmm_ref(A, x, alpha, beta, y0)
        ok, mx, _ = tolerance_ok(to_host(Y), y64.reshape(-1, k), absum.reshape(-1, k), np.diff(rp), dt, alpha, beta, y0)
        assert ok, f"{case} k={k}: max normalised error {mx}"
    plain = torch.empty(A.num_rows, dtype=to_dev(X).dtype, device="cuda")
    L.LeSpMV(1.0, M, to_dev(np.ascontiguousarray(X[:, 0])), 0.0, plain)
    pad = [torch.cat([to_dev(v)[:1] if len(v) else to_dev(np.zeros(1, v.dtype)), to_dev(v)])[1:]
           for v in (A.col_index, A.values)]  # one element off 16-byte alignment
    y = torch.ops.sspmv.spmv_csr(to_dev(rp), *pad, 901, to_dev(np.ascontiguousarray(X[:, 0])))
    assert torch.equal(y, plain), case
