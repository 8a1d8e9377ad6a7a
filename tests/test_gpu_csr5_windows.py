"""The CSR5 kernel at the edges of its windows: tile shapes (sigma a multiple
of 8 and not, every omega), matrices of one tile, of full tiles only and with a
short last tile, rows over many windows, runs of empty rows."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu

LENS = {"one": [1], "one_tile": [3, 0, 17], "full_tiles": [32] * 512, "long": [5, 40_000, 0, 3, 9000, 1],
        "short": [1, 2, 3, 0] * 3000, "ragged": list(np.random.default_rng(4).integers(0, 60, 2777))}


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", [(16, 4), (16, 8), (16, 32), (32, 16), (32, 32), (8, 32), (12, 8), (5, 16), (40, 4)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("case", list(LENS))
def test_csr5_windows(case, shape, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(7)
    rp = np.concatenate([[0], np.cumsum(LENS[case])]).astype(np.int32)
    A = HostCSR(len(LENS[case]), 901, rp, rng.integers(0, 901, rp[-1]).astype(np.int32),
                rng.uniform(-1, 1, rp[-1]).astype(dt))
    M = L.csr_to_csr5(L.csr_from_host(A), *shape)
    for k, alpha, beta in [(1, 1.0, 0.0), (1, 0.8, 0.7), (4, 0.8, 0.7), (8, 1.0, 0.0)]:
        X = rng.uniform(-1, 1, (901, k)).astype(dt)
        Y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
        Y = to_dev(Y0)
        L.spmm(alpha, M, to_dev(X), beta, Y)
        y64, absum = oracle_lib.spmm_ref(A, X, alpha, beta, Y0)
        y64, absum = y64.reshape(-1, k), absum.reshape(-1, k)
        ok, mx, _ = tolerance_ok(to_host(Y), y64, absum, np.diff(rp), dt, alpha, beta, Y0)
        assert ok, f"{case} {shape} k={k}: max normalised error {mx}"
