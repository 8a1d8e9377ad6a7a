"""CSR5 with tiles larger than the matrix (a single tile, in CSR order) and with
long columns: sigma up to the format's limit, where 32 sigma passes the 32-bit
range."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", [(1000, 4), (4096, 8), (13_421_773, 4), (1 << 26, 4), (1 << 27, 4), (1 << 30, 1)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_csr5_large_sigma(shape, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(11)
    lens = np.concatenate([[0, 20_000, 0], rng.integers(0, 40, 2000), [5000, 1, 0]])
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    A = HostCSR(len(lens), 701, rp, rng.integers(0, 701, rp[-1]).astype(np.int32),
                rng.uniform(-1, 1, rp[-1]).astype(dt))
    M = L.csr_to_csr5(L.csr_from_host(A), *shape)
    for k, alpha, beta in [(1, 1.0, 0.0), (1, 0.8, 0.7), (5, 0.8, 0.7), (8, 1.0, 0.0)]:
        X = rng.uniform(-1, 1, (701, k)).astype(dt)
        Y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
        Y = to_dev(Y0)
        L.spmm(alpha, M, to_dev(X), beta, Y)
        y64, absum = oracle_lib.spmm_ref(A, X, alpha, beta, Y0)
        y64, absum = y64.reshape(-1, k), absum.reshape(-1, k)
        ok, mx, _ = tolerance_ok(to_host(Y), y64, absum, lens, dt, alpha, beta, Y0)
        assert ok, f"{shape} k={k}: max normalised error {mx}"
