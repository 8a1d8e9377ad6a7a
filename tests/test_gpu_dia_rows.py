"""DIA with as many rows as its strided grid covers and more.  Against the FP64
oracle with the per-row bound of the parity tests."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu


def _check(A, M, dt, oracle_lib, products=((1.0, 0.0), (0.8, 0.7), (0.8, 0.0))):
    from sspmv_gb300 import lespmv as L
    rng = np.random.default_rng(1)
    for alpha, beta in products:
        x = rng.uniform(-1, 1, A.num_cols).astype(dt)
        y0 = rng.uniform(-1, 1, A.num_rows).astype(dt)
        y = to_dev(y0)
        L.LeSpMV(alpha, M, to_dev(x), beta, y)
        y64, absum = oracle_lib.spmm_ref(A, x, alpha, beta, y0)
        ok, mx, _ = tolerance_ok(to_host(y), y64, absum, np.diff(A.row_offset), dt, alpha, beta, y0)
        assert ok, f"alpha={alpha} beta={beta}: max normalised error {mx}"


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("m", [622_592, 622_593, 700_001])
def test_dia_many_rows(m, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300 import synth
    A = synth.generate(synth.banded(m), 2, dt)
    _check(A, L.csr_to_dia(L.csr_from_host(A)), dt, oracle_lib)
