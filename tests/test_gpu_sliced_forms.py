"""The forms of the sliced formats' thread pass and the rules that choose one:
every width up to 13 and wider ones, with and without padding, even and uneven
rows, grids around a whole number of waves, more rows than a strided grid
covers.  Against the FP64 oracle with the per-row bound of the parity tests."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu


def _matrix(lens, n, dt, seed=5):
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    nnz = int(rp[-1])
    return HostCSR(len(lens), n, rp, rng.integers(0, n, nnz).astype(np.int32), rng.uniform(-1, 1, nnz).astype(dt))


def _convert(A, fmt, align):
    from sspmv_gb300 import lespmv as L
    M = L.csr_from_host(A)
    if fmt == "ell":
        return L.csr_to_ell(M)
    if fmt == "sell_c_sigma":
        return L.csr_to_sell_c_sigma(M, 256, 32, align)
    return getattr(L, "csr_to_" + fmt)(M, 32, align)


def _check(A, M, dt, products, oracle_lib):
    from sspmv_gb300 import lespmv as L
    rng = np.random.default_rng(1)
    for k, alpha, beta in products:
        X = rng.uniform(-1, 1, (A.num_cols, k)).astype(dt)
        Y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
        Y = to_dev(Y0)
        L.spmm(alpha, M, to_dev(X), beta, Y)
        y64, absum = oracle_lib.spmm_ref(A, X, alpha, beta, Y0)
        ok, mx, _ = tolerance_ok(to_host(Y), y64.reshape(-1, k), absum.reshape(-1, k), np.diff(A.row_offset), dt, alpha,
                                 beta, Y0)
        assert ok, f"k={k} alpha={alpha} beta={beta}: max normalised error {mx}"


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("align", [1, 0])
@pytest.mark.parametrize("fmt", ["ell", "sell", "sell_c_sigma", "sell_c_R"])
def test_widths(fmt, align, dt, oracle_lib):
    rng = np.random.default_rng(2)
    for width in [*range(1, 14), 20, 33, 70]:
        for lens in (np.full(1027, width), rng.integers(0, width + 1, 1027)):
            A = _matrix(lens, 611, dt, width)
            _check(A, _convert(A, fmt, align), dt, [(1, 1.0, 0.0), (1, 0.8, 0.7), (2, 0.8, 0.7), (4, 1.0, 0.0),
                                                    (8, 0.8, 0.7)], oracle_lib)


# 256 rows a block on 152 SMs: 6 and 8 resident blocks an SM, a grid that strides
@pytest.mark.parametrize("m", [6 * 152 * 256, 6 * 152 * 256 + 1, 8 * 152 * 256, 8 * 152 * 256 + 1])
def test_fp64_waves(m, oracle_lib):
    for width in (2, 5, 36):
        A = _matrix(np.full(m, width), 1000, np.float64)
        _check(A, _convert(A, "sell", 1), np.float64, [(1, 1.0, 0.0), (1, 0.8, 0.7)], oracle_lib)


@pytest.mark.parametrize("fmt", ["ell", "sell", "sell_c_sigma", "sell_c_R"])
def test_many_rows(fmt, oracle_lib):
    """700,001 rows: past a strided grid, and past the bound over which short
    uneven rows stay in the thread pass for k = 2 and 4 and for sorted rows."""
    rng = np.random.default_rng(3)
    blocks = rng.poisson(1.0, 175_001).clip(max=12)
    for lens in (np.full(700_001, 5), np.repeat(4 * blocks, 4)[:700_001]):
        A = _matrix(lens, 5000, np.float32)
        _check(A, _convert(A, fmt, 0), np.float32, [(1, 0.8, 0.7), (2, 0.8, 0.7), (4, 1.0, 0.0), (8, 0.8, 0.7)],
               oracle_lib)
