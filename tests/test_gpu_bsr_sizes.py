"""BSR's block stream by the number of blocks (one block a group in half a step,
half a step of several, whole windows): uneven block rows, empty ones, long ones
over many windows.  Against the FP64 oracle with the per-row bound of the parity
tests."""
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
@pytest.mark.parametrize("shape", [(1, 1), (2, 2), (4, 4), (8, 2), (32, 1), (4, 16)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("blocks", [300, 6000, 30_000, 60_000, 250_000])
def test_bsr_by_blocks(blocks, shape, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    r, c = shape
    rng = np.random.default_rng(blocks + r)
    mb = blocks // 3
    lens = rng.integers(0, 6, mb)
    lens[mb // 2] = blocks // 20  # one block row over many windows
    nb = max(4000, blocks // 20 + 1)
    bcol = np.concatenate([np.sort(rng.choice(nb, int(k), replace=False)) for k in lens]) if blocks < 1e5 else \
        np.concatenate([np.arange(k) * (nb // max(int(k), 1)) + rng.integers(0, nb // max(int(k), 1)) for k in lens])
    brow = np.repeat(np.arange(mb), lens)
    rows = np.repeat(lens, r) * c
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    first = np.concatenate([[0], np.cumsum(lens)])
    col = np.empty(int(rp[-1]), np.int32)
    inner = (bcol[:, None] * c + np.arange(c)).astype(np.int32)  # a block's columns
    rank = np.arange(len(bcol)) - first[brow]
    for q in range(r):
        at = rp[brow * r + q] + rank * c
        col[(at[:, None] + np.arange(c)).ravel()] = inner.ravel()
    A = HostCSR(mb * r, nb * c, rp.astype(np.int32), col, rng.uniform(-1, 1, len(col)).astype(dt))
    M = L.csr_to_bsr(L.csr_from_host(A), r, c)
    M.set_kernel(2, 0)
    _check(A, M, dt, oracle_lib)
