"""SELL-c-sigma's order of the rows, from the shared-memory sort (sigma up to
16384, several slices a block for short ones) and the global one past it: length
descending in each slice, equal lengths by descending row; rows of one to three
digits of length, ragged last slice and chunk; and the product on the slab."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [4, 12, 256, 1028, 2048, 4096, 4100, 8192, 12288, 16384, 16388])
@pytest.mark.parametrize("m,longest", [(1, 3), (37, 200), (2049, 70_000), (16_384, 9), (50_001, 3000)])
def test_slice_order(m, longest, sigma, oracle_lib):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(m + sigma)
    lens = np.minimum(rng.zipf(1.6, m) - 1, longest)
    lens[rng.integers(0, m)] = longest
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    A = HostCSR(m, 997, rp, rng.integers(0, 997, rp[-1]).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    S = L.csr_to_sell_c_sigma(L.csr_from_host(A), sigma, 4)
    row = np.arange(m)
    want = np.lexsort((-row, -lens, row // sigma))
    assert np.array_equal(S.export()["reorder"][:m], want)
    x, y0 = rng.uniform(-1, 1, 997), rng.uniform(-1, 1, m)
    y = to_dev(y0)
    L.LeSpMV(0.8, S, to_dev(x), 0.7, y)
    y64, absum = oracle_lib.spmm_ref(A, x.reshape(-1, 1), 0.8, 0.7, y0.reshape(-1, 1))
    ok, mx, _ = tolerance_ok(to_host(y).reshape(-1, 1), y64, absum, lens, np.float64, 0.8, 0.7, y0.reshape(-1, 1))
    assert ok, f"max normalised error {mx}"
