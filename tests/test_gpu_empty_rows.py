"""Matrices of mostly empty rows (far more of them than nonzeros): y = beta * y
there, exactly, and written at the speed of the rows' bytes rather than by the
few warps that the nonzeros need.  CSR, COO, CSR5, BSR's block stream and the
request server's batches."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev, to_host
from oracle import tolerance_ok

pytestmark = pytest.mark.gpu


def _sparse(m, n, filled, dt, seed=3):
    """`filled` nonempty rows of 1 to 9 nonzeros among m, and one of 3000."""
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(seed)
    lens = np.zeros(m, np.int64)
    at = np.sort(rng.choice(m, filled, replace=False))
    lens[at] = rng.integers(1, 10, filled)
    lens[at[filled // 2]] = 3000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in lens[at]]).astype(np.int32)
    return HostCSR(m, n, rp, col, rng.uniform(-1, 1, rp[-1]).astype(dt)), at


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("fmt", ["csr", "coo", "csr5", "bsr"])
@pytest.mark.parametrize("m", [257, 512, 70_001])
def test_mostly_empty_rows(m, fmt, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    A, at = _sparse(m, 5000, 17, dt)
    M = L.csr_from_host(A)
    M = M if fmt == "csr" else L.csr_to_bsr(M, 4, 4) if fmt == "bsr" else getattr(L, f"csr_to_{fmt}")(M)
    if fmt == "bsr":
        M.set_kernel(2, 0)
    rng = np.random.default_rng(1)
    for k, pad, alpha, beta in [(1, 0, 1.0, 0.0), (1, 0, 0.8, 0.7), (2, 0, 0.8, 0.7), (4, 1, 0.8, 0.7), (8, 0, 1.0, 0.0),
                                (8, 0, 0.8, 0.7), (8, 3, 0.8, 0.7)]:
        X = rng.uniform(-1, 1, (5000, k + pad)).astype(dt)
        Y0 = rng.uniform(-1, 1, (m, k + pad)).astype(dt)
        Y = to_dev(Y0)
        L.spmm(alpha, M, to_dev(X), beta, Y, k=k, ldx=k + pad, ldy=k + pad)
        got = to_host(Y)
        y64, absum = oracle_lib.spmm_ref(A, np.ascontiguousarray(X[:, :k]), alpha, beta,
                                         np.ascontiguousarray(Y0[:, :k]))
        ok, mx, _ = tolerance_ok(got[:, :k], y64.reshape(m, k), absum.reshape(m, k), np.diff(A.row_offset), dt, alpha,
                                 beta, Y0[:, :k])
        assert ok, f"k={k} pad={pad} beta={beta}: max normalised error {mx}"
        empty = np.ones(m, bool)
        empty[at] = False
        assert np.array_equal(got[empty, :k], dt(beta) * Y0[empty, :k])
        assert np.array_equal(got[:, k:], Y0[:, k:])


@pytest.mark.parametrize("fmt", ["csr", "coo", "csr5"])
def test_empty_rows_take_the_time_of_their_bytes(fmt):
    """4M rows, about 10,000 nonzeros: against a scaling of y, which moves the
    same bytes but the list's.  A few warps writing all rows take a hundred
    times as long."""
    from sspmv_gb300 import lespmv as L
    m = 1 << 22
    A, _ = _sparse(m, 5000, 1400, np.float64)
    M = L.csr_from_host(A)
    M = M if fmt == "csr" else getattr(L, f"csr_to_{fmt}")(M)
    x, y = torch.ones(5000, dtype=torch.float64, device="cuda"), torch.ones(m, dtype=torch.float64, device="cuda")

    def best(call):
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    scale = best(lambda: y.mul_(0.999))
    product = best(lambda: L.LeSpMV(0.8, M, x, 0.7, y))
    assert product < 4 * scale + 0.02, (product, scale)


def test_batches_of_mostly_empty_rows():
    """Batched requests on such matrices, of several sizes together, give the
    bits of lone calls."""
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.serving import Server
    rng = np.random.default_rng(8)
    for dt in (np.float64, np.float32):
        mats = [_sparse(m, 5000, f, dt, 40 + i)[0] for i, (m, f) in enumerate([(30_000, 9), (257, 250), (513, 3), (90_000, 400)])]
        with Server() as s:
            for i, A in enumerate(mats):
                s.add_matrix(i, A)
                s.preload(i)
            for k in (1, 2, 4, 8):
                jobs = []
                for i, A in enumerate(mats * 3):
                    x = rng.uniform(-1, 1, (5000, k)).astype(dt)
                    y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
                    y = y0.copy()
                    jobs.append((i % len(mats), A, x, y0, y, s.submit(i % len(mats), x, y, 0.8, 0.7)))
                for i, A, x, y0, y, t in jobs:
                    assert s.wait(t, 60.0)["status"] == 0
                    want = to_dev(y0)
                    L.spmm(0.8, L.csr_from_host(A), to_dev(x), 0.7, want)
                    assert np.array_equal(y, to_host(want))
