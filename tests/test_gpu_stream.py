"""The stream kernel (csr_stream.cu) where its windows, steps and column
groups have their edges: rows that end on, before and after a window's end,
split rows over many windows, runs of empty rows, one nonzero; CSR and COO; k
right-hand sides with aligned, unaligned and padded X and Y; Inf and NaN in x
and in values that only other rows use.  Against the FP64 oracle with the
per-row bound of the parity tests."""
import ctypes as C

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


_rng = np.random.default_rng(9)
LENS = {
    "one": [1],
    "one_row_of_many_windows": [50_000],
    "window_edges": [479, 1, 480, 481, 1, 478, 511, 1, 512, 513, 447, 33, 448, 1, 31, 32],
    "split_edges": [1, 511, 1, 512, 1, 513, 200, 792, 3, 960, 2, 961, 5, 4000, 0, 0, 7],
    "empty_runs": [0] * 700 + [3, 0, 2000, 0, 0, 1] + [0] * 1500 + [2] * 600 + [0] * 40,
    "short": list(_rng.integers(1, 4, 9000)),
    "mixed": list(np.minimum(_rng.zipf(1.5, 6000), 9000)),
    "ragged": list(_rng.integers(0, 70, 3001)),
}


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("fmt", ["csr", "coo"])
@pytest.mark.parametrize("case", list(LENS))
def test_stream_rows_and_widths(case, fmt, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    A = _matrix(LENS[case], 1237, dt)
    M = L.csr_from_host(A)
    M = L.csr_to_coo(M) if fmt == "coo" else M
    nz = np.diff(A.row_offset)
    rng = np.random.default_rng(1)
    for k, pad, alpha, beta in [(1, 0, 1.0, 0.0), (1, 0, 0.8, 0.7), (1, 2, 1.0, 0.0), (2, 0, 1.0, 0.0), (2, 1, 0.8, 0.7),
                                (4, 0, 0.8, 0.7), (4, 4, 1.0, 0.0), (8, 0, 1.0, 0.0), (8, 0, 0.8, 0.7), (8, 1, 0.8, 0.0),
                                (15, 0, 1.0, 0.7)]:
        X = rng.uniform(-1, 1, (A.num_cols, k + pad)).astype(dt)
        Y0 = rng.uniform(-1, 1, (A.num_rows, k + pad)).astype(dt)
        Y = to_dev(Y0)
        L.spmm(alpha, M, to_dev(X), beta, Y, k=k, ldx=k + pad, ldy=k + pad)
        got = to_host(Y)
        y64, absum = oracle_lib.spmm_ref(A, np.ascontiguousarray(X[:, :k]), alpha, beta,
                                         np.ascontiguousarray(Y0[:, :k]))
        y64, absum = y64.reshape(A.num_rows, k), absum.reshape(A.num_rows, k)
        ok, mx, _ = tolerance_ok(got[:, :k], y64, absum, nz, dt, alpha, beta, Y0[:, :k])
        assert ok, f"{case} k={k} pad={pad} alpha={alpha} beta={beta}: max normalised error {mx}"
        assert np.array_equal(got[:, k:], Y0[:, k:])  # padding columns untouched


@pytest.mark.parametrize("k", [1, 4, 8])
def test_stream_keeps_inf_and_nan_to_their_rows(k):
    """A window's first and last lanes hold other windows' elements: an Inf or
    NaN there, in a value or in x, must not reach this window's rows."""
    from sspmv_gb300 import lespmv as L
    lens = [480, 470, 9, 490, 1, 460, 64] * 9
    A = _matrix(lens, 4000, np.float64)
    row = np.repeat(np.arange(A.num_rows), lens)
    bad = row % 7 == 3
    A.col_index[~bad] %= 2000        # columns 2000.. belong to the bad rows alone
    A.col_index[bad] = 2000 + A.col_index[bad] % 2000
    A.values[bad & (np.arange(A.nnz) % 5 == 0)] = np.nan
    X = np.random.default_rng(2).uniform(-1, 1, (4000, k))
    X[2000:] = np.inf
    Y = to_dev(np.zeros((A.num_rows, k)))
    L.spmm(1.0, L.csr_from_host(A), to_dev(X), 0.0, Y)
    y = to_host(Y)
    good = np.arange(A.num_rows) % 7 != 3
    assert np.all(np.isfinite(y[good])) and np.all(np.isnan(y[~good]))


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
def test_stream_unaligned_arrays(dt, oracle_lib):
    """Arrays one element into larger buffers (no vector loads), and the last
    nonzeros of the arrays."""
    import torch
    from sspmv_gb300 import _lib
    from sspmv_gb300 import lespmv as L
    for nnz_tail in (1, 5, 7):
        A = _matrix([37] * 500 + [nnz_tail], 999, dt)
        ci = torch.zeros(A.nnz + 1, dtype=torch.int32, device="cuda")
        cv = torch.zeros(A.nnz + 1, dtype=torch.float64 if dt is np.float64 else torch.float32, device="cuda")
        rp = to_dev(A.row_offset)
        ci[1:].copy_(torch.from_numpy(A.col_index))
        cv[1:].copy_(torch.from_numpy(A.values))
        s = _lib.Csr()
        _lib.call("sspmv_csr_wrap", C.byref(s), _lib.F64 if dt is np.float64 else _lib.F32, A.num_rows, A.num_cols,
                  A.nnz, C.c_void_p(rp.data_ptr()), C.c_void_p(ci[1:].data_ptr()), C.c_void_p(cv[1:].data_ptr()))
        W = L.CSR_Matrix(s)
        x = np.random.default_rng(3).uniform(-1, 1, A.num_cols).astype(dt)
        y64, absum = oracle_lib.spmm_ref(A, x, 1.0, 0.0)
        for M in (W, L.csr_from_host(A)):
            y = to_dev(np.full(A.num_rows, np.nan, dt))
            L.LeSpMV(1.0, M, to_dev(x), 0.0, y)
            ok, mx, _ = tolerance_ok(to_host(y), y64, absum, np.diff(A.row_offset), dt)
            assert ok, mx
