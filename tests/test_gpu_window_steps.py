"""Windows of one to five steps (the stream and CSR5 kernels take more steps the
more nonzeros a matrix has): rows that end on, before and after a window's end,
rows that run on past it by as much as a warp finishes and by one more, rows
over several windows, runs of empty rows; CSR, COO and CSR5, k right-hand
sides, with alpha and beta, with an X past L2, and in the request server's
batches.  Against the FP64 oracle with the per-row bound of the parity tests;
the device's window records against the numpy restatement of the plan."""
import ctypes as C
import math

import numpy as np
import pytest

from gpu_util import to_dev, to_host
from oracle import tolerance_ok
from test_stream_windows import windows

pytestmark = pytest.mark.gpu

SMS = 152  # GB300


def _steps(nnz, step, first, warps):
    """window_steps: the number of steps of least modelled time."""
    costs = []
    for n in range(1, 6):
        waves = nnz / ((n - 1) * step + first) / (SMS * warps)
        costs.append((math.ceil(waves) if waves <= 6 else waves + 0.5) * (n + 0.35))
    return 1 + int(np.argmin(costs))


def _lens(nnz, T, seed):
    rng = np.random.default_rng(seed)
    edge = [T - 1, 1, T, T + 1, 1, T - 2, T + 31, 1, T + 32, 1, T + 33, T - 33, 33, T - 32, 1, 31, 32, 0, 0, 4 * T + 5, 3,
            *[0] * 300, 2 * T, 256, 255, 257, 7]
    parts, have = [], 0
    while have < nnz:
        parts += [edge, rng.integers(0, 40, 900), rng.integers(1, 4, 300)]
        have += sum(edge) + int(parts[-2].sum()) + int(parts[-1].sum())
    return np.concatenate(parts)


def _matrix(lens, n, dt, seed=5):
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    nnz = int(rp[-1])
    return HostCSR(len(lens), n, rp, rng.integers(0, n, nnz).astype(np.int32), rng.uniform(-1, 1, nnz).astype(dt))


PRODUCTS = [(1, 1.0, 0.0), (1, 0.8, 0.7), (2, 0.8, 0.7), (4, 1.0, 0.0), (4, 0.8, 0.7), (8, 1.0, 0.0), (8, 0.8, 0.7)]


def _check(A, mats, dt, products, oracle_lib):
    from sspmv_gb300 import lespmv as L
    rng = np.random.default_rng(1)
    lens = np.diff(A.row_offset)
    for k, alpha, beta in products:
        X = rng.uniform(-1, 1, (A.num_cols, k)).astype(dt)
        Y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
        y64, absum = oracle_lib.spmm_ref(A, X, alpha, beta, Y0)
        y64, absum = y64.reshape(-1, k), absum.reshape(-1, k)
        for name, M in mats.items():
            Y = to_dev(Y0)
            L.spmm(alpha, M, to_dev(X), beta, Y)
            ok, mx, _ = tolerance_ok(to_host(Y), y64, absum, lens, dt, alpha, beta, Y0)
            assert ok, f"{name} k={k} alpha={alpha} beta={beta}: max normalised error {mx}"


STREAM = [(np.float64, n, int(m * 1e6)) for n, m in ((1, .6), (2, 1.6), (3, 2.8), (4, 4), (5, 5.2))] + \
         [(np.float32, n, int(m * 1e6)) for n, m in ((1, .6), (2, 2), (3, 3.6), (4, 5.2), (5, 6.8))]
IDS = [f"{'f64' if d is np.float64 else 'f32'}-{n}" for d, n, _ in STREAM]


@pytest.mark.parametrize("dt,n,nnz", STREAM, ids=IDS)
def test_stream_steps(dt, n, nnz, oracle_lib):
    from sspmv_gb300 import lespmv as L
    T = 256 * n - 32
    A = _matrix(_lens(nnz, T, n), 3001, dt)
    assert _steps(A.nnz, 256, 224, 30 if dt is np.float64 else 40) == n
    csr = L.csr_from_host(A)
    _check(A, {"csr": csr, "coo": L.csr_to_coo(csr)}, dt, PRODUCTS, oracle_lib)


@pytest.mark.parametrize("dt,n,nnz", STREAM, ids=IDS)
def test_window_records(dt, n, nnz):
    """rec and the split rows of the plan that hangs off the matrix (csrc/plan.cuh:
    Plan), which a first product has built."""
    import torch
    from sspmv_gb300 import lespmv as L
    T = 256 * n - 32
    A = _matrix(_lens(nnz, T, n), 3001, dt)
    M = L.csr_from_host(A)
    L.LeSpMV(1.0, M, to_dev(np.ones(3001, dt)), 0.0, to_dev(np.zeros(A.num_rows, dt)))
    torch.cuda.synchronize()

    class Head(C.Structure):
        _fields_ = [("window", C.c_int), ("windows", C.c_int64), ("rec", C.c_void_p), ("split", C.c_void_p),
                    ("nsplit", C.c_int64)]

    class Raw:
        def __init__(self, address, rows):
            self.__cuda_array_interface__ = dict(shape=(rows, 4), typestr="<i4", data=(address, False), version=2)

    head = Head.from_address(M.s.f.priv + 8)  # StreamPlan, 8-aligned behind Plan::kind
    assert head.window == T and head.windows == -(-A.nnz // T)
    recs, split = windows(A.row_offset.astype(np.int64), T)
    rec = torch.as_tensor(Raw(head.rec, head.windows), device="cuda").cpu().numpy()
    want = np.array(recs)
    live = want[:, 0] < want[:, 1]           # a window without elements names no row
    assert np.array_equal(rec[:, [0, 1, 3]], want[:, [0, 1, 3]]) and np.array_equal(rec[live, 2], want[live, 2])
    got = torch.as_tensor(Raw(head.split, head.nsplit), device="cuda").cpu().numpy()[:, :3]
    assert sorted(map(tuple, got.tolist())) == sorted(split)


@pytest.mark.parametrize("dt,k", [(np.float32, 8), (np.float64, 4)], ids=["f32", "f64"])
def test_steps_with_x_past_l2(dt, k, oracle_lib):
    from sspmv_gb300 import lespmv as L
    A = _matrix(_lens(3_600_000 if dt is np.float32 else 2_800_000, 736, 3), (101 << 20) // 32 + 5, dt)
    _check(A, {"csr": L.csr_from_host(A)}, dt, [(k, 1.0, 0.0), (k, 0.8, 0.7)], oracle_lib)


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("sigma,n,nnz", [(16, 2, 4_400_000), (16, 4, 9_900_000), (12, 3, 5_400_000), (32, 2, 8_000_000)])
def test_csr5_steps(sigma, n, nnz, dt, oracle_lib):
    from sspmv_gb300 import lespmv as L
    A = _matrix(_lens(nnz, 32 * sigma * n, n), 3001, dt)
    assert _steps(A.nnz, 32 * sigma, 32 * sigma, 36 if dt is np.float64 else 40) == n
    M = L.csr_to_csr5(L.csr_from_host(A), sigma, 8)
    _check(A, {"csr5": M}, dt, [PRODUCTS[i] for i in (0, 1, 4, 5)], oracle_lib)


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
def test_batched_steps_equal_lone_calls(dt):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.serving import Server
    mats = [_matrix(_lens(int(m * 1e6), T, T), 3001, dt) for m, T in ((1.8, 480), (3.0, 736), (0.2, 224))]
    rng = np.random.default_rng(4)
    with Server() as s:
        for i, A in enumerate(mats):
            s.add_matrix(i, A)
            s.preload(i)
        lone = [L.csr_from_host(A) for A in mats]
        for k in (1, 2, 4, 8):
            jobs = []
            for i, A in list(enumerate(mats)) * 2:
                x = rng.uniform(-1, 1, (3001, k)).astype(dt)
                y0 = rng.uniform(-1, 1, (A.num_rows, k)).astype(dt)
                y = y0.copy()
                jobs.append((i, x, y0, y, s.submit(i, x, y, 0.8, 0.7)))
            for i, x, y0, y, t in jobs:
                assert s.wait(t, 60.0)["status"] == 0
                want = to_dev(y0)
                L.spmm(0.8, lone[i], to_dev(x), 0.7, want)
                assert np.array_equal(y, to_host(want))
