"""The stream kernel's form for an X that does not fit in L2 (rows of 32 bytes,
more than 100 MB of them): the same bits as the form for a small X, on the same
matrix with its columns drawn from the first rows of X."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (0.8, 0.7)])
@pytest.mark.parametrize("dt,k", [(np.float32, 8), (np.float64, 4)], ids=["f32", "f64"])
def test_big_x_same_bits(dt, k, alpha, beta):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300.synth import HostCSR
    rng = np.random.default_rng(3)
    lens = np.concatenate([rng.integers(0, 40, 4000), [30_000, 0, 1]])
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 1000, rp[-1]).astype(np.int32)
    cv = rng.uniform(-1, 1, rp[-1]).astype(dt)
    big = (101 << 20) // 32 + 7
    out = []
    for n in (1000, big):
        M = L.csr_from_host(HostCSR(len(lens), n, rp, ci, cv))
        X = torch.full((n, k), float("nan"), dtype=torch.float32 if dt == np.float32 else torch.float64, device="cuda")
        X[:1000] = torch.from_numpy(rng.uniform(-1, 1, (1000, k)).astype(dt)).cuda() if not out else out[0][0][:1000]
        Y = torch.ones((len(lens), k), dtype=X.dtype, device="cuda")
        L.spmm(alpha, M, X, beta, Y)
        out.append((X, Y))
    assert torch.isfinite(out[0][1]).all()
    assert torch.equal(out[0][1], out[1][1])
