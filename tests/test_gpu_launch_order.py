"""Calls whose later kernels start under the earlier ones' last wave (long rows,
thread pass, split rows; merge path and its fix-up): a chain of products, each
reading the one before, gives the bits of the same chain with the device
synchronised after every call, launched directly and replayed from a graph."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("fmt", ["csr", "merge", "coo", "csr5", "sell", "sell_c_sigma", "sell_c_R"])
def test_chained_products(fmt, dt):
    from sspmv_gb300 import lespmv as L
    from sspmv_gb300 import synth
    A = synth.generate(synth.powerlaw(60_000, 1.8, 16.0, 30_000, 0.05), 5, dt)
    M = L.csr_from_host(A)
    M = M if fmt in ("csr", "merge") else getattr(L, f"csr_to_{fmt}")(M)
    M.set_kernel(2 if fmt == "merge" else 0, 0)
    x = to_dev(synth.vector(A.num_cols, 0, dt))
    step = 8

    def chain(v, sync):
        for i in range(step):
            L.LeSpMV(0.01, M, v[i], 0.5, v[i + 1])
            if sync:
                torch.cuda.synchronize()

    def fresh():
        return [x.clone()] + [torch.ones_like(x) for _ in range(step)]

    want, got = fresh(), fresh()
    torch.cuda.synchronize()
    chain(want, True)
    chain(got, False)
    torch.cuda.synchronize()
    for a, b in zip(want, got):
        assert torch.equal(a, b)
    rep = fresh()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(rep, False)
    for v, f in zip(rep, fresh()):
        v.copy_(f)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(want, rep):
        assert torch.equal(a, b)
