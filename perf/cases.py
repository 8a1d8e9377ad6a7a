"""The workloads that the library's speed is measured on.

A case is one call a user's program makes again and again: y = alpha*A*x +
beta*y on a matrix it has converted once (kind "spmv"), the same for k
right-hand sides ("spmm"), the PyTorch operator on a model's own CSR tensors
("torch"), or the arrival of a new matrix -- conversion from CSR and the first
product with it ("load").  Matrices come from the five families of the
synthetic suite (2-D Laplacian, banded, power-law rows, 4x4 blocks, uniform
random columns), made on the GPU from the seed; every matrix runs the
library's default kernel.

Ranges: 1,000 to 4.2 million rows, at most about 1.2 GB moved by a product
except for the suite's largest matrix, FP32 and FP64, all nine formats, 1 to
16 right-hand sides, y = A*x and y = 0.8*A*x + 0.7*y, rows without nonzeros.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

BAND = (0, 1, -1, 2, -2, 1024, -1024, 2048, -2048)
BLOCK = 4
ZIPF_CAP = 50_000

# What each format is used for: padding within a few times the nonzeros,
# DIA and BSR where the structure is there (duplicate columns of the
# random families have no place in a block).
FAMILIES = {
    "csr": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "coo": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "csr5": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "sell": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "sell_c_sigma": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "sell_c_R": ("laplacian", "banded", "powerlaw", "block", "uniform"),
    "ell": ("laplacian", "banded", "uniform"),
    "dia": ("laplacian", "banded"),
    "bsr": ("block", "banded", "laplacian"),
}


def _case(name=None, kind="spmv", fmt="csr", family="powerlaw", n=1 << 20, per=16, empty=0.0, dtype="f64", k=1,
          alpha=1.0, beta=0.0, p0=0, p1=0):
    """p0, p1: the converter's first two parameters (0 = the library's
    default): SELL-c-sigma (sigma, C), S-ELL and SELL-c-R (C, alignment), BSR
    (r, c), CSR5 (sigma, omega)."""
    c = dict(kind=kind, fmt=fmt, family=family, n=n, per=per, empty=empty, dtype=dtype, k=k, alpha=alpha, beta=beta,
             p0=p0, p1=p1)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # the smallest solver step: a 64 x 64 grid, where launches and the call itself are the time
        _case("csr_laplacian_64_f64", family="laplacian", n=64 * 64),
        # the plain CSR benchmark matrix: 5-point Laplacian on a 1024 x 1024 grid
        _case("csr_laplacian_1024_f64", family="laplacian", n=1024 * 1024),
        # a graph's adjacency matrix in an iteration y = alpha*A*x + beta*y (ranking, diffusion)
        _case("csr_powerlaw_4M_f32", n=1 << 22, dtype="f32", alpha=0.8, beta=0.7),
        # a few right-hand sides at once: block solvers, features of a graph layer, the served k = 8
        _case("csr_spmm8_powerlaw_2M_f32", kind="spmm", n=1 << 21, dtype="f32", k=8),
        # the PyTorch operator in a training or inference step, ragged size, some empty rows
        _case("torch_powerlaw_500k_f32", kind="torch", n=500_009, dtype="f32", empty=0.05),
        # the suite's largest: triplets as they come from an assembly, 134 million nonzeros
        _case("coo_uniform_4M_f64", fmt="coo", family="uniform", n=1 << 22, per=32),
        # a stencil in the padded format, ragged size, single precision
        _case("ell_banded_1M_f32", fmt="ell", family="banded", n=1_000_003, dtype="f32"),
        # sliced and sorted rows with the layout used on GPUs (C = 32, sigma = 4096), odd size
        _case("sell_c_sigma_powerlaw_1M_f64", fmt="sell_c_sigma", n=1_000_003, p0=4096, p1=32),
        # a banded operator by diagonals
        _case("dia_banded_2M_f64", fmt="dia", family="banded", n=1 << 21),
        # small dense blocks (several unknowns per node)
        _case("bsr_block4_2M_f32", fmt="bsr", family="block", n=1 << 21, dtype="f32", p0=4, p1=4),
        # the load-balanced format on uneven rows, the reference's tile size
        _case("csr5_powerlaw_1M_f64", fmt="csr5", n=1 << 20),
        # a new matrix arrives: conversion and the first product (a server's first request)
        _case("load_sell_c_sigma_powerlaw_500k_f64", kind="load", fmt="sell_c_sigma", n=500_000),
    ]


def draw(rng):
    kind = rng.choice(["spmv"] * 6 + ["spmm"] * 2 + ["torch"] + ["load"])
    fmt = "csr" if kind == "torch" else rng.choice(sorted(FAMILIES))
    if kind == "load" and fmt == "csr":
        fmt = "coo"
    family = rng.choice(FAMILIES[fmt])
    n = int(math.exp(rng.uniform(math.log(1000), math.log(1 << (20 if kind == "load" else 22)))))
    if family == "laplacian":
        n = math.isqrt(n) ** 2
    c = _case(kind=kind, fmt=fmt, family=family, n=n,
              per=int(math.exp(rng.uniform(math.log(2), math.log(64)))) if family == "uniform" else 16,
              empty=rng.choice([0.0, 0.0, 0.05]) if family in ("powerlaw", "uniform") else 0.0,
              dtype=rng.choice(["f32", "f64"]),
              k=rng.choice([2, 3, 4, 5, 8, 16]) if kind == "spmm" else rng.choice([1, 1, 4]) if kind == "torch" else 1)
    if kind in ("spmv", "spmm") and rng.random() < 0.4:
        c["alpha"], c["beta"] = 0.8, 0.7
    if fmt == "sell_c_sigma" and rng.random() < 0.6:
        c["p0"], c["p1"] = rng.choice([256, 4096]), rng.choice([8, 16, 32])
    elif fmt in ("sell", "sell_c_R") and rng.random() < 0.6:
        c["p0"], c["p1"] = rng.choice([8, 16, 32]), rng.choice([0, 1])
    elif fmt == "bsr":
        c["p0"] = c["p1"] = rng.choice([2, 4, 4, 8])
    elif fmt == "csr5" and rng.random() < 0.5:
        c["p0"], c["p1"] = rng.choice([16, 32]), rng.choice([16, 32])
    while work(c)["bytes"] > 1.2e9:
        c["n"] = c["n"] // 2 + rng.randrange(3)
        if family == "laplacian":
            c["n"] = math.isqrt(c["n"]) ** 2
    return c


# ---------------------------------------------------------------- matrices --
@functools.lru_cache(maxsize=None)
def _zipf(alpha, cap):
    """Cumulative Zipf law on [1, cap] and its mean."""
    w = np.arange(1, cap + 1, dtype=np.float64) ** -alpha
    return np.cumsum(w) / w.sum(), float((w * np.arange(1, cap + 1)).sum() / w.sum())


def _nnz(case):
    """Expected number of nonzeros."""
    n, fam = case["n"], case["family"]
    if fam == "laplacian":
        return 5 * n - 4 * math.isqrt(n)
    if fam == "banded":
        return sum(max(0, n - abs(o)) for o in BAND)
    if fam == "block":
        return (n // 4) * BLOCK * BLOCK
    return int(n * case["per"] * (1.0 - case["empty"]))


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _csr(case, seed):
    """The case's matrix as CSR tensors on the GPU (int32 indices).  A load's
    row lengths and blocks are those of the case, so that the arrays it
    returns have the same sizes for every seed; its columns and values are the
    seed's."""
    dev, n, fam, per = "cuda", case["n"], case["family"], case["per"]
    g = torch.Generator(dev).manual_seed(seed)
    shape = torch.Generator(dev).manual_seed(n) if case["kind"] == "load" else g
    rand = lambda *s: torch.rand(*s, generator=shape, device=dev, dtype=torch.float64)  # noqa: E731
    if fam in ("laplacian", "banded"):
        i = torch.arange(n, device=dev).unsqueeze(1)
        if fam == "banded":
            off = torch.tensor(sorted(BAND), device=dev)
            cols = i + off
            ok = (cols >= 0) & (cols < n)
        else:
            e = math.isqrt(n)
            off = torch.tensor([-e, -1, 0, 1, e], device=dev)
            cols = i + off
            ok = (cols >= 0) & (cols < n)
            ok &= ~((off == -1) & (i % e == 0)) & ~((off == 1) & (i % e == e - 1))
        lens = ok.sum(1)
        col = cols[ok]
    elif fam == "block":
        nb = -(-n // BLOCK)
        key = torch.unique(torch.randint(nb * nb, (n // 4,), generator=shape, device=dev))
        inner = torch.arange(BLOCK, device=dev)
        row = ((key // nb) * BLOCK).view(-1, 1, 1) + inner.view(1, -1, 1)
        col = ((key % nb) * BLOCK).view(-1, 1, 1) + inner.view(1, 1, -1)
        row, col = torch.broadcast_tensors(row, col)
        ok = (row < n) & (col < n)
        key = torch.sort(row[ok] * n + col[ok]).values
        lens = torch.bincount(key // n, minlength=n)
        col = key % n
    elif fam == "uniform" and not case["empty"]:
        lens = torch.full((n,), per, device=dev)
        col = torch.randint(n, (n, per), generator=g, device=dev, dtype=torch.int32).sort(1).values.reshape(-1)
    else:
        if fam == "uniform":
            lens = torch.full((n,), per, device=dev)
        else:
            cdf, mean = _zipf(1.8, min(ZIPF_CAP, n))
            z = torch.searchsorted(torch.from_numpy(cdf).to(dev), rand(n)) + 1
            lens = torch.floor(z * (per / mean) + rand(n)).long().clamp(1, min(ZIPF_CAP, n))
        if case["empty"]:
            lens = torch.where(rand(n) < case["empty"], 0, lens)
        row = torch.repeat_interleave(torch.arange(n, device=dev), lens)
        col = torch.randint(n, (row.numel(),), generator=g, device=dev)
        col = torch.sort(row * n + col).values % n
    rp = torch.zeros(n + 1, dtype=torch.int32, device=dev)
    rp[1:] = torch.cumsum(lens, 0)
    nnz = col.numel()
    if fam == "laplacian":
        row = torch.repeat_interleave(torch.arange(n, device=dev), lens)
        val = torch.where(col == row, 4.0, -1.0).to(_dtype(case))
    else:
        val = (torch.rand(nnz, generator=g, device=dev, dtype=_dtype(case)) * 2 - 1)
    return rp, col.to(torch.int32), val


def _vectors(case, seed):
    g = torch.Generator("cuda").manual_seed(seed ^ 0x5EED)
    shape = (case["n"],) if case["k"] == 1 else (case["n"], case["k"])
    return [torch.rand(shape, generator=g, device="cuda", dtype=_dtype(case)) * 2 - 1 for _ in range(2)]


# ------------------------------------------------------------------- calls --
def _matrix(csr):
    """A library matrix from a program's own device arrays."""
    from sspmv_gb300 import _lib
    from sspmv_gb300 import lespmv as L
    rp, col, val = csr
    s = _lib.Csr()
    n = rp.numel() - 1
    _lib.call("sspmv_csr_create", ctypes.byref(s), _lib.F64 if val.dtype == torch.float64 else _lib.F32, n, n,
              col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr(), 0,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.current_stream().synchronize()
    return L.CSR_Matrix(s)


def _convert(case, csr):
    from sspmv_gb300 import lespmv as L
    fmt = case["fmt"]
    convert = getattr(L, "csr_to_" + fmt)
    return convert(csr, case["p0"], case["p1"]) if fmt in ("sell", "sell_c_sigma", "sell_c_R", "bsr", "csr5") \
        else convert(csr)


def prepare(case, seed):
    csr = _csr(case, seed)
    x, y = _vectors(case, seed)
    state = dict(case=case, x=x, y=y)
    if case["kind"] == "torch":
        import sspmv_gb300.torch_ops  # noqa: F401  (registers the operator)
        state["csr"] = csr
        return state
    A = _matrix(csr)
    if case["kind"] == "load" or case["fmt"] == "csr":
        state["A"] = A
        return state
    state["A"] = _convert(case, A)
    A.delete()
    return state


class _Array:
    """A matrix's own device array, for torch.as_tensor, which keeps this
    object and so the matrix."""

    def __init__(self, owner, pointer, count, kind):
        self.owner = owner
        address = ctypes.cast(pointer, ctypes.c_void_p).value
        self.__cuda_array_interface__ = dict(shape=(count,), typestr=kind, data=(address, False), version=2)


def _arrays(A):
    """The arrays of a converted matrix."""
    s, n, nnz = A.s, A.num_rows, A.num_nnzs
    v = "<f8" if A.dtype is np.float64 else "<f4"
    if A.fmt in ("sell", "sell_c_sigma", "sell_c_R"):
        chunks = s.chunk_num if A.fmt == "sell" else s.validchunkNum
        out = dict(chunk_ptr=(s.chunk_ptr, chunks + 1, "<i8"), col=(s.col_index, s.total_slots, "<i4"),
                   values=(s.values, s.total_slots, v))
        if A.fmt != "sell":
            out["reorder"] = (s.reorder, n, "<i4")
    elif A.fmt == "ell":
        out = dict(col=(s.col_index, n * s.max_row_width, "<i4"), values=(s.values, n * s.max_row_width, v))
    elif A.fmt == "coo":
        out = dict(row=(s.row_index, nnz, "<i4"), col=(s.col_index, nnz, "<i4"), values=(s.values, nnz, v))
    elif A.fmt == "dia":
        out = dict(offsets=(s.diag_offsets, s.complete_ndiags, "<i8"),
                   values=(s.diag_data, s.complete_ndiags * s.stride, v))
    elif A.fmt == "bsr":
        out = dict(row_ptr=(s.row_ptr, s.mb + 1, "<i4"), col=(s.block_colindex, s.nnzb, "<i4"),
                   values=(s.block_data, s.nnzb * s.blockNNZ, v))
    else:
        out = dict(col=(s.col_index, nnz, "<i4"), values=(s.values, nnz, v), tile_ptr=(s.tile_ptr, s._p + 1, "<i4"),
                   tile_desc=(s.tile_desc, s._p * s.omega * s.num_packets, "<i4"))
    return {k: torch.as_tensor(_Array(A, *a), device="cuda") for k, a in out.items()}


def run(state):
    from sspmv_gb300 import lespmv as L
    case, x, y = state["case"], state["x"], state["y"]
    kind = case["kind"]
    if kind == "spmv":
        L.LeSpMV(case["alpha"], state["A"], x, case["beta"], y)
        return y
    if kind == "spmm":
        L.spmm(case["alpha"], state["A"], x, case["beta"], y)
        return y
    if kind == "torch":
        rp, col, val = state["csr"]
        return torch.ops.sspmv.spmv_csr(rp, col, val, case["n"], x)
    if "B" in state:
        state.pop("B").delete()  # the matrix that the new one replaces
    state["B"] = B = _convert(case, state["A"])
    L.LeSpMV(case["alpha"], B, x, case["beta"], y)
    return dict(_arrays(B), y=y)


def work(case):
    """One product: the format's structure and values (no padding), x once, y
    once (twice with beta != 0).  A load also reads CSR and writes the format."""
    n, nnz, k = case["n"], _nnz(case), case["k"]
    sv = 8 if case["dtype"] == "f64" else 4
    csr = nnz * (sv + 4) + 4 * n
    own = {"coo": nnz * (sv + 8), "dia": nnz * sv, "ell": nnz * (sv + 4)}.get(case["fmt"], csr)
    if case["fmt"] == "bsr" and case["family"] == "block" and case["p0"] == BLOCK:
        own = nnz * sv + nnz // 16 * 4 + n
    vectors = n * k * sv * (3 if case["beta"] else 2)
    return dict(bytes=own + vectors + (csr if case["kind"] == "load" else 0), flops=2 * nnz * k)


def exact(case, seed):
    """The product in 64 bits; the arrays of a converted matrix are copies."""
    rp, col, val = _csr(case, seed)
    x, y = (t.double() for t in _vectors(case, seed))
    n, k = case["n"], case["k"]
    out = torch.zeros((n, k), dtype=torch.float64, device="cuda")
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    x2 = x.reshape(n, k)
    step = max(1, (1 << 25) // k)
    for a in range(0, col.numel(), step):
        c = col[a:a + step].long()
        out.index_add_(0, row[a:a + step], val[a:a + step].double().unsqueeze(1) * x2[c])
    out = out.reshape(y.shape)
    if case["kind"] != "torch":
        out = case["alpha"] * out + (case["beta"] * y if case["beta"] else 0.0)
    if case["kind"] != "load":
        return out
    names = {"ell": ("col", "values"), "coo": ("row", "col", "values"), "dia": ("offsets", "values"),
             "bsr": ("row_ptr", "col", "values"), "csr5": ("col", "values", "tile_ptr", "tile_desc"),
             "sell": ("chunk_ptr", "col", "values")}.get(case["fmt"], ("chunk_ptr", "col", "values", "reorder"))
    return dict({m: None for m in names}, y=out)
