"""The work a user of this package has it do, as cases that can be timed.

A case is one call of a public entry point on one sparse matrix:

  op "spmm"       C = S @ X.  float32: ``rode_sddmm.rode_spmm`` on a ``RoDeCSR`` (the Python entry point, popularity
                  hints at their default); float64: ``capi.spmm`` (the Python entry point is float32 only).
  op "sddmm"      values * (lhs @ rhs^T) at the stored entries: ``rode_sddmm.rode_sddmm`` on a ``RoDeCSR``.
  op "decompose"  the row decomposition of a CSR row pointer that is on the GPU, into buffers the caller keeps from
                  step to step: ``capi.preprocess_raw`` (rode_preprocess), with the segment length that ``RoDeCSR``
                  uses for that width (512, or 32 for width 128).

SpMM is a graph layer's forward pass and, on the transposed graph, its backward pass with respect to the features;
SDDMM is the backward pass with respect to the edge values, and attention scores; the decomposition is paid whenever
the sparsity changes.  The matrices are the families of ``rode_b200.workloads`` (the benchmark's own) at their
benchmark sizes, and smaller, odd and rectangular ones, cut to a number of nonzeros that is the same for every seed.
"""
from __future__ import annotations

import math

import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from rode_b200.rode_sddmm import RoDeCSR, rode_sddmm, rode_spmm

DEVICE = "cuda"


def _case(op, family, rows, cols, mean, width, dtype="f32"):
    """rows, cols: shape (stencil: a cube, rmat: a power of two); mean: nonzeros per row (rmat: before duplicates go)."""
    return {"op": op, "family": family, "rows": rows, "cols": cols, "mean": float(mean), "width": width, "dtype": dtype}


def listed():
    stencil, power, graph = 128**3, 1 << 20, 1 << 23
    return [
        # a mini-batch's sampled block: a few thousand nonzeros, where the call itself is what costs
        {"name": "spmm_tiny_n32", **_case("spmm", "bernoulli", 1000, 1000, 10, 32)},
        # one sparse mask small enough to be checked on the CPU (benchmark configuration 1)
        {"name": "sddmm_bernoulli4096_k32", **_case("sddmm", "bernoulli", 4096, 4096, 40.96, 32)},
        # heavy-tailed rows at a medium size: a citation or product graph (benchmark configuration 2)
        {"name": "spmm_zipf65536_n128", **_case("spmm", "zipf", 65536, 65536, 16, 128)},
        # regular short rows: a 27-point stencil or mesh (benchmark configuration 3)
        {"name": "spmm_stencil128_n64", **_case("spmm", "stencil", stencil, stencil, 27, 64)},
        {"name": "sddmm_stencil128_k64", **_case("sddmm", "stencil", stencil, stencil, 27, 64)},
        # power-law degrees with uniform columns: a large interaction graph (benchmark configuration 4)
        {"name": "spmm_pareto20_n32", **_case("spmm", "pareto", power, power, 32, 32)},
        {"name": "sddmm_pareto20_k128", **_case("sddmm", "pareto", power, power, 32, 128)},
        # a web-scale graph on one GPU (benchmark configuration 5)
        {"name": "spmm_rmat23_n128", **_case("spmm", "rmat", graph, graph, 16, 128)},
        {"name": "sddmm_rmat23_k64", **_case("sddmm", "rmat", graph, graph, 16, 64)},
        # double precision, an odd number of rows: a scientific code's block of vectors
        {"name": "spmm_f64_pareto_odd_n64", **_case("spmm", "pareto", 300007, 300007, 24, 64, "f64")},
        # a rectangular matrix with odd sides and a width no tile divides: users x items
        {"name": "sddmm_rect_odd_k96", **_case("sddmm", "zipf", 100003, 50021, 20, 96)},
        # a new sparsity pattern every step: the decomposition of the largest graph's row pointer
        {"name": "decompose_rmat23", **_case("decompose", "rmat", graph, graph, 16, 32)},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """Sizes over their logarithm from a few hundred rows to millions; common widths, and any multiple of four."""
    while True:
        op = rng.choice(["spmm", "spmm", "spmm", "sddmm", "sddmm", "sddmm", "decompose"])
        # (a stencil's sparsity is fixed by its size: nothing to decompose anew)
        family = rng.choice(["bernoulli", "zipf", "pareto", "rmat"] + (["stencil"] if op != "decompose" else []))
        dtype = "f64" if op == "spmm" and rng.random() < 0.2 else "f32"
        width = rng.choice([32, 64, 128]) if rng.random() < 0.7 else 4 * rng.randint(1, 64)
        mean = _log_uniform(rng, 4, 64)
        if family == "bernoulli":
            rows = cols = round(_log_uniform(rng, 500, 12000))
        elif family == "stencil":
            rows = cols = round(_log_uniform(rng, 8, 140)) ** 3
            mean = 27
        elif family == "rmat":
            rows = cols = 1 << rng.randint(10, 22)
        else:
            rows = cols = round(_log_uniform(rng, 500, 1 << 22))
            if rng.random() < 0.4:
                cols = round(_log_uniform(rng, max(500, rows / 4), rows * 4))
        elements = (rows + cols) * width * (2 if dtype == "f64" else 1)
        if rows * mean <= 1 << 26 and rows * mean * width <= 1 << 33 and elements <= 1 << 30:
            return _case(op, family, rows, cols, round(mean, 3), width, dtype)


def _grid(case):
    return round(case["rows"] ** (1 / 3))


def _cut(A, nnz):
    """A without the entries, evenly spaced over it, that it holds beyond ``nnz``."""
    drop = A.nnz - nnz
    if drop < 0:
        raise RuntimeError(f"{A.nnz} entries drawn, {nnz} wanted")
    if drop == 0:
        return A
    at = torch.arange(drop, device=A.col.device, dtype=torch.int64) * A.nnz // drop
    keep = torch.ones(A.nnz, dtype=torch.bool, device=A.col.device)
    keep[at] = False
    row_ptr = A.row_ptr - torch.searchsorted(at, A.row_ptr.to(torch.int64)).to(torch.int32)
    return W.CSR(A.m, A.n, row_ptr, A.col[keep], A.val[keep])


def _matrix(case, seed):
    m, n, mean = case["rows"], case["cols"], case["mean"]
    nnz = _counts(case)[0]
    if case["family"] == "stencil":
        return W.stencil27(_grid(case), device=DEVICE, seed=seed)
    if case["family"] == "bernoulli":
        return _cut(W.bernoulli(m, n, mean / n, device=DEVICE, seed=seed), nnz)
    if case["family"] == "zipf":
        return _cut(W.zipf_rows(m, n, cap=max(64, n // 4), mean=mean, device=DEVICE, seed=seed), nnz)
    if case["family"] == "pareto":
        return _cut(W.pareto_rows(m, n, mean=mean, device=DEVICE, seed=seed), nnz)
    return _cut(W.rmat(scale=m.bit_length() - 1, edge_factor=max(1, round(mean)), device=DEVICE, seed=seed), nnz)


def prepare(case, seed):
    A = _matrix(case, seed)
    op, width = case["op"], case["width"]
    state = {"op": op}
    if op == "decompose":
        seg_len = RoDeCSR.config_for(width)["seg_length"]
        capacity = capi.preprocess_capacity(seg_len, 4, A.m, A.nnz)
        ints = {"block_r_ind": capacity, "st_off": capacity + 1, "residue_r_ind": A.m, "counts": 2}
        state.update(seg_len=seg_len, row_ptr=A.row_ptr,
                     workspace=torch.empty(capi.preprocess_workspace_bytes(A.m), dtype=torch.uint8, device=DEVICE),
                     out={k: torch.zeros(v, dtype=torch.int32, device=DEVICE) for k, v in ints.items()})
        return state
    if case["dtype"] == "f64":
        # (the values and features of a double-precision program have more than 24 significant bits)
        val = A.val.double() * (1.0 + 1e-9 * torch.arange(A.nnz, device=DEVICE, dtype=torch.float64) / A.nnz)
        X = W.dense(A.n, width, device=DEVICE, seed=seed + 1, dtype=torch.float64)
        X *= 1.0 + 1e-9 * torch.arange(width, device=DEVICE, dtype=torch.float64)
        state.update(op="spmm_f64", meta=capi.preprocess(A.row_ptr, A.nnz), row_ptr=A.row_ptr, col=A.col, val=val, X=X)
        return state
    # SpMM takes the decomposition of width 32 (512-long segments) at every width
    S = RoDeCSR(A.row_ptr, A.col, A.val, torch.device(DEVICE), A.m, A.n, k=32 if op == "spmm" else width)
    state["S"] = S
    if op == "spmm":
        state["X"] = W.dense(A.n, width, device=DEVICE, seed=seed + 1)
    else:
        state["lhs"] = W.dense(A.m, width, device=DEVICE, seed=seed + 1)
        state["rhs"] = W.dense(A.n, width, device=DEVICE, seed=seed + 2)
    return state


def run(state):
    op = state["op"]
    if op == "spmm":
        return rode_spmm(state["S"], state["X"])
    if op == "sddmm":
        return rode_sddmm(state["S"], state["lhs"], state["rhs"])
    if op == "spmm_f64":
        return capi.spmm(state["meta"], state["row_ptr"], state["col"], state["val"], state["X"])
    rp, out, ws = state["row_ptr"], state["out"], state["workspace"]
    counts = out["counts"].data_ptr()
    capi.preprocess_raw(state["seg_len"], 32, 4, rp.numel() - 1, rp.data_ptr(), out["block_r_ind"].data_ptr(),
                        out["st_off"].data_ptr(), out["residue_r_ind"].data_ptr(), counts, counts + 4, ws.data_ptr(),
                        ws.numel(), torch.cuda.current_stream())
    return out


def _counts(case):
    """(nonzeros, columns that hold one, rows that hold one): the first exact, the others as expected."""
    m, n, mean = case["rows"], case["cols"], case["mean"]
    if case["family"] == "stencil":
        return (3 * _grid(case) - 2) ** 3, n, m
    if case["family"] == "rmat":
        s = m.bit_length() - 1
        edges = max(1, round(mean)) * m
        a, b, d = 0.57, 0.19, 0.05
        distinct = sum(math.comb(s, i) * math.comb(s - i, j) * 2**j * -math.expm1(-edges * a**i * b**j * d ** (s - i - j))
                       for i in range(s + 1) for j in range(s - i + 1))
        touched = sum(math.comb(s, i) * -math.expm1(-edges * (a + b) ** i * (b + d) ** (s - i)) for i in range(s + 1))
        return int(distinct - 6 * math.sqrt(distinct)), touched, touched
    nnz = int(m * mean - 6 * math.sqrt(m * mean))  # (what six standard deviations leave of a random number of entries)
    return nnz, n * -math.expm1(-nnz / n), m


def work(case):
    nnz, touched_cols, nonempty_rows = _counts(case)
    m, width = case["rows"], case["width"]
    size = 8 if case["dtype"] == "f64" else 4
    if case["op"] == "spmm":    # column and value per nonzero, the row pointer, X's touched rows, all of C
        return {"bytes": (4 + size) * nnz + 4 * (m + 1) + size * width * (touched_cols + m), "flops": 2 * nnz * width}
    if case["op"] == "sddmm":   # column, value and result per nonzero, the row pointer, the touched rows of both operands
        return {"bytes": 12 * nnz + 4 * (m + 1) + 4 * width * (touched_cols + nonempty_rows), "flops": 2 * nnz * width}
    seg_len = RoDeCSR.config_for(width)["seg_length"]
    return {"bytes": 4 * (m + 1) + 8 * nnz / seg_len + 4 * nonempty_rows, "flops": 0}


def tolerance(case):
    if case["op"] == "decompose":
        return "exact"
    # sums of up to 1e5 products: a relative error of a few roundings in the norm, whatever the order of summation
    return {"rel": 1e-14} if case["dtype"] == "f64" else {"rel": 1e-5}
