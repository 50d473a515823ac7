"""Calls that order their segments by columns by themselves (rode_spmm, rode_sddmm) at the sizes where they do: warps go through many
bundles of the list and claim from its counters, and the ordering itself runs in hundreds of CTAs."""
import numpy as np
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from rode_b200.rode_sddmm import RoDeCSR, rode_sddmm, rode_sddmm_cuda, rode_spmm
from tests.helpers import (assert_close_to_truth, graph_nodes, sample_rows_csr, sddmm_abs_scale, spmm_abs_scale)
from tests.test_gpu_call_order import _late

pytestmark = pytest.mark.gpu

MATRICES = {
    "pareto": lambda: W.pareto_rows(m=1 << 20, n=1 << 20, mean=24, device="cuda"),
    "zipf": lambda: W.zipf_rows(m=450_007, n=900_001, cap=200_000, mean=40, device="cuda"),
}
_made = {}


def _matrix(which):
    if which not in _made:
        _made.clear()  # one at a time
        _made[which] = MATRICES[which]()
    return _made[which]


def _csr(A, k):
    return RoDeCSR(A.row_ptr, A.col, A.val, torch.device("cuda"), A.m, A.n, k=k)


def _some_rows(A):
    """The longest rows and a sample of all."""
    lens = A.row_ptr[1:] - A.row_ptr[:-1]
    return torch.unique(torch.cat([torch.topk(lens, 6).indices, torch.arange(0, A.m, A.m // 150, device="cuda")]))


def _launches(call, *wanted):
    nodes = graph_nodes(call)
    return all(any(w in name for name in nodes) for w in wanted)


# (64 and 128: tiles of their own; 100: a partly idle tile; 160: two tiles, which share the warps and have a counter each)
@pytest.mark.parametrize("width", [64, 100, 128, 160])
@pytest.mark.parametrize("which", list(MATRICES))
def test_spmm_that_orders_itself(oracle_cpu, which, width):
    A = _matrix(which)
    S, X = _csr(A, 32), W.dense(A.n, width, device="cuda", seed=4)
    assert S.m1 > (80_000 if which == "pareto" else 37_888)  # (75,776 segments make a persistent grid of one tile, 37,888 of two)
    assert _launches(lambda: rode_spmm(S, X), "order_pieces", "spmm_block")
    C = rode_spmm(S, X)
    assert torch.equal(C, rode_spmm(S, X, hints=False)) and torch.equal(C, rode_spmm(S, X))
    rows = _some_rows(A)
    rp, col, val, _ = sample_rows_csr(A, rows)
    Xh = X.cpu().numpy()
    truth = oracle_cpu.spmm_f64acc(rp, col, val, Xh)
    assert_close_to_truth(C[rows].cpu().numpy(), truth, spmm_abs_scale(rp, col, val, Xh), f"{which} N={width}")


@pytest.mark.parametrize("k", [64, 96, 100, 128, 132])
@pytest.mark.parametrize("which", list(MATRICES))
def test_sddmm_that_orders_itself(oracle_cpu, which, k):
    A = _matrix(which)
    S = _csr(A, k)
    lhs, rhs = W.dense(A.m, k, device="cuda", seed=5), W.dense(A.n, k, device="cuda", seed=6)
    assert _launches(lambda: rode_sddmm(S, lhs, rhs), "order_pieces", "sddmm_pieces")
    out = rode_sddmm(S, lhs, rhs)
    assert torch.equal(out, rode_sddmm(S, lhs, rhs))
    meta = capi.RodeMeta(S.block_indices, S.st_offsets, S.residue_indices, S.m1, S.m2, 0, 32, 4)
    plain = capi.sddmm(meta, S.row_offsets, S.column_indices, S.values, lhs, rhs)
    assert float((out - plain).norm() / plain.norm()) < 1e-6  # the additions of a dot product in another order
    rows = _some_rows(A)
    rp, col, val, idx = sample_rows_csr(A, rows)
    L, R = lhs[rows].cpu().numpy(), rhs.cpu().numpy()
    truth = oracle_cpu.sddmm_f64acc(rp, col, val, L, R)
    assert_close_to_truth(out[torch.from_numpy(idx).cuda()].cpu().numpy(), truth, sddmm_abs_scale(rp, col, val, L, R), f"{which} K={k}")


def test_binding_orders_double_precision(oracle_cpu):
    A = _matrix("pareto")
    S, n = _csr(A, 32), 32
    X, val = W.dense(A.n, n, device="cuda", seed=4, dtype=torch.float64), A.val.double()
    args = (S.block_indices, S.residue_indices, S.st_offsets, S.m1, S.m2, S.row_offsets, S.column_indices, val, S.m, S.n, X)
    assert _launches(lambda: rode_sddmm_cuda.spmm_forward(*args, None, True), "order_pieces", "spmm_block")
    C = rode_sddmm_cuda.spmm_forward(*args, None, True)
    plain = rode_sddmm_cuda.spmm_forward(*args)
    assert torch.equal(C, plain)
    rows = _some_rows(A)
    rp, col, v, _ = sample_rows_csr(A, rows)
    Xh = X.float().cpu().numpy()  # (both inputs are numbers of 24 bits)
    truth, scale = oracle_cpu.spmm_f64acc(rp, col, v, Xh), spmm_abs_scale(rp, col, v, Xh)
    # a sum of T products, in any order, is off by at most T 2^-53 times the sum of their magnitudes: both sides' errors
    terms = np.diff(rp)[:, None]
    assert (np.abs(C[rows].cpu().numpy() - truth) <= 2 * terms * 2.0**-53 * scale).all()


def test_binding_orders_values_that_the_rows_do_not_cover():
    k = 128
    A = _matrix("zipf")
    pad = torch.zeros(7, dtype=torch.int32, device="cuda")
    S = RoDeCSR(A.row_ptr, torch.cat([A.col, pad]), torch.cat([A.val, pad.float() + 1]), torch.device("cuda"), A.m, A.n, k=k)
    lhs, rhs = W.dense(A.m, k, device="cuda", seed=5), W.dense(A.n, k, device="cuda", seed=6)
    assert _launches(lambda: rode_sddmm(S, lhs, rhs), "sddmm_pieces")
    out = rode_sddmm(S, lhs, rhs)
    assert torch.equal(out[:-7], rode_sddmm(_csr(A, k), lhs, rhs)) and bool((out[-7:] == 0).all())


@pytest.mark.parametrize("dtype,n", [(torch.float32, 64), (torch.float32, 128), (torch.float32, 160), (torch.float64, 32)])
def test_ordered_spmm_captured_and_on_two_streams(dtype, n):
    A = _matrix("pareto")
    meta, X, val = capi.preprocess(A.row_ptr, A.nnz), W.dense(A.n, n, device="cuda", seed=4, dtype=dtype), A.val.to(dtype)
    want = capi.spmm(meta, A.row_ptr, A.col, val, X)
    ws = torch.empty(capi.spmm_ordered_workspace_bytes(meta.m1, n, X.element_size()), dtype=torch.uint8, device="cuda")
    C = torch.full_like(want, float("nan"))

    def call(s1, s2):
        capi.spmm_ordered_raw(dtype, A.m, meta.m1, A.n, n, A.nnz, val.data_ptr(), A.col.data_ptr(), A.row_ptr.data_ptr(),
                              meta.block_r_ind.data_ptr(), meta.st_off.data_ptr(), X.data_ptr(), C.data_ptr(), ws.data_ptr(),
                              ws.numel(), s1, s2)

    torch.cuda.synchronize()
    call(torch.cuda.Stream(), torch.cuda.Stream())
    torch.cuda.synchronize()
    assert torch.equal(C, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(torch.cuda.current_stream(), torch.cuda.current_stream())
    for _ in range(2):
        C.fill_(float("nan"))
        ws.fill_(0xAB)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(C, want)


@pytest.mark.parametrize("width", [64, 100, 128, 160])
def test_ordered_calls_read_behind_the_work_before_them(width):
    """Every input is written right before the call, by kernels behind a kernel that keeps the GPU busy."""
    A = _matrix("zipf")
    meta = capi.preprocess(A.row_ptr, A.nnz, 32 if width == 128 else 512)
    X, Y = W.dense(A.n, width, device="cuda", seed=1), W.dense(A.m, width, device="cuda", seed=2)
    want_o = capi.sddmm(meta, A.row_ptr, A.col, A.val, Y, X, ordered=True)
    need = capi.spmm_ordered_workspace_bytes(meta.m1, width)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")

    def spmm(blk, st, rp, col, val, x, out):
        capi.spmm_ordered_raw(torch.float32, A.m, meta.m1, A.n, width, A.nnz, val.data_ptr(), col.data_ptr(), rp.data_ptr(),
                              blk.data_ptr(), st.data_ptr(), x.data_ptr(), out.data_ptr(), ws.data_ptr(), need)

    want_c = torch.empty((A.m, width), device="cuda")
    spmm(meta.block_r_ind, meta.st_off, A.row_ptr, A.col, A.val, X, want_c)
    for _ in range(2):
        blk, st, res, rp, col, val, x, y = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, A.val, X, Y)
        c = torch.empty_like(want_c)
        for _ in range(2):  # back to back: the second starts in the end of the first
            spmm(blk, st, rp, col, val, x, c)
        later = c.clone()
        torch.cuda.synchronize()
        assert torch.equal(c, want_c) and torch.equal(later, want_c)
        blk, st, res, rp, col, val, x, y = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, A.val, X, Y)
        late, o = capi.RodeMeta(blk, st, res, meta.m1, meta.m2, meta.seg_len, 32, 4), torch.empty_like(val)
        for _ in range(2):
            capi.sddmm(late, rp, col, val, y, x, out=o, ordered=True)
        later = o.clone()
        torch.cuda.synchronize()
        assert torch.equal(o, want_o) and torch.equal(later, want_o)
