"""SpMM and SDDMM with the segments in the order of their columns (rode_*_ordered), and the verdict on where that pays."""
import numpy as np
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from tests.helpers import assert_close_to_truth, sddmm_abs_scale

pytestmark = pytest.mark.gpu


def _matrix(n, seed=3):
    """Rows of every length around the pieces' and segments' edges, in a shuffled order, some with shuffled columns; five
    entries in front of the first row and three behind the last belong to no row."""
    rng = np.random.default_rng(seed)
    lens = np.concatenate([np.arange(0, 200), [511, 512, 513, 543, 544, 545, 575, 1023, 1024, 1057, 3001]])
    rng.shuffle(lens)
    rp = (5 + np.concatenate([[0], np.cumsum(lens)])).astype(np.int32)
    col = np.concatenate([np.zeros(5)] + [rng.choice(n, l, replace=False) if i % 5 == 0 else np.sort(rng.choice(n, l, replace=False))
                                          for i, l in enumerate(lens)] + [np.zeros(3)]).astype(np.int32)
    val = rng.uniform(-1, 1, len(col)).astype(np.float32)
    return W.CSR(len(lens), n, torch.from_numpy(rp), torch.from_numpy(col), torch.from_numpy(val))


@pytest.mark.parametrize("seg_len", [32, 512])
@pytest.mark.parametrize("k", [4, 32, 36, 64, 68, 96, 100, 128, 132, 256])
def test_ordered_matches_oracle_and_stays_inside_its_workspace(oracle_cpu, k, seg_len):
    A = _matrix(4099)
    lhs, rhs = W.dense(A.m, k, seed=5), W.dense(A.n, k, seed=6)
    d, lhs_d, rhs_d = A.to("cuda"), lhs.cuda(), rhs.cuda()
    meta = capi.preprocess(d.row_ptr, d.nnz, seg_len)
    need = capi.sddmm_workspace_bytes(meta.m1, k, A.nnz)
    ws = torch.full((need + 256,), 0xAB, dtype=torch.uint8, device="cuda")
    outs = []
    for _ in range(2):  # twice: the second call finds the first one's scratch
        out = torch.full((A.nnz,), float("nan"), device="cuda")
        capi.sddmm_ordered_raw(A.m, meta.m1, meta.m2, A.n, k, A.nnz, meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(),
                               meta.st_off.data_ptr(), d.row_ptr.data_ptr(), d.col.data_ptr(), d.val.data_ptr(),
                               lhs_d.data_ptr(), rhs_d.data_ptr(), out.data_ptr(), ws.data_ptr(), need)
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0][5:-3], outs[1][5:-3]) and bool((ws[need:] == 0xAB).all())
    assert bool(torch.isnan(outs[0][:5]).all()) and bool(torch.isnan(outs[0][-3:]).all())  # entries of no row are left alone
    rp, col, val = A.row_ptr.numpy(), A.col.numpy(), A.val.numpy()
    truth = oracle_cpu.sddmm_f64acc(rp, col, val, lhs.numpy(), rhs.numpy(), threads=oracle_cpu.max_threads())
    scale = sddmm_abs_scale(rp, col, val, lhs.numpy(), rhs.numpy())
    assert_close_to_truth(outs[0].cpu().numpy()[5:-3], truth[5:-3], scale[5:-3], f"k={k} seg_len={seg_len}")
    with pytest.raises(capi.RodeError):
        capi.sddmm_ordered_raw(A.m, meta.m1, meta.m2, A.n, k, A.nnz, *[ws.data_ptr()] * 9, ws.data_ptr(), need - 1)
    # the order changes nothing but the rounding, and not that where the lanes share a row in the same way
    plain = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs_d, rhs_d)
    ordered = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs_d, rhs_d, ordered=True)
    assert bool((plain[:5] == 0).all()) and bool((ordered[:5] == 0).all())
    assert float((ordered - plain).norm() / plain.norm()) < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [4, 32, 64, 96, 100, 128, 132, 256])
def test_ordered_spmm_is_the_same_product(n, dtype):
    A = _matrix(4099)
    d, B = A.to("cuda"), W.dense(A.n, n, seed=6, dtype=dtype).cuda()
    val = d.val.to(dtype)
    for seg_len in (32, 512):
        meta = capi.preprocess(d.row_ptr, d.nnz, seg_len)
        want = capi.spmm(meta, d.row_ptr, d.col, val, B)
        need = capi.spmm_ordered_workspace_bytes(meta.m1, n, B.element_size())
        ws = torch.full((need + 256,), 0xAB, dtype=torch.uint8, device="cuda")
        C = torch.full((A.m, n), float("nan"), device="cuda", dtype=dtype)
        call = [dtype, A.m, meta.m1, A.n, n, A.nnz, val.data_ptr(), d.col.data_ptr(), d.row_ptr.data_ptr(), meta.block_r_ind.data_ptr(),
                meta.st_off.data_ptr(), B.data_ptr(), C.data_ptr(), ws.data_ptr()]
        capi.spmm_ordered_raw(*call, need)
        torch.cuda.synchronize()
        # grids of this size take another kernel without the order: the same sums in another order
        assert float((C - want).norm() / want.norm()) < (1e-6 if dtype == torch.float32 else 1e-15)
        assert bool((ws[need:] == 0xAB).all())
        again = torch.full_like(C, float("nan"))
        call[12] = again.data_ptr()
        capi.spmm_ordered_raw(*call, need)
        assert torch.equal(C, again)
        with pytest.raises(capi.RodeError):
            capi.spmm_ordered_raw(*call, need - 1)


def test_ordered_calls_captured_and_on_two_streams():
    k = 64
    A = _matrix(4099).to("cuda")
    meta = capi.preprocess(A.row_ptr, A.nnz)
    lhs, rhs = W.dense(A.m, k, seed=5).cuda(), W.dense(A.n, k, seed=6).cuda()
    want = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, ordered=True)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    got = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, stream1=s1, stream2=s2, ordered=True)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    out = torch.empty_like(want)
    ws = torch.empty(capi.sddmm_workspace_bytes(meta.m1, k, A.nnz), dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        capi.sddmm_ordered_raw(A.m, meta.m1, meta.m2, A.n, k, A.nnz, meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(),
                               meta.st_off.data_ptr(), A.row_ptr.data_ptr(), A.col.data_ptr(), A.val.data_ptr(), lhs.data_ptr(),
                               rhs.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream(),
                               torch.cuda.current_stream())
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[5:-3], want[5:-3])


def test_verdict():
    n, per, m = 700_001, 40, 70_000
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    u = torch.rand((m, per), generator=g, device="cuda", dtype=torch.float64)
    row_ptr = (torch.arange(m + 1, device="cuda") * per).to(torch.int32)
    kinds = {"uniform": u * n, "skewed": u**12 * n, "band": (torch.arange(m, device="cuda")[:, None] * (n // m) + u * 1000)}
    for kind, c in kinds.items():
        col = c.clamp(0, n - 1).to(torch.int32).sort(1).values.reshape(-1).contiguous()
        meta = capi.preprocess(row_ptr, col.numel())
        assert meta.m1 == m
        verdict = capi.order_verdict(meta, row_ptr, col, n)
        pays = [capi.sddmm_order_pays(verdict, m, meta.m1, n, k, col.numel()) for k in (32, 64, 128)]
        nnz = 12 * n  # as if there were a few more references per column
        assert [capi.spmm_order_pays(verdict, meta.m1, n, k, nnz) for k in (32, 64, 128)] == {
            "uniform": [False, True, True], "skewed": [False, True, True], "band": [False] * 3}[kind], kind
        # 90 MB, 179 MB, 358 MB of rhs
        assert pays == {"uniform": [False, True, True], "skewed": [False, False, True], "band": [False] * 3}[kind], kind
