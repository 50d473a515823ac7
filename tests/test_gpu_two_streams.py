"""Calls whose two streams are not ordered with each other."""
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W

pytestmark = pytest.mark.gpu

BUSY = 50_000_000  # cycles that keep a stream busy, some 25 ms


def test_claims_of_the_rows_are_not_cleared_from_the_other_stream():
    """Segments and rows both claim their work, on streams of their own, and the segments' stream is late: what it clears must
    be the segments' counters alone, or rows still to be claimed start over."""
    n, longs, shorts, cols = 132, 40_000, 1_250_000, 1000  # two column tiles: 37,888 segments and 1.21 million rows, on 148 SMs
    lens = torch.cat([torch.full((longs,), 40), torch.ones(shorts)]).to(torch.int64)
    rp = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]).to(torch.int32).cuda()
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    col = torch.randint(0, cols, (int(rp[-1]),), generator=g, device="cuda", dtype=torch.int32)
    val = torch.rand(col.numel(), generator=g, device="cuda")
    B = W.dense(cols, n, device="cuda", seed=8)
    meta = capi.preprocess(rp, col.numel())
    want = capi.spmm(meta, rp, col, val, B)
    need = capi.spmm_workspace_bytes(meta.m1, n)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    C = torch.full_like(want, float("nan"))
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(BUSY)
    capi.spmm_all_raw(torch.float32, rp.numel() - 1, meta.m1, cols, n, val.data_ptr(), col.data_ptr(), rp.data_ptr(),
                      meta.block_r_ind.data_ptr(), meta.st_off.data_ptr(), B.data_ptr(), C.data_ptr(), ws.data_ptr(), need,
                      s1, s2, nnz=col.numel())
    torch.cuda.synchronize()
    assert torch.equal(C, want)
    segments, rows = ws[need - 256:need - 256 + 16].view(torch.int32).view(2, 2).tolist()  # claims per column tile
    assert min(segments) > 0 and min(rows) > 0
