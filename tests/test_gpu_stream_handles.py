"""The default stream by its raw handle, 0."""
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W

pytestmark = pytest.mark.gpu

BUSY = 50_000_000  # cycles that keep a stream busy, some 25 ms


def test_handle_zero_is_the_default_stream():
    dev = torch.device("cuda", torch.cuda.current_device())
    assert capi._stream_object(0, dev).cuda_stream == 0
    A = W.pareto_rows(m=3000, n=2000, mean=24, cap=900, device="cuda")
    want = capi.preprocess(A.row_ptr, A.nnz)
    X, Y = W.dense(A.n, 32, device="cuda", seed=1), W.dense(A.m, 32, device="cuda", seed=2)
    want_o = capi.sddmm(want, A.row_ptr, A.col, A.val, Y, X)
    side = torch.cuda.Stream()
    late = torch.zeros_like(A.row_ptr)
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    late.copy_(A.row_ptr)                      # on the default stream
    with torch.cuda.stream(side):
        got = capi.preprocess(late, A.nnz, stream=0)
    assert (got.m1, got.m2) == (want.m1, want.m2) and torch.equal(got.block_r_ind, want.block_r_ind)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):              # the fill of a result made here, on a stream that is late
        torch.cuda._sleep(BUSY)
        o = capi.sddmm(want, A.row_ptr, A.col, A.val, Y, X, stream1=0, stream2=0)
    torch.cuda.synchronize()
    assert torch.equal(o, want_o)
