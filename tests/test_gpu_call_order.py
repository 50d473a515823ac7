"""The first grid of a call starts while the work before it on the stream ends: it must not read before that work has written.
Every input of the call is written right before it, behind a kernel that keeps the GPU busy, and so is what the call
writes read by the kernels before it."""
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W

pytestmark = pytest.mark.gpu

MATRICES = {
    "one launch": lambda: W.bernoulli(1000, 1000, 0.01, device="cuda"),
    "segments and rows": lambda: W.pareto_rows(m=40000, n=30000, mean=24, cap=9000, device="cuda"),
    "rows only": lambda: W.stencil27(30, device="cuda"),
    "long rows only": lambda: W.bernoulli(300, 4000, 0.1, device="cuda"),
}


def _late(*tensors):
    """Copies of the tensors that hold something harmless (zeros) until a kernel behind 0.5 ms of work fills them."""
    late = [torch.zeros_like(t) for t in tensors]
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000)
    for a, b in zip(late, tensors):
        torch.add(b, 0, out=a)  # (a kernel, not a copy: only kernels let the next one start early)
    return late


@pytest.mark.parametrize("width", [32, 64, 128])
@pytest.mark.parametrize("which", list(MATRICES))
def test_call_reads_behind_the_work_before_it(which, width):
    A = MATRICES[which]()
    meta = capi.preprocess(A.row_ptr, A.nnz, 32 if width == 128 else 512)
    X, Y = W.dense(A.n, width, device="cuda", seed=1), W.dense(A.m, width, device="cuda", seed=2)
    want_c = capi.spmm(meta, A.row_ptr, A.col, A.val, X)
    want_o = capi.sddmm(meta, A.row_ptr, A.col, A.val, Y, X)
    for _ in range(3):
        blk, st, res, rp, col, val, x, y = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, A.val, X, Y)
        late = capi.RodeMeta(blk, st, res, meta.m1, meta.m2, meta.seg_len, 32, 4)
        c = capi.spmm(late, rp, col, val, x)
        c2 = capi.spmm(late, rp, col, val, x)        # back to back: the second starts in the end of the first
        later = c.clone()
        torch.cuda.synchronize()
        assert torch.equal(c, want_c) and torch.equal(c2, want_c) and torch.equal(later, want_c)
        blk, st, res, rp, col, val, x, y = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, A.val, X, Y)
        late = capi.RodeMeta(blk, st, res, meta.m1, meta.m2, meta.seg_len, 32, 4)
        o = torch.empty_like(val)
        for _ in range(2):
            capi.sddmm(late, rp, col, val, y, x, out=o)
        later = o.clone()
        torch.cuda.synchronize()
        assert torch.equal(o, want_o) and torch.equal(later, want_o)


@pytest.mark.parametrize("rows", [1000, 40000])
def test_preprocess_reads_behind_the_work_before_it(rows):
    A = W.pareto_rows(m=rows, n=rows, mean=24, cap=rows // 4, device="cuda")
    want = capi.preprocess(A.row_ptr, A.nnz)
    for _ in range(3):
        (rp,) = _late(A.row_ptr)
        got = capi.preprocess(rp, A.nnz)
        assert (got.m1, got.m2) == (want.m1, want.m2)
        assert all(torch.equal(a, b) for a, b in zip((got.block_r_ind, got.st_off, got.residue_r_ind),
                                                     (want.block_r_ind, want.st_off, want.residue_r_ind)))


def test_a_call_does_not_overwrite_what_earlier_kernels_still_read():
    """Chains of calls whose results feed the next call and whose memory the allocator hands out again."""
    A = MATRICES["one launch"]()
    meta = capi.preprocess(A.row_ptr, A.nnz)
    X = W.dense(A.n, 32, device="cuda", seed=1)

    def chain(sync):
        x = X
        for _ in range(40):
            x = capi.spmm(meta, A.row_ptr, A.col, A.val, x) * 0.05
            if sync:
                torch.cuda.synchronize()
        return x

    want = chain(True)
    for _ in range(5):
        assert torch.equal(chain(False), want)
