"""As test_gpu_call_order, for the forms that its matrices and widths do not reach: persistent block grids, hinted gathers, ragged
widths and double precision, each of which has a wait of its own."""
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from tests.helpers import graph_nodes
from tests.test_gpu_call_order import MATRICES, _late

pytestmark = pytest.mark.gpu


def _many_segments():
    """80,000 rows of 40 and as many of 5, columns skewed: more segments than 16 waves of warps, and columns worth marking."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    n, lens = 30_000, torch.cat([torch.full((80_000,), 40), torch.full((80_000,), 5)]).cuda()
    rp = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), lens.cumsum(0)]).to(torch.int32)
    col = (torch.rand(int(rp[-1]), generator=g, device="cuda") ** 4 * n).to(torch.int32).clamp_max(n - 1)
    return W.CSR(lens.numel(), n, rp, col, torch.rand(col.numel(), generator=g, device="cuda"))


def _check_spmm(A, width, dtype=torch.float32, hot=None):
    meta, X, val = capi.preprocess(A.row_ptr, A.nnz), W.dense(A.n, width, device="cuda", seed=1, dtype=dtype), A.val.to(dtype)
    want = capi.spmm(meta, A.row_ptr, A.col, val, X, hot=hot)
    for _ in range(2):
        blk, st, res, rp, col, v, x, *marks = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, val, X,
                                                    *([] if hot is None else [hot]))
        late = capi.RodeMeta(blk, st, res, meta.m1, meta.m2, meta.seg_len, 32, 4)
        c = capi.spmm(late, rp, col, v, x, hot=marks[0] if marks else None)
        c2 = capi.spmm(late, rp, col, v, x, hot=marks[0] if marks else None)  # back to back
        later = c2.clone()
        torch.cuda.synchronize()
        assert torch.equal(c, want) and torch.equal(c2, want) and torch.equal(later, want)


def _check_sddmm(A, k):
    meta = capi.preprocess(A.row_ptr, A.nnz, 32 if k == 128 else 512)
    X, Y = W.dense(A.n, k, device="cuda", seed=1), W.dense(A.m, k, device="cuda", seed=2)
    want = capi.sddmm(meta, A.row_ptr, A.col, A.val, Y, X)
    for _ in range(2):
        blk, st, res, rp, col, v, x, y = _late(meta.block_r_ind, meta.st_off, meta.residue_r_ind, A.row_ptr, A.col, A.val, X, Y)
        late, o = capi.RodeMeta(blk, st, res, meta.m1, meta.m2, meta.seg_len, 32, 4), torch.empty_like(v)
        for _ in range(2):
            capi.sddmm(late, rp, col, v, y, x, out=o)
        later = o.clone()
        torch.cuda.synchronize()
        assert torch.equal(o, want) and torch.equal(later, want)


@pytest.mark.parametrize("which", list(MATRICES))
@pytest.mark.parametrize("width", [36, 96, 132])
def test_ragged_widths(which, width):
    A = MATRICES[which]()
    _check_spmm(A, width)
    _check_sddmm(A, width)


@pytest.mark.parametrize("which", list(MATRICES))
@pytest.mark.parametrize("width", [16, 32, 36, 64])
def test_double_precision(which, width):
    _check_spmm(MATRICES[which](), width, torch.float64)


@pytest.mark.parametrize("width", [32, 36, 64, 96, 100, 128, 132])
def test_persistent_grids(width):
    A = _many_segments()
    meta = capi.preprocess(A.row_ptr, A.nnz)
    assert meta.m1 > 16 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    X = W.dense(A.n, width, device="cuda", seed=1)
    assert "memset" in graph_nodes(lambda: capi.spmm(meta, A.row_ptr, A.col, A.val, X))  # of the claim counters
    _check_spmm(A, width)
    _check_sddmm(A, width)


@pytest.mark.parametrize("width", [128, 256])
def test_hinted_gathers(width):
    A = _many_segments()
    hot = capi.hot_columns(A.col, A.n, 4 * width, budget_bytes=2000 * 4 * width)
    assert hot is not None
    _check_spmm(A, width, hot=hot)
