"""The row kernel that fetches all pairs of its rows at once (spmm_rows_simple_staged): every row length, the last rows of a list,
rows without a nonzero, widths on both sides of the tiles, beside segments and alone."""
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from tests.helpers import graph_nodes

pytestmark = pytest.mark.gpu


def _matrix(m, n, long_rows):
    g = torch.Generator(device="cuda").manual_seed(5)
    lens = torch.randint(0, 29, (m,), device="cuda", generator=g)
    lens[:29] = torch.arange(29, device="cuda")
    lens[-3:] = torch.tensor([28, 0, 1], device="cuda")
    lens[torch.randperm(m - 64, device="cuda", generator=g)[:long_rows] + 32] = 700
    return W._from_sorted_keys(W._distinct_columns(lens, n, g), m, n, -1.0, 1.0, g)


@pytest.mark.parametrize("m,long_rows", [(20011, 0), ((1 << 19) + 3, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_rows_against_fp64(m, long_rows, dtype):
    A = _matrix(m, 3001, long_rows)
    meta = capi.preprocess(A.row_ptr, A.nnz)
    assert (meta.m1 > 0) == (long_rows > 0)
    val = A.val.to(dtype)
    sparse = torch.sparse_csr_tensor(A.row_ptr.long(), A.col.long(), val.double(), size=(A.m, A.n))
    size = 4 if dtype == torch.float32 else 8
    for n in (4, 16, 128 // size, 36, 256 // size, 96, 512 // size, 1024 // size):  # (512 bytes and more: the 256-byte tile's kernel)
        B = W.dense(A.n, n, device="cuda", seed=n, dtype=dtype)
        out = []
        nodes = graph_nodes(lambda: out.append(capi.spmm(meta, A.row_ptr, A.col, val, B)))
        if n * size <= 256 or (long_rows == 0 and n * size % 512 == 0):
            assert any("spmm_rows_simple" in k for k in nodes), nodes
        C = capi.spmm(meta, A.row_ptr, A.col, val, B)
        want = sparse @ B.double()
        # sums of fewer than 32 products of magnitude below 1 (700 in the long rows): (terms + 1) roundings each at most
        eps = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
        bound = 33 * eps * 32 if long_rows == 0 else 701 * eps * 64
        assert float((C.double() - want).abs().max()) < bound, n
        listed = torch.zeros_like(C)
        capi.spmm(meta, A.row_ptr, A.col, val, B, C=listed)
        assert torch.equal(listed, C), n
