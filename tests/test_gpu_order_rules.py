"""Which matrices an order of the segments by their columns is taken for: the samples that the verdict rests on, and the lines
of rode_spmm_order_pays and rode_sddmm_order_pays between matrices on which both sides were timed."""
import pytest
import torch

from rode_b200 import capi

pytestmark = pytest.mark.gpu


def _rows_of(length, rows, n, seed=1):
    """Rows of one length with uniform columns, ascending."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    col = torch.randint(0, n, (rows, length), generator=g, device="cuda", dtype=torch.int32).sort(1).values
    row_ptr = (torch.arange(rows + 1, device="cuda") * length).to(torch.int32)
    meta = capi.preprocess(row_ptr, col.numel())
    col = col.reshape(-1).contiguous()
    return meta, col.numel(), capi.order_verdict(meta, row_ptr, col, n)


@pytest.mark.parametrize("length", [1000, 1024, 1536])
def test_rows_as_long_as_the_distance_of_the_samples_are_not_skewed(length):
    n = 1 << 20
    meta, nnz, verdict = _rows_of(length, 8192, n)
    assert capi.spmm_order_pays(verdict, meta.m1, n, 96, nnz)  # (skewed columns take no order at this width)


@pytest.mark.parametrize("length,rows,pays", [  # 256-byte and 512-byte rows
    (256, 40000, (True, False)), (400, 30000, (True, False)), (500, 30000, (True, False)), (500, 9000, (True, False)),
    (100, 200000, (False, False)), (160, 80000, (True, True)), (600, 7000, (True, True)), (1500, 4000, (True, True)),
    (100, 20000, (False, False))])
def test_spmm_orders_segments_that_span_little_of_the_columns(length, rows, pays):
    n = 700_001
    meta, nnz, verdict = _rows_of(length, rows, n)
    assert tuple(capi.spmm_order_pays(verdict, meta.m1, n, width, nnz) for width in (64, 128)) == pays
    assert not capi.spmm_order_pays(-1, meta.m1, n, 128, nnz)


def test_spmm_of_128_byte_rows_orders_no_wide_segments():
    meta, nnz, verdict = _rows_of(100, 200_000, 1_400_001)
    assert not capi.spmm_order_pays(verdict, 100_000, 1_400_001, 32, nnz)
    meta, nnz, verdict = _rows_of(3000, 8000, 1_400_001)
    assert capi.spmm_order_pays(verdict, meta.m1, 1_400_001, 32, nnz)


@pytest.mark.parametrize("n,k,length,per_column,pays", [
    (1_400_001, 32, 64, 2, False), (1_400_001, 32, 64, 4, True), (700_001, 64, 40, 3, False), (700_001, 64, 128, 7, True),
    (700_001, 96, 40, 3, False), (700_001, 96, 40, 4, True), (1_400_001, 96, 2000, 4, False),
    (1_400_001, 96, 2000, 7, True), (700_001, 128, 32, 1, False), (700_001, 128, 32, 3, True)])
def test_sddmm_orders_where_columns_are_shared(n, k, length, per_column, pays):
    meta, nnz, verdict = _rows_of(length, per_column * n // length + 1, n)
    assert verdict >= 0
    m1 = meta.m1 if length > 512 else max(meta.m1, 1 << 15)
    assert capi.sddmm_order_pays(verdict, nnz // length, m1, n, k, nnz) is pays
    assert not capi.sddmm_order_pays(-1, meta.m1, 1 << 15, n, k, nnz) and not capi.sddmm_order_pays(-3, meta.m1, 1 << 15, n, k, nnz)
