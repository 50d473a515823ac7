"""SpMM into a C of any contents (rode_spmm_f32_all / _f64_all): every row is written, the empty ones with
zeros, in every form of the residue kernel, and rows cut into few and into many segments are summed."""
import numpy as np
import pytest
import torch

from rode_b200 import capi
from rode_b200 import workloads as W
from tests.helpers import assert_close_to_truth, spmm_abs_scale

pytestmark = pytest.mark.gpu


def _matrix(rows, seed=0):
    """Row lengths 0..40 with many empty rows at every start alignment, and rows of 24, 25, 26 and 100
    segments of 32."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 41, rows) * (rng.random(rows) < 0.6)
    for r, l in zip((1, rows // 3, rows // 2, rows - 2), (768, 800, 832, 3201)):
        lens[r] = l
    lens[-1] = 0
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, 5000, rp[-1]).astype(np.int32)
    val = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    return W.CSR(rows, 5000, torch.from_numpy(rp), torch.from_numpy(col), torch.from_numpy(val))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rows", [37, 5000, 70001])     # one warp per row; between; a lane group or bundle per row
@pytest.mark.parametrize("n", [4, 32, 48, 64, 96, 100, 128, 160, 224, 256])
def test_every_row_is_written(oracle_cpu, n, rows, dtype):
    A = _matrix(rows)
    d = A.to("cuda")
    B = W.dense(A.n, n, seed=n)
    rp, col, val = A.row_ptr.numpy(), A.col.numpy(), A.val.numpy()
    truth = oracle_cpu.spmm_f64acc(rp, col, val, B.numpy(), threads=oracle_cpu.max_threads())
    scale = spmm_abs_scale(rp, col, val, B.numpy())
    for seg in (32, 512):
        meta = capi.preprocess(d.row_ptr, d.nnz, seg, 32, 4)
        vd, Bd = d.val.to(dtype), B.to("cuda", dtype)
        ws = torch.empty(capi.spmm_workspace_bytes(meta.m1, n, Bd.element_size()), dtype=torch.uint8, device="cuda")
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        # one chain; two streams; the kernels for a known number of nonzeros
        for streams, nnz in (((None, None), -1), ((None, side), -1), ((None, None), A.nnz)):
            buf = torch.full((A.m + 2, n), float("nan"), dtype=dtype, device="cuda")
            torch.cuda.synchronize()
            C = buf[1:-1]
            capi.spmm_all_raw(dtype, A.m, meta.m1, A.n, n, vd.data_ptr(), d.col.data_ptr(), d.row_ptr.data_ptr(),
                              meta.block_r_ind.data_ptr(), meta.st_off.data_ptr(), Bd.data_ptr(), C.data_ptr(),
                              ws.data_ptr(), ws.numel(), *streams, nnz=nnz)
            torch.cuda.synchronize()
            assert_close_to_truth(C.cpu().numpy(), truth, scale, f"n={n} rows={rows} seg={seg}")
            assert torch.isnan(buf[0]).all() and torch.isnan(buf[-1]).all()
            assert bool((C[torch.from_numpy(np.diff(rp) == 0).cuda()] == 0).all())
            # the list form, into a zero-filled C, gives the same bits
            if nnz < 0:
                Z = torch.zeros_like(C)
                capi.spmm(meta, d.row_ptr, d.col, vd, Bd, C=Z, workspace=ws)
                assert torch.equal(Z, C)
