"""ctypes binding of the C ABI in ``include/rode_b200.h`` (``librode_b200.so``).

torch is used only for device memory and streams: every function takes CUDA tensors (or
raw device addresses) and hands plain pointers and sizes to the library.  There is no CPU
path here: if the library is missing, loading fails loudly.
"""
from __future__ import annotations

import contextlib
import ctypes
import functools
import os
from dataclasses import dataclass
from typing import Optional

import torch

_PKG = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_PKG, "librode_b200.so")

RODE_OK = 0
RODE_ERR_INVALID_ARGUMENT = 1
RODE_ERR_WORKSPACE = 2
RODE_ERR_CUDA = 3
RODE_ERR_NO_DEVICE = 4

# Every symbol include/rode_b200.h declares.
C_ABI_SYMBOLS = (
    "rode_last_error", "rode_version", "rode_preprocess_workspace_bytes", "rode_preprocess_capacity",
    "rode_preprocess", "rode_preprocess_noalloc", "rode_preprocess_cpu", "rode_spmm_workspace_bytes", "rode_spmm_f32", "rode_spmm_f64",
    "rode_sddmm_f32", "rode_hot_columns_workspace_bytes", "rode_hot_columns_words", "rode_hot_columns",
    "rode_spmm_f32_hot", "rode_spmm_f64_hot", "rode_spmm_f32_all", "rode_spmm_f64_all",
    "rode_order_verdict", "rode_sddmm_order_pays", "rode_sddmm_workspace_bytes", "rode_sddmm_f32_ordered",
    "rode_spmm_order_pays", "rode_spmm_ordered_workspace_bytes", "rode_spmm_f32_ordered", "rode_spmm_f64_ordered",
)
# Itanium-ABI names of the C++ entry points declared in RoDeSpmm.h / RoDeSddmm.h /
# RoDePreprocess.h; identical to the names the reference's own objects export.
CPP_SYMBOLS = {
    "RoDeSpmm_n32_f32": "_Z12RoDeSpmm_n32iiiiPKfPKiS2_S2_S2_S2_S0_PfP11CUstream_stS5_",
    "RoDeSpmm_n128_f32": "_Z13RoDeSpmm_n128iiiiPKfPKiS2_S2_S2_S2_S0_PfP11CUstream_stS5_",
    "RoDeSpmm_n32_f64": "_Z12RoDeSpmm_n32iiiiPKdPKiS2_S2_S2_S2_S0_PdP11CUstream_stS5_",
    "RoDeSpmm_n128_f64": "_Z13RoDeSpmm_n128iiiiPKdPKiS2_S2_S2_S2_S0_PdP11CUstream_stS5_",
    "RoDeSDDMM_n32": "_Z13RoDeSDDMM_n32iiiiPKiS0_S0_S0_S0_PKfS2_S2_PfP11CUstream_stS5_",
    "RoDeSDDMM_n64": "_Z13RoDeSDDMM_n64iiiiPKiS0_S0_S0_S0_PKfS2_S2_PfP11CUstream_stS5_",
    "RoDeSDDMM_n128": "_Z14RoDeSDDMM_n128iiiiPKiS0_S0_S0_S0_PKfS2_S2_PfP11CUstream_stS5_",
    "RoDe_preprocess": "_Z15RoDe_preprocessiiiiPKiPiS1_S1_S1_S1_",
    "RoDe_preprocess_cpu": "_Z19RoDe_preprocess_cpuiiiiPKiPiS1_S1_RiS2_",
}


class RodeError(RuntimeError):
    def __init__(self, status: int, message: str):
        super().__init__(f"rode_b200 status {status}: {message}")
        self.status = status


_lib: Optional[ctypes.CDLL] = None


def load() -> ctypes.CDLL:
    """Load ``librode_b200.so`` (built by ``python -m rode_b200.build``).  No fallback."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise RuntimeError(
            f"{LIB_PATH} is missing: build it with `python -m rode_b200.build` (nvcc, sm_100a). "
            "rode_b200 has no CPU or PyTorch fallback."
        )
    lib = ctypes.CDLL(LIB_PATH)
    vp, ci, sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
    lib.rode_last_error.restype = ctypes.c_char_p
    lib.rode_version.restype = ctypes.c_char_p
    lib.rode_preprocess_workspace_bytes.argtypes = [ci, ctypes.POINTER(sz)]
    lib.rode_preprocess_capacity.argtypes = [ci, ci, ci, ctypes.c_longlong, ctypes.POINTER(ctypes.c_longlong)]
    lib.rode_preprocess.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp, vp, sz, vp]
    lib.rode_preprocess_noalloc.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp, vp]
    lib.rode_preprocess_cpu.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp]
    lib.rode_spmm_workspace_bytes.argtypes = [ci, ci, ci, ctypes.POINTER(sz)]
    lib.rode_spmm_f32.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp, vp, vp, vp, sz, vp, vp]
    lib.rode_spmm_f64.argtypes = lib.rode_spmm_f32.argtypes
    lib.rode_sddmm_f32.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, vp]
    lib.rode_hot_columns_workspace_bytes.argtypes = [ci, ctypes.POINTER(sz)]
    lib.rode_hot_columns_words.argtypes = [ci, ctypes.POINTER(sz)]
    lib.rode_hot_columns.argtypes = [ctypes.c_longlong, ci, vp, sz, sz, vp, vp, sz, vp]
    lib.rode_spmm_f32_hot.argtypes = [ci, ci, ci, ci, vp, vp, vp, vp, vp, vp, vp, vp, vp, sz, vp, vp, vp]
    lib.rode_spmm_f64_hot.argtypes = lib.rode_spmm_f32_hot.argtypes
    lib.rode_spmm_f32_all.argtypes = [ci, ci, ci, ci, ctypes.c_longlong, vp, vp, vp, vp, vp, vp, vp, vp, sz, vp, vp, vp]
    lib.rode_spmm_f64_all.argtypes = lib.rode_spmm_f32_all.argtypes
    lib.rode_order_verdict.argtypes = [ci, ci, ctypes.c_longlong, vp, vp, vp, ctypes.POINTER(ci), vp, vp]
    lib.rode_sddmm_order_pays.argtypes = [ci] * 5 + [ctypes.c_longlong]
    lib.rode_spmm_order_pays.argtypes = [ci] * 4 + [ctypes.c_longlong, ci]
    lib.rode_spmm_ordered_workspace_bytes.argtypes = [ci, ci, ci, ctypes.POINTER(sz)]
    lib.rode_spmm_f32_ordered.argtypes = [ci, ci, ci, ci, ctypes.c_longlong, vp, vp, vp, vp, vp, vp, vp, vp, sz, vp, vp]
    lib.rode_spmm_f64_ordered.argtypes = lib.rode_spmm_f32_ordered.argtypes
    lib.rode_sddmm_workspace_bytes.argtypes = [ci, ci, ctypes.c_longlong, ctypes.POINTER(sz)]
    lib.rode_sddmm_f32_ordered.argtypes = [ci, ci, ci, ci, ci, ctypes.c_longlong] + [vp] * 10 + [sz, vp, vp]
    for name in ("rode_preprocess_workspace_bytes", "rode_preprocess_capacity", "rode_preprocess",
                 "rode_preprocess_noalloc", "rode_preprocess_cpu", "rode_spmm_workspace_bytes", "rode_spmm_f32", "rode_spmm_f64",
                 "rode_sddmm_f32", "rode_hot_columns_workspace_bytes", "rode_hot_columns_words", "rode_hot_columns",
                 "rode_spmm_f32_hot", "rode_spmm_f64_hot", "rode_spmm_f32_all", "rode_spmm_f64_all",
                 "rode_order_verdict", "rode_sddmm_order_pays", "rode_sddmm_workspace_bytes", "rode_sddmm_f32_ordered",
                 "rode_spmm_order_pays", "rode_spmm_ordered_workspace_bytes", "rode_spmm_f32_ordered", "rode_spmm_f64_ordered"):
        getattr(lib, name).restype = ci
    _lib = lib
    return lib


def check(status: int) -> None:
    if status != RODE_OK:
        raise RodeError(status, load().rode_last_error().decode())


def version() -> str:
    return load().rode_version().decode()


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _stream(s) -> Optional[int]:
    if s is None:
        return None
    if isinstance(s, torch.cuda.Stream):
        return s.cuda_stream or None
    return int(s) or None


def _dev_i32(t: torch.Tensor, name: str) -> torch.Tensor:
    if not (t.is_cuda and t.dtype == torch.int32 and t.is_contiguous()):
        raise ValueError(f"{name} must be a contiguous CUDA int32 tensor")
    return t


# ---------------------------------------------------------------------------------------
@dataclass
class RodeMeta:
    """Row-decomposition metadata on the device (outputs of the preprocessing)."""

    block_r_ind: torch.Tensor   # int32[max(m1, 1)]
    st_off: torch.Tensor        # int32[m1 + 1]
    residue_r_ind: torch.Tensor  # int32[max(m2, 1)]
    m1: int
    m2: int
    seg_len: int
    k_block: int
    vec_len: int


def preprocess_workspace_bytes(M: int) -> int:
    out = ctypes.c_size_t(0)
    check(load().rode_preprocess_workspace_bytes(M, ctypes.byref(out)))
    return out.value


def preprocess_capacity(seg_len: int, vec_len: int, M: int, nnz: int) -> int:
    out = ctypes.c_longlong(0)
    check(load().rode_preprocess_capacity(seg_len, vec_len, M, nnz, ctypes.byref(out)))
    return out.value


def preprocess_raw(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk, n_res,
                   workspace, workspace_bytes, stream=None) -> None:
    """rode_preprocess on raw device addresses (ints) or tensors' data_ptr()."""
    check(load().rode_preprocess(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk,
                                 n_res, workspace, workspace_bytes, _stream(stream)))


def preprocess_noalloc_raw(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk, n_res,
                           stream=None) -> None:
    """rode_preprocess_noalloc on raw device addresses: the variant for callers that cannot
    allocate device memory (scratch is a fixed array inside the library, M <= 2**24)."""
    check(load().rode_preprocess_noalloc(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind,
                                         n_blk, n_res, _stream(stream)))


def preprocess(row_ptr: torch.Tensor, nnz: int, seg_len: int = 512, k_block: int = 32, vec_len: int = 4,
               stream=None, trim: bool = True) -> RodeMeta:
    """Device-side row decomposition of a CSR row pointer (int32 CUDA tensor [M+1]).

    Allocates outputs at the capacity bound, runs the two kernels on ``stream`` (default:
    torch's current stream), reads the two counts back (one 8-byte D2H copy, which
    synchronises the stream) and returns views trimmed to the counts."""
    _dev_i32(row_ptr, "row_ptr")
    M = row_ptr.numel() - 1
    dev = row_ptr.device
    cap = preprocess_capacity(seg_len, vec_len, M, int(nnz))
    with torch.cuda.device(dev):
        stream = _stream_object(stream, dev)
        with torch.cuda.stream(stream):
            blk = torch.empty(max(cap, 1), dtype=torch.int32, device=dev)
            st = torch.empty(cap + 1, dtype=torch.int32, device=dev)
            res = torch.empty(max(M, 1), dtype=torch.int32, device=dev)
            counts = torch.empty(2, dtype=torch.int32, device=dev)
            ws_bytes = preprocess_workspace_bytes(M)
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
            preprocess_raw(seg_len, k_block, vec_len, M, row_ptr.data_ptr(), blk.data_ptr(), st.data_ptr(),
                           res.data_ptr(), counts.data_ptr(), counts.data_ptr() + 4, ws.data_ptr(), ws_bytes,
                           stream)
            m1, m2 = (int(x) for x in counts.cpu().tolist())
    if trim:
        blk, st, res = blk[: max(m1, 1)], st[: m1 + 1], res[: max(m2, 1)]
    return RodeMeta(blk, st, res, m1, m2, seg_len, k_block, vec_len)


_NULL = contextlib.nullcontext()


def _stream_object(s, dev: torch.device) -> torch.cuda.Stream:
    """The stream of a torch stream, a raw handle (0: the default stream), or None (torch's current one)."""
    if s is None:
        return torch.cuda.current_stream(dev)
    if isinstance(s, torch.cuda.Stream):
        return s
    # (ExternalStream(0) would be a stream of torch's pool)
    return torch.cuda.ExternalStream(int(s), device=dev) if int(s) else torch.cuda.default_stream(dev)


def _current(dev: torch.device) -> int:
    """Handle of torch's current stream (torch.cuda.current_stream builds an object for it, 2 us)."""
    return torch._C._cuda_getCurrentRawStream(dev.index)


def _on(dev: torch.device):
    """torch.cuda.device(dev), or nothing where dev is current already (entering and leaving the
    context costs as much as a launch)."""
    return _NULL if torch.cuda.current_device() == dev.index else torch.cuda.device(dev)


def _used_on(streams, cur: int, dev: torch.device, *tensors) -> None:
    """Tensors just made on the current stream for kernels on others: these wait for it (for a fill, and for earlier
    work on memory that came back to the allocator), and the allocator learns who uses them, so that they are not
    handed out again while those streams still work on them."""
    for s in streams:
        if s is cur:
            continue
        s = _stream_object(s, dev)
        if s.cuda_stream != cur:
            s.wait_stream(torch.cuda.current_stream(dev))
            for t in tensors:
                t.record_stream(s)


def preprocess_cpu(row_ptr: torch.Tensor, seg_len: int = 512, k_block: int = 32, vec_len: int = 4):
    """rode_preprocess_cpu on a HOST int32 tensor (the reference's RoDe_preprocess_cpu API).

    Returns host tensors (block_r_ind[m1], st_off[m1+1], residue_r_ind[m2], m1, m2)."""
    if row_ptr.is_cuda or row_ptr.dtype != torch.int32:
        raise ValueError("row_ptr must be a CPU int32 tensor")
    row_ptr = row_ptr.contiguous()
    M = row_ptr.numel() - 1
    nnz = int(row_ptr[-1]) if M >= 0 and row_ptr.numel() > 0 else 0
    cap = preprocess_capacity(seg_len, vec_len, M, nnz)
    blk = torch.empty(max(cap, 1), dtype=torch.int32)
    st = torch.empty(cap + 1, dtype=torch.int32)
    res = torch.empty(max(M, 1), dtype=torch.int32)
    nb, nr = ctypes.c_int(0), ctypes.c_int(0)
    check(load().rode_preprocess_cpu(seg_len, k_block, vec_len, M, row_ptr.data_ptr(), blk.data_ptr(), st.data_ptr(),
                                     res.data_ptr(), ctypes.addressof(nb), ctypes.addressof(nr)))
    return blk[: nb.value].clone(), st[: nb.value + 1].clone(), res[: nr.value].clone(), nb.value, nr.value


# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=256)
def spmm_workspace_bytes(m1: int, n: int, elem_size: int = 4) -> int:
    out = ctypes.c_size_t(0)
    check(load().rode_spmm_workspace_bytes(m1, n, elem_size, ctypes.byref(out)))
    return out.value


def spmm_raw(dtype, m1, m2, k, n, values, col, row_ptr, blk, res, st, B, C, workspace, workspace_bytes,
             stream1=None, stream2=None, hot=None) -> None:
    """rode_spmm_f32 / _f64 on raw device addresses; with ``hot`` (address of a popularity
    bitmap from ``hot_columns``) the _hot entry points."""
    if hot is None:
        fn = load().rode_spmm_f32 if dtype == torch.float32 else load().rode_spmm_f64
        check(fn(m1, m2, k, n, values, col, row_ptr, blk, res, st, B, C, workspace, workspace_bytes,
                 _stream(stream1), _stream(stream2)))
    else:
        fn = load().rode_spmm_f32_hot if dtype == torch.float32 else load().rode_spmm_f64_hot
        check(fn(m1, m2, k, n, values, col, row_ptr, blk, res, st, B, C, workspace, workspace_bytes, hot,
                 _stream(stream1), _stream(stream2)))


def spmm_all_raw(dtype, M, m1, k, n, values, col, row_ptr, blk, st, B, C, workspace, workspace_bytes, stream1=None,
                 stream2=None, hot=None, nnz=-1) -> None:
    """rode_spmm_f32_all / _f64_all on raw device addresses: C may hold anything, every row is written."""
    fn = load().rode_spmm_f32_all if dtype == torch.float32 else load().rode_spmm_f64_all
    check(fn(M, m1, k, n, nnz, values, col, row_ptr, blk, st, B, C, workspace, workspace_bytes, hot, _stream(stream1),
             _stream(stream2)))


def order_verdict(meta: RodeMeta, row_ptr: torch.Tensor, col: torch.Tensor, n_cols: int) -> int:
    """What rode_order_verdict says of the columns, for ``spmm_order_pays`` and ``sddmm_order_pays``; -1 where the sizes are out
    of its range.  Reads the verdict back where they are not (4-byte D2H copy, synchronises torch's current stream)."""
    in_range, lib = ctypes.c_int(0), load()
    check(lib.rode_order_verdict(meta.m1, n_cols, col.numel(), None, None, None, ctypes.byref(in_range), None, None))
    if not in_range.value:
        return -1
    with torch.cuda.device(col.device):
        verdict = torch.empty(1, dtype=torch.int32, device=col.device)
        check(lib.rode_order_verdict(meta.m1, n_cols, col.numel(), row_ptr.data_ptr(), col.data_ptr(), meta.block_r_ind.data_ptr(),
                                     ctypes.byref(in_range), verdict.data_ptr(), _current(col.device) or None))
        return int(verdict.item())


def spmm_order_pays(verdict: int, m1: int, n_cols: int, width: int, nnz: int, elem_size: int = 4) -> bool:
    return bool(load().rode_spmm_order_pays(verdict, m1, n_cols, width, nnz, elem_size))


def sddmm_order_pays(verdict: int, M: int, m1: int, n_cols: int, k: int, nnz: int) -> bool:
    return bool(load().rode_sddmm_order_pays(verdict, M, m1, n_cols, k, nnz))


def spmm_ordered_workspace_bytes(m1: int, n: int, elem_size: int = 4) -> int:
    out = ctypes.c_size_t(0)
    check(load().rode_spmm_ordered_workspace_bytes(m1, n, elem_size, ctypes.byref(out)))
    return out.value


def spmm_ordered_raw(dtype, M, m1, k, n, nnz, values, col, row_ptr, blk, st, B, C, workspace, workspace_bytes, stream1=None,
                     stream2=None) -> None:
    """rode_spmm_f32_ordered / _f64_ordered on raw device addresses."""
    fn = load().rode_spmm_f32_ordered if dtype == torch.float32 else load().rode_spmm_f64_ordered
    check(fn(M, m1, k, n, nnz, values, col, row_ptr, blk, st, B, C, workspace, workspace_bytes, _stream(stream1),
             _stream(stream2)))


def hot_columns_raw(nnz, n_cols, col, dense_row_bytes, budget_bytes, bitmap, workspace, workspace_bytes,
                    stream=None) -> None:
    check(load().rode_hot_columns(nnz, n_cols, col, dense_row_bytes, budget_bytes, bitmap, workspace,
                                  workspace_bytes, _stream(stream)))


def hot_columns(col: torch.Tensor, n_cols: int, dense_row_bytes: int, budget_bytes: int = 0,
                stream=None) -> Optional[torch.Tensor]:
    """Popularity bitmap of the columns for ``spmm(..., hot=...)`` (rode_hot_columns), or None
    when the library finds that marks would not help on this matrix.  Reads the flag word back
    (4-byte D2H copy, synchronises the stream)."""
    _dev_i32(col, "col")
    dev = col.device
    words, need = ctypes.c_size_t(0), ctypes.c_size_t(0)
    check(load().rode_hot_columns_words(n_cols, ctypes.byref(words)))
    check(load().rode_hot_columns_workspace_bytes(n_cols, ctypes.byref(need)))
    with torch.cuda.device(dev):
        stream = _stream_object(stream, dev)
        with torch.cuda.stream(stream):
            bitmap = torch.empty(words.value, dtype=torch.int32, device=dev)
            ws = torch.empty(need.value, dtype=torch.uint8, device=dev)
            hot_columns_raw(col.numel(), n_cols, col.data_ptr(), dense_row_bytes, budget_bytes, bitmap.data_ptr(),
                            ws.data_ptr(), need.value, stream)
            useful = int(bitmap[-1].item())
    return bitmap if useful else None


def spmm(meta: RodeMeta, row_ptr: torch.Tensor, col: torch.Tensor, values: torch.Tensor, B: torch.Tensor,
         C: Optional[torch.Tensor] = None, workspace: Optional[torch.Tensor] = None, stream1=None,
         stream2=None, hot: Optional[torch.Tensor] = None) -> torch.Tensor:
    """C = S @ B through rode_spmm_f32 / rode_spmm_f64.  Asynchronous on the two streams
    (default: torch's current stream for both; other ones wait for it where ``C`` or ``workspace`` is
    made here).  A given ``C`` must be zero in the rows without a nonzero, which are not written; by
    default C is a fresh tensor of which every row is written.
    ``hot``: popularity bitmap from ``hot_columns`` (same results, fewer DRAM bytes)."""
    M = row_ptr.numel() - 1
    k, n = B.shape
    if values.dtype not in (torch.float32, torch.float64) or B.dtype != values.dtype:
        raise ValueError("values and B must both be float32 or float64")
    if not (B.is_cuda and B.is_contiguous() and values.is_contiguous() and col.is_contiguous()):
        raise ValueError("contiguous CUDA tensors required")
    dev = B.device
    with _on(dev):
        cur = _current(dev)
        s1 = cur if stream1 is None else stream1
        s2 = cur if stream2 is None else stream2
        elsewhere = s1 is not cur or s2 is not cur
        whole = C is None and (meta.m1 > 0 or meta.m2 > 0)
        if C is None:
            C = B.new_empty((M, n)) if whole else B.new_zeros((M, n))
            if elsewhere:
                _used_on((s1, s2), cur, dev, C)
        need = spmm_workspace_bytes(meta.m1, n, B.element_size())
        if workspace is None and need:
            workspace = B.new_empty(need, dtype=torch.uint8)
            if elsewhere:
                _used_on((s1, s2), cur, dev, workspace)
        ws_bytes = 0 if workspace is None else workspace.numel() * workspace.element_size()
        if whole:
            spmm_all_raw(B.dtype, M, meta.m1, k, n, values.data_ptr(), col.data_ptr(), row_ptr.data_ptr(),
                         meta.block_r_ind.data_ptr(), meta.st_off.data_ptr(), B.data_ptr(), C.data_ptr(),
                         _ptr(workspace), ws_bytes, s1, s2, hot=_ptr(hot), nnz=values.numel())
            return C
        spmm_raw(B.dtype, meta.m1, meta.m2, k, n, values.data_ptr(), col.data_ptr(), row_ptr.data_ptr(),
                 meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(), meta.st_off.data_ptr(), B.data_ptr(),
                 C.data_ptr(), _ptr(workspace), ws_bytes, s1, s2, hot=_ptr(hot))
    return C


def sddmm_raw(m1, m2, n, k, blk, res, st, row_ptr, col, values, lhs, rhs, out, stream1=None, stream2=None) -> None:
    check(load().rode_sddmm_f32(m1, m2, n, k, blk, res, st, row_ptr, col, values, lhs, rhs, out, _stream(stream1),
                                _stream(stream2)))


def sddmm_workspace_bytes(m1: int, k: int, nnz: int) -> int:
    """Scratch of ``sddmm_ordered_raw``."""
    out = ctypes.c_size_t(0)
    check(load().rode_sddmm_workspace_bytes(m1, k, nnz, ctypes.byref(out)))
    return out.value


def sddmm_ordered_raw(M, m1, m2, n, k, nnz, blk, res, st, row_ptr, col, values, lhs, rhs, out, workspace, workspace_bytes,
                      stream1=None, stream2=None) -> None:
    """rode_sddmm_f32_ordered on raw device addresses."""
    check(load().rode_sddmm_f32_ordered(M, m1, m2, n, k, nnz, blk, res, st, row_ptr, col, values, lhs, rhs, out, workspace,
                                        workspace_bytes, _stream(stream1), _stream(stream2)))


def sddmm(meta: RodeMeta, row_ptr: torch.Tensor, col: torch.Tensor, values: torch.Tensor, lhs: torch.Tensor,
          rhs: torch.Tensor, out: Optional[torch.Tensor] = None, stream1=None, stream2=None,
          ordered: bool = False) -> torch.Tensor:
    """out[e] = values[e] * <lhs[row(e)], rhs[col(e)]> through rode_sddmm_f32.  A given ``out`` keeps what it holds in the
    entries outside [row_ptr[0], row_ptr[M]); by default they are zero.  ``ordered``: through rode_sddmm_f32_ordered, with
    scratch made here (``sddmm_order_pays`` says where that is faster)."""
    k = lhs.shape[1]
    if lhs.dtype != torch.float32 or rhs.dtype != torch.float32 or values.dtype != torch.float32:
        raise ValueError("float32 tensors required")
    if rhs.shape[1] != k:
        raise ValueError("lhs and rhs must have the same number of columns")
    dev = lhs.device
    with _on(dev):
        cur = _current(dev)
        s1 = cur if stream1 is None else stream1
        s2 = cur if stream2 is None else stream2
        if out is None:  # (entries that belong to no row of row_ptr are not written)
            out = values.new_zeros(values.numel())
            _used_on((s1, s2), cur, dev, out)
        if not ordered:
            sddmm_raw(meta.m1, meta.m2, rhs.shape[0], k, meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(),
                      meta.st_off.data_ptr(), row_ptr.data_ptr(), col.data_ptr(), values.data_ptr(), lhs.data_ptr(),
                      rhs.data_ptr(), out.data_ptr(), s1, s2)
            return out
        need = sddmm_workspace_bytes(meta.m1, k, values.numel())
        workspace = values.new_empty(need, dtype=torch.uint8)
        _used_on((s1, s2), cur, dev, workspace)
        sddmm_ordered_raw(row_ptr.numel() - 1, meta.m1, meta.m2, rhs.shape[0], k, values.numel(), meta.block_r_ind.data_ptr(),
                          meta.residue_r_ind.data_ptr(), meta.st_off.data_ptr(), row_ptr.data_ptr(), col.data_ptr(),
                          values.data_ptr(), lhs.data_ptr(), rhs.data_ptr(), out.data_ptr(), workspace.data_ptr(), need, s1, s2)
    return out
