"""SDDMM through the C ABI against the reference fixtures, the CPU oracle (fp64-accumulated
ground truth), the reference's own kernels where built, and size-independent properties."""
import ctypes
import os

import numpy as np
import pytest
import torch

from oracle import ref
from rode_b200 import capi
from rode_b200 import workloads as W
from tests.helpers import assert_close_to_truth, graph_nodes, run_reference_sddmm, sample_rows_csr, sddmm_abs_scale

pytestmark = pytest.mark.gpu
SEG_FOR_K = {32: 512, 64: 512, 128: 32}   # RoDe_SDDMM/rode_sddmm.py:35-38 (K = 64 follows K = 32)


def _run(A, lhs, rhs, k):
    d = A.to("cuda")
    meta = capi.preprocess(d.row_ptr, d.nnz, SEG_FOR_K[k], 32, 4)
    out = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda())
    torch.cuda.synchronize()
    return d, meta, out


def _check(oracle_cpu, A, lhs, rhs, out, what):
    rp, col, val = A.row_ptr.numpy(), A.col.numpy(), A.val.numpy()
    truth = oracle_cpu.sddmm_f64acc(rp, col, val, lhs.numpy(), rhs.numpy(), threads=oracle_cpu.max_threads())
    return assert_close_to_truth(out.cpu().numpy(), truth,
                                 sddmm_abs_scale(rp, col, val, lhs.numpy(), rhs.numpy()), what)


def test_sddmm_matches_reference_fixtures(golden_dir):
    g = np.load(os.path.join(golden_dir, "sddmm_golden.npz"))
    for case in sorted({k.split("/")[0] for k in g.files}):
        a = {k: g[f"{case}/{k}"] for k in ("row_ptr", "col", "val", "lhs", "rhs", "out")}
        A = W.CSR(len(a["row_ptr"]) - 1, a["rhs"].shape[0], torch.from_numpy(a["row_ptr"]),
                  torch.from_numpy(a["col"]), torch.from_numpy(a["val"]))
        k = a["lhs"].shape[1]
        _, _, out = _run(A, torch.from_numpy(a["lhs"]), torch.from_numpy(a["rhs"]), k)
        # the fixture is the reference's fp32 CPU result; both sides are within the tolerance
        # of the exact value, so compare with twice the scaled floor
        scale = sddmm_abs_scale(a["row_ptr"], a["col"], a["val"], a["lhs"], a["rhs"])
        assert_close_to_truth(out.cpu().numpy(), a["out"].astype(np.float64), 2 * scale, case)


@pytest.mark.parametrize("k", [32, 64, 128])
def test_sddmm_families_against_oracle_and_reference(oracle_cpu, headroom, k):
    fams = {
        "bernoulli": W.bernoulli(),
        "zipf": W.zipf_rows(m=4096, n=4096, cap=4096),
        "stencil": W.stencil27(12),
        "pareto": W.pareto_rows(m=4096, n=8192, cap=3000),
        "rmat": W.rmat(scale=12),
    }
    for name, A in fams.items():
        lhs, rhs = W.dense(A.m, k, seed=5), W.dense(A.n, k, seed=6)
        d, meta, out = _run(A, lhs, rhs, k)
        stats = _check(oracle_cpu, A, lhs, rhs, out, f"{name} k={k}")
        config1 = name == "bernoulli" and k == 32
        if config1:
            headroom("1 Bernoulli 4096^2 SDDMM K=32 (all elements)", "ours", stats)
        assert torch.equal(out, capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda()))
        if ref.available() and k in (32, 128) and meta.m1 > 0 and meta.m2 > 0:
            oref = run_reference_sddmm(d, meta, lhs.cuda(), rhs.cuda())
            stats = _check(oracle_cpu, A, lhs, rhs, oref, f"reference {name} k={k}")
            if config1:
                headroom("1 Bernoulli 4096^2 SDDMM K=32 (all elements)", "reference kernels", stats)


def test_sddmm_edge_cases(oracle_cpu):
    def csr(lens, ncols, seed=0):
        rng = np.random.default_rng(seed)
        lens = np.asarray(lens)
        rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        col = np.concatenate([np.sort(rng.choice(ncols, l, replace=False)) for l in lens] + [np.zeros(0, np.int64)])
        val = rng.uniform(-1, 1, len(col)).astype(np.float32)
        return W.CSR(len(lens), ncols, torch.from_numpy(rp), torch.from_numpy(col.astype(np.int32)),
                     torch.from_numpy(val))

    cases = {
        "empty rows only": csr([0] * 37, 64),
        "single long row": csr([20000], 30000),
        "unaligned long rows": csr([3, 16384, 1, 1025, 2, 513, 0, 0, 545], 20000),
        "block only": csr([32, 64, 512, 1024, 96], 4096),
        "segment edges": csr([511, 512, 513, 1, 543, 544, 545, 31, 32, 33, 0, 1023, 1024, 1025, 63, 64, 65], 2048),
        "one entry": csr([1], 8),
    }
    for name, A in cases.items():
        for k in (32, 64, 128):
            lhs, rhs = W.dense(A.m, k, seed=7), W.dense(A.n, k, seed=8)
            d = A.to("cuda")
            meta = capi.preprocess(d.row_ptr, d.nnz, SEG_FOR_K[k], 32, 4)
            out0 = torch.full((max(A.nnz, 1),), float("nan"), device="cuda")[: A.nnz]
            out = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda(), out=out0)
            if A.nnz:
                _check(oracle_cpu, A, lhs, rhs, out, f"{name} k={k}")   # every entry written exactly once


def test_reference_signature_entry_points(oracle_cpu):
    lib = capi.load()
    A = W.pareto_rows(m=4096, n=8192, cap=3000)
    vp = ctypes.c_void_p
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    for name, k in (("RoDeSDDMM_n32", 32), ("RoDeSDDMM_n64", 64), ("RoDeSDDMM_n128", 128)):
        fn = getattr(lib, capi.CPP_SYMBOLS[name])
        fn.restype = None
        lhs, rhs = W.dense(A.m, k, seed=5), W.dense(A.n, k, seed=6)
        d = A.to("cuda")
        meta = capi.preprocess(d.row_ptr, d.nnz, SEG_FOR_K[k], 32, 4)
        l, r = lhs.cuda(), rhs.cuda()
        out = torch.zeros(A.nnz, device="cuda")
        torch.cuda.synchronize()
        fn(meta.m1, meta.m2, A.n, k, vp(meta.block_r_ind.data_ptr()), vp(meta.residue_r_ind.data_ptr()),
           vp(meta.st_off.data_ptr()), vp(d.row_ptr.data_ptr()), vp(d.col.data_ptr()), vp(d.val.data_ptr()),
           vp(l.data_ptr()), vp(r.data_ptr()), vp(out.data_ptr()), vp(s1.cuda_stream), vp(s2.cuda_stream))
        s1.synchronize()
        s2.synchronize()
        _check(oracle_cpu, A, lhs, rhs, out, name)


@pytest.mark.parametrize("family,k", [("stencil", 64), ("pareto", 32), ("pareto", 128), ("rmat", 64)])
def test_sddmm_full_size_properties(oracle_cpu, headroom, family, k):
    """Full-size matrices: a sample of rows against the oracle, and linearity in lhs."""
    A = {"stencil": lambda: W.stencil27(128, device="cuda"),
         "pareto": lambda: W.pareto_rows(device="cuda"),
         "rmat": lambda: W.rmat(scale=22, device="cuda")}[family]()
    meta = capi.preprocess(A.row_ptr, A.nnz, SEG_FOR_K[k], 32, 4)
    lhs1 = W.dense(A.m, k, device="cuda", seed=5)
    rhs = W.dense(A.n, k, device="cuda", seed=6)
    out1 = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs1, rhs)
    lens = (A.row_ptr[1:] - A.row_ptr[:-1]).long()
    g = torch.Generator(device="cuda").manual_seed(1)
    rows = torch.cat([torch.topk(lens, 8).indices, torch.randint(0, A.m, (4096,), device="cuda", generator=g)]).unique()
    rp, col, val, idx = sample_rows_csr(A, rows)
    lh, rh = lhs1[rows].cpu().numpy(), rhs.cpu().numpy()
    truth = oracle_cpu.sddmm_f64acc(rp, col, val, lh, rh, threads=oracle_cpu.max_threads())
    scale = sddmm_abs_scale(rp, col, val, lh, rh)
    idx_d = torch.from_numpy(idx).cuda()
    what = {"stencil": "3 stencil 128^3", "pareto": "4 Pareto 2^20", "rmat": "R-MAT 22"}[family] + f" SDDMM K={k} (row sample)"
    headroom(what, "ours", assert_close_to_truth(out1[idx_d].cpu().numpy(), truth, scale, f"{family} k={k} sample"))
    # the reference's kernels where they can run (K = 32 or 128, both lists non-empty, 32-bit offsets)
    if ref.available() and k in (32, 128) and meta.m1 > 0 and meta.m2 > 0 and (A.n - 1) * k < 2**29:
        oref = run_reference_sddmm(A, meta, lhs1, rhs)
        headroom(what, "reference kernels",
                 assert_close_to_truth(oref[idx_d].cpu().numpy(), truth, scale, f"{family} k={k} sample, reference"))
        del oref
    lhs2 = W.dense(A.m, k, device="cuda", seed=9)
    out2 = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs2, rhs)
    out3 = capi.sddmm(meta, A.row_ptr, A.col, A.val, 2 * lhs1 - lhs2, rhs)
    assert (out3 - (2 * out1 - out2)).abs().max().item() <= 1e-4


@pytest.mark.parametrize("k", [4, 36, 96, 160, 192, 252, 256])
def test_sddmm_other_widths(oracle_cpu, k):
    """Every K that is a multiple of 4 up to 256 behind the one entry point, on metadata of
    either segment length (the reference serves 32 and 128 only)."""
    A = W.pareto_rows(m=3000, n=5000, cap=2500, seed=13)
    lhs, rhs = W.dense(A.m, k, seed=5), W.dense(A.n, k, seed=6)
    d = A.to("cuda")
    for seg in (512, 32):
        meta = capi.preprocess(d.row_ptr, d.nnz, seg, 32, 4)
        out0 = torch.full((A.nnz,), float("nan"), device="cuda")
        out = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda(), out=out0)
        torch.cuda.synchronize()
        _check(oracle_cpu, A, lhs, rhs, out, f"k={k} seg={seg}")


def test_sddmm_rejects_unsupported_widths():
    A = W.bernoulli(m=64, n=64).to("cuda")
    meta = capi.preprocess(A.row_ptr, A.nnz)
    for k in (0, 6, 260):
        x = torch.zeros((64, max(k, 1)), device="cuda")
        with pytest.raises(capi.RodeError):
            capi.sddmm_raw(meta.m1, meta.m2, 64, k, meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(),
                           meta.st_off.data_ptr(), A.row_ptr.data_ptr(), A.col.data_ptr(), A.val.data_ptr(),
                           x.data_ptr(), x.data_ptr(), x.data_ptr())


@pytest.mark.parametrize("k", [32, 64])
def test_sddmm_row_mode_every_entry(oracle_cpu, k):
    """A residue list long enough for the residue kernel to give its warps 32 rows each, with
    rows of every length from 0 to 31 mixed at random and a ragged last warp: warps whose rows
    are long take the row mode (one lane group per row), the others the stream; every entry of
    the result is checked, and a NaN-filled output shows entries written never or twice."""
    m, n = 520_001, 60_000
    g = torch.Generator().manual_seed(77)
    lens = torch.randint(0, 32, (m,), generator=g)
    lens[torch.rand(m, generator=g) < 0.2] = 0                 # empty rows in between
    dense_part = slice(100_000, 200_000)                       # a stretch of long rows only
    lens[dense_part] = torch.randint(20, 32, (100_000,), generator=g)
    rp = torch.zeros(m + 1, dtype=torch.int64)
    torch.cumsum(lens, 0, out=rp[1:])
    nnz = int(rp[-1])
    # ascending distinct columns per row: a random start plus a stride, modulo nothing (n is large enough)
    row_of = torch.repeat_interleave(torch.arange(m), lens)
    pos = torch.arange(nnz) - rp[:-1][row_of]
    start = torch.randint(0, n - 32 * 40, (m,), generator=g)
    stride = torch.randint(1, 40, (m,), generator=g)
    col = (start[row_of] + pos * stride[row_of]).to(torch.int32)
    val = torch.rand(nnz, generator=g) * 2 - 1
    A = W.CSR(m, n, rp.to(torch.int32), col, val)
    lhs, rhs = W.dense(m, k, seed=5), W.dense(n, k, seed=6)
    d = A.to("cuda")
    meta = capi.preprocess(d.row_ptr, d.nnz, 512, 32, 4)
    assert meta.m2 > 31 * 4 * 24 * 148      # enough rows for 32 per warp on a 148-SM part
    out0 = torch.full((nnz,), float("nan"), device="cuda")
    out = capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda(), out=out0)
    torch.cuda.synchronize()
    _check(oracle_cpu, A, lhs, rhs, out, f"row mode k={k}")


def test_sddmm_calls_on_different_stream_pairs_run_side_by_side():
    """Large block grids run as one resident wave whose warps claim segments from a counter that
    the library keeps per pair of streams: two calls on different pairs, in flight together,
    must not disturb each other, and repeated calls on one pair reuse its counter."""
    A = W.rmat(scale=21, device="cuda")
    meta = capi.preprocess(A.row_ptr, A.nnz, 512, 32, 4)
    assert meta.m1 > 16 * 32 * 148         # enough segments for the block kernel to run as a persistent grid
    k = 64
    lhs, rhs = W.dense(A.m, k, device="cuda", seed=5), W.dense(A.n, k, device="cuda", seed=6)
    want = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs)
    torch.cuda.synchronize()
    pairs = [(torch.cuda.Stream(), torch.cuda.Stream()) for _ in range(3)]
    outs = [torch.full((A.nnz,), float("nan"), device="cuda") for _ in pairs]
    for _ in range(2):                       # second round: every pair uses its counter again
        for (s1, s2), out in zip(pairs, outs):
            out.fill_(float("nan"))
        torch.cuda.synchronize()
        for (s1, s2), out in zip(pairs, outs):
            capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, out=out, stream1=s1, stream2=s2)
        torch.cuda.synchronize()
        for out in outs:
            assert torch.equal(out, want)


@pytest.mark.parametrize("k", [4, 28, 36, 60, 68, 96, 124, 132, 252, 256])
@pytest.mark.parametrize("family", ["power law", "mesh"])    # long segments and streams; the row mode
def test_sddmm_widths_that_leave_lanes_idle(oracle_cpu, family, k):
    A = W.pareto_rows(m=40001, n=3001, mean=20, cap=1400, seed=k) if family == "power law" else W.stencil27(33, seed=k)
    d = A.to("cuda")
    meta = capi.preprocess(d.row_ptr, d.nnz, 512, 32, 4)
    lhs, rhs = W.dense(A.m, k, seed=k), W.dense(A.n, k, seed=k + 1)
    out = torch.full((A.nnz + 2,), float("nan"), device="cuda")
    capi.sddmm(meta, d.row_ptr, d.col, d.val, lhs.cuda(), rhs.cuda(), out=out[1:-1])
    rp, col, val = A.row_ptr.numpy(), A.col.numpy(), A.val.numpy()
    truth = oracle_cpu.sddmm_f64acc(rp, col, val, lhs.numpy(), rhs.numpy(), threads=oracle_cpu.max_threads())
    assert_close_to_truth(out[1:-1].cpu().numpy(), truth, sddmm_abs_scale(rp, col, val, lhs.numpy(), rhs.numpy()),
                          f"{family} k={k}")
    assert bool(torch.isnan(out[0])) and bool(torch.isnan(out[-1]))


def _persistent_grid_case(k):
    """80,000 rows of 40 nonzeros: enough segments for the block kernel to run as a persistent grid."""
    m, n = 80_000, 5_000
    rp = torch.arange(m + 1, dtype=torch.int32, device="cuda") * 40
    col = (torch.arange(m * 40, device="cuda") * 7919 % n).to(torch.int32)
    A = W.CSR(m, n, rp, col, W.dense(m, 40, device="cuda", seed=4).flatten())
    meta = capi.preprocess(A.row_ptr, A.nnz, 512, 32, 4)
    assert meta.m1 > 16 * 32 * 148
    return A, meta, W.dense(m, k, device="cuda", seed=5), W.dense(n, k, device="cuda", seed=6)


@pytest.mark.parametrize("k", [32, 64])
def test_sddmm_graphs_captured_on_one_stream_share_no_counter(k):
    """Two graphs captured on the same stream and replayed side by side on two others: a captured call uses no claim
    counter (its reset would be a memset node), so neither replay can take the other's segments."""
    A, meta, lhs, rhs = _persistent_grid_case(k)
    want = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs)
    outs = [torch.empty_like(A.val) for _ in range(2)]
    nodes = graph_nodes(lambda: capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, out=outs[0]))
    assert nodes and all("sddmm" in name for name in nodes), nodes
    capture, replay = torch.cuda.Stream(), [torch.cuda.Stream() for _ in outs]
    graphs = []
    for out in outs:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=capture):
            capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, out=out)
    for _ in range(4):
        for out in outs:
            out.fill_(float("nan"))
        torch.cuda.synchronize()
        for graph, stream in zip(graphs, replay):
            with torch.cuda.stream(stream):
                graph.replay()
        torch.cuda.synchronize()
        for out in outs:
            assert torch.allclose(out, want, rtol=1e-5, atol=1e-6 * k)
    del graphs


def test_sddmm_threads_that_share_a_stream():
    """Host threads whose calls interleave on one stream (the ctypes calls run without the GIL): the reset of the claim
    counter and the kernel that uses it stay together."""
    import threading

    A, meta, lhs, rhs = _persistent_grid_case(32)
    want = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs)
    outs = [[torch.full_like(A.val, float("nan")) for _ in range(12)] for _ in range(4)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    start = threading.Barrier(len(outs))

    def work(mine):
        start.wait()
        for out in mine:
            capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, out=out, stream1=stream, stream2=stream)

    threads = [threading.Thread(target=work, args=(mine,)) for mine in outs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for mine in outs:
        for out in mine:
            assert torch.equal(out, want)


@pytest.mark.parametrize("k", [96, 100, 128, 132, 256])
@pytest.mark.parametrize("rows", [14_000, 28_000, 31_001, 110_000, 440_001])   # 1, 2, 3 (made 4), 8 and 32 rows per warp on 148 SMs
def test_sddmm_row_mode_of_wide_rows(oracle_cpu, rows, k):
    """The residue rows of K above 64, where a warp's rows go one by one only if they are about equally long: rows of 26,
    rows of 0 to 31, rows that alternate between 31 and 16, and a short stretch, so that both forms and warps just on
    either side of the line occur; every entry is checked in a result filled with NaN."""
    g = torch.Generator().manual_seed(rows)
    lens = torch.full((rows,), 26)
    part = rows // 4
    lens[part: 2 * part] = torch.randint(0, 32, (part,), generator=g)
    lens[2 * part: 3 * part] = torch.where(torch.arange(part) % 2 == 0, 28, 16)
    lens[3 * part: 3 * part + part // 2] = torch.randint(0, 4, (part // 2,), generator=g)
    rp = torch.zeros(rows + 1, dtype=torch.int64)
    torch.cumsum(lens, 0, out=rp[1:])
    nnz, n = int(rp[-1]), 2003
    col = torch.randint(0, n, (nnz,), generator=g).to(torch.int32)
    A = W.CSR(rows, n, rp.to(torch.int32), col, torch.rand(nnz, generator=g) * 2 - 1)
    lhs, rhs = W.dense(rows, k, seed=5), W.dense(n, k, seed=6)
    d = A.to("cuda")
    lhs_d, rhs_d = lhs.cuda(), rhs.cuda()
    for seg in ((32,) if k == 128 else (512,)):
        meta = capi.preprocess(d.row_ptr, d.nnz, seg, 32, 4)
        out = torch.full((nnz + 2,), float("nan"), device="cuda")
        capi.sddmm_raw(0, meta.m2, n, k, meta.block_r_ind.data_ptr(), meta.residue_r_ind.data_ptr(), meta.st_off.data_ptr(),
                       d.row_ptr.data_ptr(), d.col.data_ptr(), d.val.data_ptr(), lhs_d.data_ptr(),
                       rhs_d.data_ptr(), out[1:-1].data_ptr())
        torch.cuda.synchronize()
        # rows of an aligned length of 32 and more belong to the segments, which were left out
        short = lens + (rp[:-1] % 4) < 32
        mine = torch.repeat_interleave(short, lens).numpy()
        truth = oracle_cpu.sddmm_f64acc(A.row_ptr.numpy(), col.numpy(), A.val.numpy(), lhs.numpy(), rhs.numpy(),
                                        threads=oracle_cpu.max_threads())
        got = out[1:-1].cpu().numpy()
        scale = sddmm_abs_scale(A.row_ptr.numpy(), col.numpy(), A.val.numpy(), lhs.numpy(), rhs.numpy())
        assert_close_to_truth(got[mine], truth[mine], scale[mine], f"rows={rows} k={k}")
        assert np.isnan(got[~mine]).all() and bool(torch.isnan(out[0])) and bool(torch.isnan(out[-1]))


@pytest.mark.parametrize("as_int", [False, True])
def test_results_made_for_other_streams(as_int):
    """Results and workspaces that capi makes for calls on streams other than the current one: the zero-fill of an SDDMM
    result comes before the kernels, and memory that such a stream still uses is not handed out again."""
    A = W.zipf_rows(m=60000, n=60000, cap=4096, mean=16, device="cuda")
    meta = capi.preprocess(A.row_ptr, A.nnz)
    lhs, rhs = W.dense(A.m, 64, device="cuda", seed=5), W.dense(A.n, 64, device="cuda", seed=6)
    want, want_c = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs), capi.spmm(meta, A.row_ptr, A.col, A.val, rhs)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    handle = side.cuda_stream if as_int else side
    counts = (meta.m1, meta.m2)
    for _ in range(5):
        with torch.cuda.stream(side):
            torch.cuda._sleep(5_000_000)       # the counts are read behind the kernels, not before
        late = capi.preprocess(A.row_ptr, A.nnz, stream=handle)
        assert (late.m1, late.m2) == counts
        torch.cuda._sleep(20_000_000)          # the current stream is late: a fill on it comes after the kernels unless they wait
        out = capi.sddmm(meta, A.row_ptr, A.col, A.val, lhs, rhs, stream1=handle, stream2=handle)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)      # the side stream is late: its workspace is still to be used
        C = capi.spmm(meta, A.row_ptr, A.col, A.val, rhs, stream1=handle, stream2=handle)
        for size in {capi.spmm_workspace_bytes(meta.m1, 64, 4), C.numel() * 4}:
            for _ in range(3):
                torch.full((size // 4 + 1,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        assert torch.equal(C, want_c)
