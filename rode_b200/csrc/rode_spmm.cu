// RoDe SpMM for sm_100a:  C[M x n] = S * B  with S in CSR + row-decomposition metadata.
//
// Stands in for the reference's block / residue kernels (RoDe_SpMM/RoDeSpmm.cu:197-476 and
// :41-195) and their launcher (:492-529).  The work split follows the reference's metadata
// (block segments, residue rows); how the work is done is new:
//
//  * A dense-row slice of the column tile (8, 16 or 32 vectors of 16 bytes) is covered by a
//    lane group of L lanes with VPL vectors per lane (LDG.128 each): 4 x 2 for 8 vectors (8 x 1 in
//    the block kernel; 4 lanes with one 32-byte load in both where the operands are aligned to 32 bytes), 8 x 2 for 16,
//    32 x 1 for 32.  Two vectors per lane halve the address
//    arithmetic per byte (measured: N = 32 power-law 0.68 -> 0.58 ms, N = 64 R-MAT-21
//    0.99 -> 0.75 ms, N = 64 stencil 0.97 -> 0.75 ms; for 32 vectors no shape beat 32 x 1).
//    A warp holds G = 32/L lane groups.
//  * Gathers are issued in batches of 8 independent LDG.128 per lane; the (column,
//    value) pairs of a chunk of 32 nonzeros are fetched two chunks ahead, stored once into a
//    double-buffered shared-memory tile and read by every lane group as 16-byte broadcast runs
//    (one shuffle per pair element and nonzero costs the SM's load/store data path as much as
//    128 bytes of gathered data).  Bytes in flight per SM = resident warps x 32 x U x 16 B, so the
//    kernels are kept at 64 registers (32 one-warp CTAs per SM, ~131 KB in flight).  Two
//    register buffers per lane (software pipelining) were measured and rejected: 168
//    registers cut the resident warps to 12 and the time went up by 30 %.
//  * spmm_block: one warp per block segment; the G groups take alternate nonzeros and are
//    combined with log2(G) shuffle steps at the end.  The LAST segment of a row also
//    consumes the row's tail (the part shorter than 32 that the reference leaves to its
//    residue kernel), so a row that fits one segment is finished by a single warp and
//    stored with plain vector stores.
//    Grids of a few segments per SM give a segment two or four warps; small products run segments and rows in
//    one launch (spmm_one_launch).
//  * Rows cut into several segments: every segment writes its partial row to a workspace
//    slot (slot = segment index); spmm_fixup, the last grid of the call,
//    sums the slots of each such row in a fixed order (fp64 accumulation) and stores the
//    row.  No floating-point atomics anywhere: results are deterministic.
//  * spmm_rows (L = 32): residue rows that have no block part (aligned length < 32).  A warp
//    takes 32 consecutive residue rows at once: lane j reads the descriptor of row j, so the
//    dependent chain row index -> row pointer -> column -> dense row is paid once per 32
//    rows, not per row.  The nonzeros of the 32 rows form one entry stream that runs through
//    the same batched gather; a row is stored when the stream passes its end.
//    spmm_rows_simple, spmm_rows_simple_staged (L < 32): one lane group per residue row, or per two short ones; spmm_rows_wide: one warp per
//    row, for lists too short to fill the GPU.  All of them also take the rows of the whole matrix in the place of
//    a list, and then store zeros in those without a nonzero.
//    Rows of the list without a nonzero are not touched (the reference stores zeros there,
//    RoDeSpmm.cu:185-194, into a C that its contract already wants zero-filled); rows with a
//    block part are skipped (spmm_block finished them).
//  * CTAs are one warp (four in spmm_rows_wide, whose rows are all shorter than 32, and in small grids): a CTA's
//    slot is held until its slowest warp finishes, and segment lengths differ by more than 10x.
//
// Per nonzero the kernels move 8 B of CSR data and 16*L bytes of the dense operand (from
// L1/L2/HBM depending on reuse); per row 4*n bytes of C.  Dense-row offsets are 64-bit.
#include <climits>
#include <type_traits>

#include "rode_common.cuh"
#include "rode_order.cuh"

namespace rode {
namespace {

// Small CTAs: a CTA's slot is held until its slowest warp is done, and segments differ in
// length by more than 10x, so fewer warps per CTA keep more warps resident on average.
constexpr int kCtaWarps = 1;
constexpr int kCtaThreads = 32 * kCtaWarps;
constexpr int kSmallGridWarps = 4;  // rows (warps) per CTA of spmm_rows_wide

// A lane group: L lanes with VPL vectors of VB bytes each (LDG.128, or the 256-bit loads of sm_100) cover a tile of a
// dense row.  16-byte shapes of the tiles of 128, 256 and 512 bytes:
// (8 x 1 in the block kernel of the 128-byte tile: a load instruction then covers whole 128-byte lines, 4
// rows per warp, where 4 x 2 covers 8 half lines.  R-MAT 23 N = 32 block kernel 2.19 -> 1.20 ms, R-MAT 21
// N = 96 1.43 -> 0.92 ms, Zipf N = 32 -7 %; uniformly random columns lose 3 %: Pareto 2^20 N = 32 0.354 ->
// 0.365 ms.  The per-row residue kernels measured faster with 4 x 2: R-MAT 23 N = 32 0.756 against 1.079 ms.)
template <int VB_, int L_, int VPL_>
struct Shape {
    static constexpr int VB = VB_, L = L_, VPL = VPL_;
};
using Block128 = Shape<16, 8, 1>;
using Rows128 = Shape<16, 4, 2>;
using Tile256 = Shape<16, 8, 2>;
using Tile512 = Shape<16, 32, 1>;  // (its rows: the batched kernel spmm_rows)
// 128-byte tile with one 32-byte load per lane and 4 lanes per dense row, where the operands are aligned to 32 bytes.
// Stencil 128^3 N = 32 0.510 -> 0.401 ms (a load instruction of the per-row kernel covers whole lines of 8 rows instead of
// half lines); the other matrices measure the same as with the 8 x 1 block shape.
using Aligned128 = Shape<32, 4, 1>;
// Claim counters of the persistent kernels, at the end of the workspace: one int per column tile for the block kernel, then
// as many for the rows.
constexpr size_t kCounterBytes = 256;
constexpr int kClaimTiles = 2;
// A grid becomes persistent (one resident wave of so many CTAs per SM, whose warps claim segments or bundles of rows)
// from so many resident waves of work on: with fewer segments per warp the claimed order's tail (one long segment claimed
// last) costs more than the launch gaps it saves (measured: gain from about 20 segments per warp, loss below 10).  Dense
// rows of 1.75 column tiles and more keep one CTA per segment or bundle: such a grid walks its tiles one after the other, and
// the slice of the dense operand that a tile gathers from stays in the L2, where one resident wave over all tiles works
// on all slices at once (ms, persistent / not: Zipf 671,008 rows of mean 40, N = 224 3.53 / 3.12, N = 512 7.91 / 6.56; R-MAT 21
// N = 224 2.40 / 2.29, N = 384 4.74 / 3.88; 1,000,000 rows of 0 to 12 and 100,000 columns, N = 512 1.55 / 0.94).  Below that the
// second tile is the smaller part of the row, and gathering a row's two parts close together pays on graphs (N = 132 and
// 160: Zipf 2.37 / 2.61 and 2.42 / 2.46, R-MAT 21 1.91 / 2.09 and 1.87 / 1.97; N = 192 and 196: Zipf 2.84 / 2.59, Pareto 200,000 of
// mean 60 0.97 / 0.88, R-MAT 20 of 40 per row 2.20 / 2.33, R-MAT 18 of 64 0.71 / 0.75).
constexpr int kPersistentMinWaves = 16;
constexpr int kPersistentCtasPerSm = 32;
template <typename T>
constexpr bool claims_work(int n, unsigned tiles) {  // (fp64, bound by DRAM on twice the bytes, measured 5 % slower with it)
    return sizeof(T) == 4 && tiles <= kClaimTiles && static_cast<long long>(n) * sizeof(T) < 896;
}
// Block grids of at most so many segments per SM give a segment four or two warps, which take its chunks in turn and add
// their rows through shared memory: the time of such a grid is the chain of batches of its longest segment, beyond that
// it is its throughput.  us, one warp with 8 rows in flight / one warp with a whole chunk in flight (163 registers, which
// these two forms replace) / two warps / four: R-MAT 14 N = 128 (1508 segments) 27 / 21 / 19 / 17, R-MAT 15 (1981) 31 / 25 / 22 /
// 21, Zipf 50000 (2800) 37 / 39 / 33 / 35, Pareto 2^14 (2949) 35 / 31 / 29 / 28, Zipf 65536 (3706) 41 / 45 / 41 / 42, Bernoulli
// 4096^2 (3911) 14.5 / 16.5 / 15 / 17.
constexpr int kSplit4WarpsPerSm = 16;
constexpr int kSplit2WarpsPerSm = 22;
// What a call knows of the rows that the residue kernels work on, those of fewer than 32 nonzeros: the number of nonzeros of
// the matrix (not always, nnz < 0 then) and of segments, which hold at most 543 each.  Their mean is therefore
// at least (nnz - 543 m1) / rows, and it is no larger than that of all rows.  Matrices with heavier tails than the
// lower bound can tell apart (Zipf of mean 40: short rows of 2.0; Pareto of mean 32: 11.8) are known by neither.
constexpr bool rows_hold(long long nnz, long long m1, long long rows, int mean) {  // at least so many on average, surely
    return nnz >= 0 && nnz - 543 * m1 >= mean * rows;
}
// Two rows per lane group in spmm_rows_simple.  us, one / two: rows of 1.6 (Zipf 671,008 N = 64) 353 / 341, of 5.2 (R-MAT 21)
// 752 / 704, of 7 (2 to 12) 72 / 70, of 27 (stencil) 700 / 724.  In the 128-byte tile long rows lose more: of 9.8 (Pareto
// 300,007 N = 32) 91.3 / 92.5, of 12 and 16 (Bernoulli 30,000) 8.3 / 10.3 and 11.4 / 13.2, of 19.5 (15 to 24) 62 / 66, of 27 401 / 444;
// in the wider ones not (of 16 N = 64 16.1 / 15.3, fp64 N = 32 16.0 / 14.4).
constexpr bool short_rows(long long nnz, long long m1, long long rows, int tile_bytes) {
    return nnz >= 0 && nnz < 20 * rows && !(tile_bytes == 128 && rows_hold(nnz, m1, rows, 10));
}
// 16-byte units a lane keeps in flight per batch (dense rows per batch = this * 16 / bytes per load / VPL).
constexpr int kLoadsInFlight = 8;

// ---------------------------------------------------------------------------------------
// One warp per block segment, or S warps (a CTA) that take its chunks in turn; grid.y walks the column tiles of
// L * VPL vectors.  U = dense rows per batch: 8 loads of 16 bytes per lane, with which 64 registers keep 32 warps
// per SM resident.
//
// kOrdered: the segments as `order` lists them, whose entries hold what the warp needs of the row pointer too.
//
// kRagged: the width is not a multiple of the tile; the last tile's lanes beyond the row's end neither
// load nor store (widths the reference's tiles do not serve: any multiple of 4 columns).
template <typename T, int VB, int L, int VPL, int U, int W, int S, bool kHints, bool kClaim, bool kRagged, bool kOrdered = false>
__global__ void __launch_bounds__(32 * W, 32 / W)
spmm_block(int m1, int n, const T *__restrict__ values, const int *__restrict__ column_indices,
           const int *__restrict__ row_offsets, const int *__restrict__ block_r_ind,
           const int *__restrict__ st_off, const T *__restrict__ B, T *__restrict__ C, T *__restrict__ partial,
           const unsigned *__restrict__ hot, int hot_flag_word, int *__restrict__ next_segment,
           const WholeSegment *__restrict__ order) {
    using V = typename VecB<T, VB>::type;
    constexpr int kLen = VecB<T, VB>::kLen;
    constexpr int G = 32 / L;             // lane groups, each takes every G-th nonzero
    constexpr int kSteps = 32 / G;        // nonzeros per group per 32-nonzero chunk
    constexpr int NB = (kSteps + U - 1) / U;
    constexpr unsigned kFull = 0xffffffffu;
    // (the first grid of the call, or behind the kernels that make the list)
    int item = after_chain(S == 1 ? blockIdx.x * W + (threadIdx.x >> 5) : blockIdx.x);
    chain_begin();
    static_assert(W % S == 0 && (S == 1 || (W == S && !kClaim)), "a CTA per split segment");
    const int part = S == 1 ? 0 : threadIdx.x >> 5;  // this warp takes every S-th chunk of its segment
    const int lane = threadIdx.x & 31;
    const int g = lane / L, l = lane % L;
    // Chunk staging (two buffers, so one __syncwarp per chunk orders both the reads after the
    // writes and the next-but-one chunk's writes after these reads).  The pair of position t
    // sits at (t % G) * kSteps + t / G: the run of a lane group is contiguous.
    static_assert(kSteps % U == 0 && U % 4 == 0, "whole batches, read as runs of four");
    __shared__ __align__(16) int s_col[W][2][32];
    __shared__ __align__(16) T s_val[W][2][32];
    const int warp_in_cta = threadIdx.x >> 5;
    const int stage_slot = (lane % G) * kSteps + lane / G;
    int stage_buf = 0;
    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const unsigned row_bytes = static_cast<unsigned>(n) * static_cast<unsigned>(sizeof(T));  // n < 2^21 elements
    const size_t col_vec = static_cast<size_t>(blockIdx.y) * L * VPL + l;  // + v * L for vector v
    const V *b_lane = reinterpret_cast<const V *>(B) + col_vec;
    auto inside = [&](int v) { return !kRagged || col_vec + v * L < row_vecs; };
    GatherPolicy policy = {};
    // the word after the bitmap is the library's verdict on this matrix (0: marks would not help)
    if constexpr (kHints) policy = make_gather_policy(__ldg(hot + hot_flag_word) != 0u);

    // Persistent form (next_segment != null, a grid of one resident wave): a warp starts with the
    // segment of its own index and then claims further ones from a counter per column tile, so no
    // warp slot waits for a new CTA to be launched into it (one-warp CTAs of a few microseconds
    // each left a fifth of the slots empty at any time).  The claim is issued before the segment's
    // work and read after it, so its latency is hidden.  Otherwise one segment per warp.
    while (item < m1) {
    int claimed = INT_MAX;
    if constexpr (kClaim) {
        if (next_segment != nullptr && lane == 0)
            claimed = static_cast<int>(gridDim.x) * W + atomicAdd(next_segment + blockIdx.y, 1);
    }
    int seg, row, seg_off, end;
    bool whole_row;
    if constexpr (kOrdered) {
        const int4 e = __ldcg(reinterpret_cast<const int4 *>(order) + item);
        const WholeSegment w = {e.x, e.y, e.z, e.w};
        seg = w.number();
        row = w.row;
        seg_off = w.off;
        end = w.end;
        whole_row = w.whole_row();
    } else {
        seg = item;
        row = __ldg(block_r_ind + seg);
        seg_off = __ldg(st_off + seg);
        const int next = (seg + 1 < m1) ? __ldg(st_off + seg + 1) : INT_MAX;
        const int row_begin = __ldg(row_offsets + row);
        const int row_end = __ldg(row_offsets + row + 1);
        end = min(row_end, next);
        whole_row = (seg_off == row_begin) && (next >= row_end);
    }
    const int off = seg_off + part * 32;

    // (column, value) of this lane's nonzero in the current and in the next chunk
    int c_cur = 0, c_nxt = 0;
    T v_cur = T(0), v_nxt = T(0);
    if (off + lane < end) {
        c_cur = ld_stream(column_indices + off + lane);
        v_cur = ld_stream(values + off + lane);
    }
    if (off + 32 * S + lane < end) {
        c_nxt = ld_stream(column_indices + off + 32 * S + lane);
        v_nxt = ld_stream(values + off + 32 * S + lane);
    }
    // With popularity hints a column index carries its mark in bit 31.  The bitmap word of a
    // column is fetched one chunk after the column itself (which has arrived by then) and one
    // chunk before the column is used, so the lookup adds no exposed latency after the first.
    if constexpr (kHints) c_cur = tag_hot(c_cur, hot_word(hot, c_cur));

    V acc[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) acc[v] = vzero(static_cast<V *>(nullptr));
    for (int base = off; base < end; base += 32 * S) {
        const int cnt = min(32, end - base);
        int c_pre = 0;
        T v_pre = T(0);
        if (base + 64 * S + lane < end) {  // pairs of the chunk after next
            c_pre = ld_stream(column_indices + base + 64 * S + lane);
            v_pre = ld_stream(values + base + 64 * S + lane);
        }
        unsigned w_nxt = 0;
        if constexpr (kHints) w_nxt = hot_word(hot, c_nxt);
        s_col[warp_in_cta][stage_buf][stage_slot] = c_cur;
        s_val[warp_in_cta][stage_buf][stage_slot] = v_cur;
        __syncwarp();
        // One chunk of the batched gather.  A full chunk (every chunk of a segment but its last) can take
        // a form without bounds: no predicate per gather and no zero-fill of the row buffers (ncu counted
        // 23 warp instructions per gathered row in the predicated form: 4 FMA, 1 load, the rest address,
        // policy, predicate and zero-fill work).
        auto chunk = [&](auto full_tag) {
            constexpr bool kFullChunk = decltype(full_tag)::value;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                if constexpr (!kFullChunk) {
                    if (b * U * G >= cnt) break;  // warp-uniform
                }
                V buf[U][VPL];
                T vv[U];
                int cc[U];
                ld_shared_run<U>(&s_col[warp_in_cta][stage_buf][g * kSteps + b * U], cc);
                ld_shared_run<U>(&s_val[warp_in_cta][stage_buf][g * kSteps + b * U], vv);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int t = (b * U + u) * G + g;  // position inside the chunk
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        if constexpr (kFullChunk && !kRagged) {
                            buf[u][v] = gather<kHints>(b_lane + v * L, cc[u], row_bytes, policy);
                        } else {
                            buf[u][v] = vzero(static_cast<V *>(nullptr));
                            if ((kFullChunk || t < cnt) && inside(v))
                                buf[u][v] = gather<kHints>(b_lane + v * L, cc[u], row_bytes, policy);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int v = 0; v < VPL; ++v) vfma(acc[v], vv[u], buf[u][v]);
            }
        };
        // (only the 512-byte tile of large grids: R-MAT 21 N = 128 block kernel 0.818 -> 0.787 ms, R-MAT 23
        // step 4.76 -> 4.62 ms; the narrower shapes measured 1-2 % slower with it)
        if (L == 32 && cnt == 32)
            chunk(std::true_type{});
        else
            chunk(std::false_type{});
        c_cur = kHints ? tag_hot(c_nxt, w_nxt) : c_nxt;
        v_cur = v_nxt;
        c_nxt = c_pre;
        v_nxt = v_pre;
        stage_buf ^= 1;
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v)
#pragma unroll
        for (int w = L; w < 32; w <<= 1) vadd(acc[v], vshfl_xor(kFull, acc[v], w));

    if constexpr (S > 1) {  // the parts are added in order
        __shared__ __align__(32) V s_part[S - 1][L * VPL];
        if (part > 0 && g == 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) s_part[part - 1][l + v * L] = acc[v];
        }
        __syncthreads();
        if (part > 0) return;
        if (g == 0) {
#pragma unroll
            for (int w = 0; w < S - 1; ++w)
#pragma unroll
                for (int v = 0; v < VPL; ++v) vadd(acc[v], s_part[w][l + v * L]);
        }
    }
    if (g == 0) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            if (!inside(v)) continue;
            if (whole_row)
                st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row) * row_vecs + col_vec + v * L, acc[v]);
            else
                reinterpret_cast<V *>(partial)[static_cast<size_t>(seg) * row_vecs + col_vec + v * L] = acc[v];
        }
    }
    item = kClaim ? __shfl_sync(kFull, claimed, 0) : INT_MAX;
    }  // segments of this warp
}

// ---------------------------------------------------------------------------------------
// Segments and rows of a small matrix in one launch: its kernels take a few microseconds each, less than the
// host needs to launch them.  A CTA of four warps takes four segments, far apart in the list (neighbours are
// often pieces of one long row), and splits their chunks of 32 nonzeros evenly over the warps, whatever the
// segments' lengths; a warp writes its partial row of every segment it touched to shared memory, and warp s adds
// those of segment s in a fixed order.  The CTAs behind the segments take the rows without a block part (list or
// all rows, as in the residue kernels), a warp per row: fewer than 32 nonzeros, so one chunk.
// SpMM calls through the C ABI, back to back, us: Bernoulli 4096^2 N = 32 15.3 -> 11.9, 2000^2 11.3 -> 8.2, R-MAT 12 11.4
// -> 8.9.  As the kernel of larger grids it is slower than one warp per segment with the whole chunk in flight
// (Zipf 65536 N = 128 45 -> 51 us, R-MAT 19 as long as the persistent grids' threshold 262 -> 306).
constexpr int kOneLaunchWarps = 4;
template <typename T, int VB, int L, int VPL, int U, bool kRagged>
__global__ void __launch_bounds__(32 * kOneLaunchWarps, 5)  // 96 registers
spmm_one_launch(int m1, int seg_ctas, int rows, int n, const T *__restrict__ values, const int *__restrict__ column_indices,
                const int *__restrict__ row_offsets, const int *__restrict__ block_r_ind, const int *__restrict__ st_off,
                const int *__restrict__ residue_r_ind, const T *__restrict__ B, T *__restrict__ C, T *__restrict__ partial) {
    using V = typename VecB<T, VB>::type;
    constexpr int kLen = VecB<T, VB>::kLen;
    constexpr int W = kOneLaunchWarps;
    constexpr int G = 32 / L;   // lane groups, each takes every G-th nonzero of a chunk
    constexpr int NB = L / U;   // batches per chunk
    static_assert(L % U == 0, "a chunk is a whole number of batches");
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int kAlign = 4;    // vec_len of the preprocessing
    constexpr int kBlockK = 32;  // k_block of the preprocessing
    __shared__ __align__(16) int s_col[W][2][32];
    __shared__ __align__(16) T s_val[W][2][32];
    __shared__ __align__(32) V s_acc[W][W][L * VPL];  // [warp][segment]
    const int cta = after_chain(blockIdx.x);
    chain_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane / L, l = lane % L;
    const int stage_slot = (lane % G) * L + lane / G;
    int stage_buf = 0;
    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const unsigned row_bytes = static_cast<unsigned>(n) * static_cast<unsigned>(sizeof(T));  // n < 2^21 elements
    const size_t tile_vec = static_cast<size_t>(blockIdx.y) * L * VPL;
    const V *b_lane = reinterpret_cast<const V *>(B) + tile_vec + l;
    auto inside = [&](int v) { return !kRagged || tile_vec + l + v * L < row_vecs; };
    V acc[VPL];
    auto clear = [&]() {
#pragma unroll
        for (int v = 0; v < VPL; ++v) acc[v] = vzero(static_cast<V *>(nullptr));
    };
    // one chunk: lane t holds nonzero t < cnt
    auto chunk = [&](int c, T val, int cnt) {
        s_col[warp][stage_buf][stage_slot] = c;
        s_val[warp][stage_buf][stage_slot] = val;
        __syncwarp();
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if (b * U * G >= cnt) break;  // warp-uniform
            V buf[U][VPL];
            T vv[U];
            int cc[U];
            ld_shared_run<U>(&s_col[warp][stage_buf][g * L + b * U], cc);
            ld_shared_run<U>(&s_val[warp][stage_buf][g * L + b * U], vv);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    buf[u][v] = vzero(static_cast<V *>(nullptr));
                    if ((b * U + u) * G + g < cnt && inside(v))
                        buf[u][v] = ld_dense(dense_row(b_lane + v * L, static_cast<unsigned>(cc[u]), row_bytes));
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < VPL; ++v) vfma(acc[v], vv[u], buf[u][v]);
        }
        stage_buf ^= 1;
    };
    auto add_groups = [&]() {
#pragma unroll
        for (int v = 0; v < VPL; ++v)
#pragma unroll
            for (int w = L; w < 32; w <<= 1) vadd(acc[v], vshfl_xor(kFull, acc[v], w));
    };

    if (cta >= seg_ctas) {  // ---- a row per warp -----------------------------------
        const int item = (cta - seg_ctas) * W + warp;
        if (item >= rows) return;
        const int row = residue_r_ind != nullptr ? __ldg(residue_r_ind + item) : item;
        const int begin = __ldg(row_offsets + row), end = __ldg(row_offsets + row + 1);
        // aligned length >= k_block: a block part exists and its last segment took the tail; list form, no
        // nonzero: the row stays as the caller zero-filled it
        if (end - begin + (begin % kAlign) >= kBlockK || (end == begin && residue_r_ind != nullptr)) return;
        int c = 0;
        T val = T(0);
        if (begin + lane < end) {
            c = ld_stream(column_indices + begin + lane);
            val = ld_stream(values + begin + lane);
        }
        clear();
        chunk(c, val, end - begin);
        add_groups();
        if (g == 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v)
                if (inside(v))
                    st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row) * row_vecs + tile_vec + l + v * L, acc[v]);
        }
        return;
    }

    // ---- four segments, far apart: lane j < W of every warp holds segment j ---------------------------------
    const int my_seg = cta + lane * seg_ctas;
    int row = 0, off = 0, end = 0;
    bool whole = false;
    if (lane < W && my_seg < m1) {
        row = __ldg(block_r_ind + my_seg);
        off = __ldg(st_off + my_seg);
        const int next = (my_seg + 1 < m1) ? __ldg(st_off + my_seg + 1) : INT_MAX;
        const int row_begin = __ldg(row_offsets + row), row_end = __ldg(row_offsets + row + 1);
        end = min(row_end, next);
        whole = off == row_begin && next >= row_end;
    }
    const int chunks = (end - off + 31) / 32;
    int incl = chunks;  // prefix sum over the segments
#pragma unroll
    for (int d = 1; d < W; d <<= 1) {
        const int up = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += up;
    }
    const int total = __shfl_sync(kFull, incl, W - 1);
    const int per = (total + W - 1) / W;
    const int q_end = min((warp + 1) * per, total);
    struct Chunk {
        int seg, base, end;
    };
    auto locate = [&](int q) {  // chunk q of the CTA
        Chunk k;
        k.seg = min(__popc(__ballot_sync(kFull, lane < W && incl <= q)), W - 1);
        k.base = __shfl_sync(kFull, off - (incl - chunks) * 32, k.seg) + q * 32;
        const int seg_end = __shfl_sync(kFull, end, k.seg);
        k.end = q < q_end ? seg_end : 0;
        return k;
    };
    auto fetch = [&](const Chunk &k, int &c, T &val) {
        c = 0;
        val = T(0);
        if (k.base + lane < k.end) {
            c = ld_stream(column_indices + k.base + lane);
            val = ld_stream(values + k.base + lane);
        }
    };
    auto flush = [&](int s) {
        add_groups();
        if (g == 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v) s_acc[warp][s][l + v * L] = acc[v];
        }
        clear();
    };
    int q = warp * per;
    Chunk cur = locate(q), nxt = locate(q + 1);
    int c_cur, c_nxt;
    T v_cur, v_nxt;
    fetch(cur, c_cur, v_cur);
    fetch(nxt, c_nxt, v_nxt);
    clear();
    for (; q < q_end; ++q) {
        const Chunk pre = locate(q + 2);
        int c_pre;
        T v_pre;
        fetch(pre, c_pre, v_pre);
        chunk(c_cur, v_cur, min(32, cur.end - cur.base));
        if (q + 1 == q_end || nxt.seg != cur.seg) flush(cur.seg);  // warp-uniform
        cur = nxt;
        nxt = pre;
        c_cur = c_nxt;
        v_cur = v_nxt;
        c_nxt = c_pre;
        v_nxt = v_pre;
    }
    __syncthreads();
    // warp s adds the partial rows of segment s, in the order of the warps
    const int seg = cta + warp * seg_ctas;
    if (seg >= m1) return;
    const int first = __shfl_sync(kFull, incl - chunks, warp) / per, last = (__shfl_sync(kFull, incl, warp) - 1) / per;
    const int out_row = __shfl_sync(kFull, row, warp);
    const bool out_whole = __shfl_sync(kFull, static_cast<int>(whole), warp) != 0;
    if (lane < L * VPL && (!kRagged || tile_vec + lane < row_vecs)) {
        V sum = s_acc[first][warp][lane];
        for (int w = first + 1; w <= last; ++w) vadd(sum, s_acc[w][warp][lane]);
        if (out_whole)
            st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(out_row) * row_vecs + tile_vec + lane, sum);
        else
            reinterpret_cast<V *>(partial)[static_cast<size_t>(seg) * row_vecs + tile_vec + lane] = sum;
    }
}

// ---------------------------------------------------------------------------------------
// Sums the workspace slots of every row that was cut into several segments, with fp64
// accumulation and in an order that the code fixes, so the result is deterministic.
//
// What bounds it: latency, at the very end of the call (its time is not hidden behind anything).  A CTA
// looks at up to kFixupThreads consecutive segments, one per thread, and lists the rows that begin among
// them and were cut; its warps then take the listed rows one each, eight slots of 16 bytes per lane in
// flight, and rows of more than kFixupWideSlots slots are taken by all warps together.  (One warp for 32
// segments, which added its rows one after the other with 4-byte loads, took 7 us after the block grid's
// end on the Zipf matrix, 25 us on Pareto 2^20 and 74 to 140 us on R-MAT scale 23, whose longest row has 470
// slots.)
constexpr int kFixupThreads = 256;
constexpr int kFixupWarps = kFixupThreads / 32;
constexpr int kFixupUnroll = 8;      // workspace slots in flight per lane
constexpr int kFixupWideSlots = 24;  // rows with more slots are summed by the whole CTA

// Sum over the slots s = s0, s0 + step, ... < cnt of vector x of a split row, `row_slots` = its first slot.
template <typename T>
__device__ __forceinline__ void fixup_sum(const typename Vec16<T>::type *__restrict__ row_slots, size_t row_vecs, int x,
                                          int s0, int step, int cnt, double (&acc)[Vec16<T>::kLen]) {
    using V = typename Vec16<T>::type;
#pragma unroll
    for (int j = 0; j < Vec16<T>::kLen; ++j) acc[j] = 0.0;
    for (int s = s0; s < cnt; s += step * kFixupUnroll) {
        V v[kFixupUnroll];
#pragma unroll
        for (int u = 0; u < kFixupUnroll; ++u) {
            v[u] = vzero(static_cast<V *>(nullptr));
            if (s + u * step < cnt) v[u] = __ldcg(row_slots + static_cast<size_t>(s + u * step) * row_vecs + x);
        }
#pragma unroll
        for (int u = 0; u < kFixupUnroll; ++u) {
            __align__(16) T e[Vec16<T>::kLen];
            *reinterpret_cast<V *>(e) = v[u];
#pragma unroll
            for (int j = 0; j < Vec16<T>::kLen; ++j) acc[j] += static_cast<double>(e[j]);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kFixupThreads)
spmm_fixup(int m1, int segs_per_cta, int n, const int *__restrict__ row_offsets, const int *__restrict__ block_r_ind,
           const int *__restrict__ st_off, const T *__restrict__ partial, T *__restrict__ C) {
    using V = typename Vec16<T>::type;
    constexpr int kLen = Vec16<T>::kLen;
    constexpr unsigned kFull = 0xffffffffu;
    // split rows that begin in this CTA's range: narrow ones from the front, wide ones from the back
    __shared__ int s_row[kFixupThreads], s_first[kFixupThreads], s_cnt[kFixupThreads];
    __shared__ int n_narrow, n_wide;
    __shared__ double s_part[kFixupWarps][32][kLen];
    chain_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) n_narrow = n_wide = 0;
    __syncthreads();
    const int seg = blockIdx.x * segs_per_cta + threadIdx.x;
    if (static_cast<int>(threadIdx.x) < segs_per_cta && seg < m1) {
        const int row = __ldg(block_r_ind + seg);
        const int off = __ldg(st_off + seg);
        const int next = (seg + 1 < m1) ? __ldg(st_off + seg + 1) : INT_MAX;
        const int row_begin = __ldg(row_offsets + row);
        const int row_end = __ldg(row_offsets + row + 1);
        if ((off == row_begin) && (next < row_end)) {
            // number of segments of the row = pieces of (next - aligned start) nonzeros
            const int aligned = row_begin - row_begin % 4;
            const int piece = next - aligned;
            int count = (row_end - aligned + piece - 1) / piece;
            // the last piece is a segment only if it is >= 32 long; otherwise it was a
            // residue tail that the previous segment consumed
            if (row_end - aligned - (count - 1) * piece < 32) --count;
            const int slot = count > kFixupWideSlots ? kFixupThreads - 1 - atomicAdd(&n_wide, 1) : atomicAdd(&n_narrow, 1);
            s_row[slot] = row;
            s_first[slot] = seg;
            s_cnt[slot] = count;
        }
    }
    __syncthreads();
    const int narrow = n_narrow, wide = n_wide;
    if (narrow + wide == 0) {
        // No split row begins among these segments: nothing to read from the workspace.  The first
        // CTA still waits for the grids before this one, so that this grid as a whole cannot complete
        // before spmm_block has completed and flushed its stores: whatever the caller enqueues
        // on the stream afterwards (an event, a copy of C, the next kernel) is then ordered
        // after the block grid through this grid, as with a plain launch.
        if (blockIdx.x == 0) chain_wait();
        return;
    }
    // Everything above read only the caller's metadata; the workspace is written by the
    // preceding spmm_block grid: wait for it (no-op when launched without the attribute).
    const T *const finished = after_chain(partial);

    // `width` lanes cover a row of up to 32 vectors; narrower rows leave 32 / width groups of lanes that
    // take alternate slots and are combined by shuffles.
    const int row_vecs = n / kLen;
    int width = 1;
    while (width < row_vecs && width < 32) width <<= 1;
    const int groups = 32 / width;
    const int g = lane / width, l = lane % width;
    auto combine_groups = [&](double (&acc)[kLen]) {
        for (int w = width; w < 32; w <<= 1)
#pragma unroll
            for (int j = 0; j < kLen; ++j) acc[j] += __shfl_xor_sync(kFull, acc[j], w);
    };
    auto store = [&](int row, int x, const double (&acc)[kLen]) {
        __align__(16) T e[kLen];
#pragma unroll
        for (int j = 0; j < kLen; ++j) e[j] = static_cast<T>(acc[j]);
        st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row) * row_vecs + x, *reinterpret_cast<const V *>(e));
    };
    for (int i = warp; i < narrow; i += kFixupWarps) {
        const V *slots = reinterpret_cast<const V *>(finished) + static_cast<size_t>(s_first[i]) * row_vecs;
        const int row = s_row[i], cnt = s_cnt[i];
        for (int x0 = 0; x0 < row_vecs; x0 += 32) {
            const int x = x0 + l;
            double acc[kLen];
            fixup_sum<T>(slots, row_vecs, x, x < row_vecs ? g : cnt, groups, cnt, acc);
            combine_groups(acc);
            if (g == 0 && x < row_vecs) store(row, x, acc);
        }
    }
    for (int i = 0; i < wide; ++i) {
        const int at = kFixupThreads - 1 - i;
        const V *slots = reinterpret_cast<const V *>(finished) + static_cast<size_t>(s_first[at]) * row_vecs;
        const int row = s_row[at], cnt = s_cnt[at];
        for (int x0 = 0; x0 < row_vecs; x0 += 32) {
            const int x = x0 + l;
            double acc[kLen];
            fixup_sum<T>(slots, row_vecs, x, x < row_vecs ? warp * groups + g : cnt, kFixupWarps * groups, cnt, acc);
            combine_groups(acc);
#pragma unroll
            for (int j = 0; j < kLen; ++j) s_part[warp][lane][j] = acc[j];
            __syncthreads();
            if (warp == 0 && g == 0 && x < row_vecs) {
                for (int w = 1; w < kFixupWarps; ++w)
#pragma unroll
                    for (int j = 0; j < kLen; ++j) acc[j] += s_part[w][lane][j];
                store(row, x, acc);
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------------------
// Rows without a block part: the entries of residue_r_ind, or, where that is null, all rows of the matrix
// (n_items = their number; rows with a block part are skipped, rows without a nonzero stored as zeros).
// One lane group per L consecutive entries; grid.y walks the column tiles.
template <typename T, int L, bool kRagged>
__global__ void __launch_bounds__(kCtaThreads, (sizeof(T) == 4 ? 32 : 16) / kCtaWarps)  // fp32: 64 registers
spmm_rows(int m2, int rows_per_group, int n, const T *__restrict__ values,
          const int *__restrict__ column_indices, const int *__restrict__ row_offsets,
          const int *__restrict__ residue_r_ind, const T *__restrict__ B, T *__restrict__ C,
          int *__restrict__ next_group, bool first) {
    using V = typename Vec16<T>::type;
    constexpr int kLen = Vec16<T>::kLen;
    constexpr int U = (kLoadsInFlight < L) ? kLoadsInFlight : L;  // rows per batch
    constexpr int NB = (L + U - 1) / U;  // batches per L-nonzero chunk
    constexpr int kAlign = 4;            // vec_len of the preprocessing
    constexpr int kBlockK = 32;          // k_block of the preprocessing
    const int lane = threadIdx.x & 31;
    const int l = lane % L;
    const unsigned gmask = group_mask<L>(lane);
    const int gshift = lane & ~(L - 1);
    // chunk staging in shared memory as in spmm_block (one region of L pairs per lane group)
    static_assert(L % U == 0 && U % 4 == 0, "whole batches, read as runs of four");
    __shared__ __align__(16) int s_col[2][kCtaThreads];
    __shared__ __align__(16) T s_val[2][kCtaThreads];
    const int stage_base = (threadIdx.x / L) * L;  // first slot of this group's region
    int stage_buf = 0;
    // Persistent form (next_group != null, a grid of one resident wave): a lane group starts with
    // the bundle of rows of its own index and claims further bundles from a counter per column
    // tile; the claim is issued before the bundle's work and read after it.
    const long long n_groups = (static_cast<long long>(m2) + rows_per_group - 1) / rows_per_group;
    const unsigned cta = after_chain_if(first, blockIdx.x);
    long long group = (static_cast<long long>(cta) * kCtaThreads + threadIdx.x) / L;
    while (group < n_groups) {
    int claimed = INT_MAX;
    constexpr bool kClaim = sizeof(T) == 4;  // fp64: 12 more registers for it cost more than it gains
    if constexpr (kClaim) {
        if (next_group != nullptr && l == 0)
            claimed = static_cast<int>(gridDim.x) * (kCtaThreads / L) + atomicAdd(next_group + blockIdx.y, 1);
    }
    [&]() {
    const int item0 = static_cast<int>(group * rows_per_group);

    // ---- descriptors: lane j of the group owns residue row item0 + j -----------------------
    int row = 0, begin = 0, len = 0;
    bool empty = false;  // all-rows form: a row of zeros
    if (l < rows_per_group && item0 + l < m2) {
        row = residue_r_ind != nullptr ? __ldg(residue_r_ind + item0 + l) : item0 + l;
        begin = __ldg(row_offsets + row);
        const int end = __ldg(row_offsets + row + 1);
        // aligned length >= k_block: a block part exists and its last segment took the tail
        if (end - begin + (begin % kAlign) < kBlockK) len = end - begin;
        empty = end == begin && residue_r_ind == nullptr;
    }
    int start = len;  // exclusive prefix sum of len inside the group
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
        const int up = __shfl_up_sync(gmask, start, d, L);
        if (l >= d) start += up;
    }
    const int total = __shfl_sync(gmask, start, L - 1, L);
    start -= len;

    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const unsigned row_bytes = static_cast<unsigned>(n) * static_cast<unsigned>(sizeof(T));  // n < 2^21 elements
    const size_t col_vec = static_cast<size_t>(blockIdx.y) * L + l;
    const V *b_lane = reinterpret_cast<const V *>(B) + col_vec;
    V *c_lane = reinterpret_cast<V *>(C) + col_vec;
    const bool inside = !kRagged || col_vec < row_vecs;  // ragged widths: lanes beyond the row's end idle

    // Rows of the list without a nonzero are left alone: C arrives zero-filled (the contract of
    // the reference's entry points).  In the all-rows form C arrives with any contents, and the rows
    // without a nonzero, which are in no list when they start at a multiple of four, are stored here.
    for (unsigned zeros = (__ballot_sync(gmask, empty) & gmask) >> gshift; zeros != 0; zeros &= zeros - 1) {
        const int r = item0 + __ffs(zeros) - 1;
        if (inside) st_stream(c_lane + static_cast<size_t>(r) * row_vecs, vzero(static_cast<V *>(nullptr)));
    }
    unsigned todo = (__ballot_sync(gmask, len > 0) & gmask) >> gshift;  // rows with nonzeros, in order
    if (todo == 0) return;

    // ---- entry stream: position p -> nonzero index -------------------------------------------------
    auto fetch = [&](int p, int &c, T &v) {  // all lanes of the group call
        int lo = 0;
#pragma unroll
        for (int step = L / 2; step >= 1; step >>= 1) {
            const int s = __shfl_sync(gmask, start, lo + step, L);
            if (s <= p) lo += step;
        }
        const int b0 = __shfl_sync(gmask, begin, lo, L);
        const int s0 = __shfl_sync(gmask, start, lo, L);
        c = 0;
        v = T(0);
        if (p < total) {
            c = ld_stream(column_indices + b0 + (p - s0));
            v = ld_stream(values + b0 + (p - s0));
        }
    };
    int c_cur, c_nxt;
    T v_cur, v_nxt;
    fetch(l, c_cur, v_cur);
    fetch(L + l, c_nxt, v_nxt);

    // ---- consumer state: the row being accumulated -------------------------------------------------
    int cur = __ffs(todo) - 1;
    todo &= todo - 1;
    int cur_row = __shfl_sync(gmask, row, cur, L);
    int cur_end = __shfl_sync(gmask, start, cur, L) + __shfl_sync(gmask, len, cur, L);
    int pos = 0;
    V acc = vzero(static_cast<V *>(nullptr));

    for (int base = 0; base < total; base += L) {
        const int cnt = min(L, total - base);
        int c_pre;
        T v_pre;
        fetch(base + 2 * L + l, c_pre, v_pre);
        s_col[stage_buf][stage_base + l] = c_cur;
        s_val[stage_buf][stage_base + l] = v_cur;
        __syncwarp(gmask);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if (b * U >= cnt) break;  // group-uniform
            V buf[U];
            T vv[U];
            int cc[U];
            ld_shared_run<U>(&s_col[stage_buf][stage_base + b * U], cc);
            ld_shared_run<U>(&s_val[stage_buf][stage_base + b * U], vv);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = b * U + u;  // position inside the chunk
                buf[u] = vzero(static_cast<V *>(nullptr));
                if (t < cnt && inside) buf[u] = ld_dense(dense_row(b_lane, static_cast<unsigned>(cc[u]), row_bytes));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                vfma(acc, vv[u], buf[u]);
                ++pos;
                if (pos == cur_end) {  // the stream passed the end of a row: store it, start the next
                    if (inside) st_stream(c_lane + static_cast<size_t>(cur_row) * row_vecs, acc);
                    acc = vzero(static_cast<V *>(nullptr));
                    if (todo) {
                        cur = __ffs(todo) - 1;
                        todo &= todo - 1;
                        cur_row = __shfl_sync(gmask, row, cur, L);
                        cur_end = __shfl_sync(gmask, start, cur, L) + __shfl_sync(gmask, len, cur, L);
                    } else {
                        cur_end = INT_MAX;
                    }
                }
            }
        }
        c_cur = c_nxt;
        v_cur = v_nxt;
        c_nxt = c_pre;
        v_nxt = v_pre;
        stage_buf ^= 1;
    }
    }();
    group = kClaim ? __shfl_sync(gmask, claimed, 0, L) : n_groups;
    }  // bundles of this group
    if (blockIdx.x == 0 && blockIdx.y == 0) chain_wait();
}

// ---------------------------------------------------------------------------------------
// Residue rows without a block part, one lane group (L lanes x VPL vectors) per R neighbouring rows.  Used
// where a warp holds several groups: there the groups would run different entry streams in
// spmm_rows and diverge, which measured slower (stencil N = 64: 1.43 ms against 0.93 ms),
// while for 32-lane groups the batched kernel wins (R-MAT N = 128: 327 us against 770 us).
constexpr int kRowsCtaThreads = 32;
constexpr long long kWideRowsWaves = 2;  // spmm_rows_wide (a warp per row) serves lists of at most so many waves of 32 warps per SM

template <typename T, int VB, int L, int VPL, int R, bool kRagged, bool kFirst>
__global__ void __launch_bounds__(kRowsCtaThreads, 1024 / kRowsCtaThreads)  // 64 registers: 32 warps per SM
spmm_rows_simple(int m2, int n, const T *__restrict__ values, const int *__restrict__ column_indices,
                 const int *__restrict__ row_offsets, const int *__restrict__ residue_r_ind,
                 const T *__restrict__ B, T *__restrict__ C) {
    using V = typename VecB<T, VB>::type;
    constexpr int kLen = VecB<T, VB>::kLen;
    constexpr int kInFlight = kLoadsInFlight * 16 / VB / VPL;  // dense rows per batch
    constexpr int U = (kInFlight < L) ? kInFlight : L;
    constexpr int kAlign = 4;    // vec_len of the preprocessing
    constexpr int kBlockK = 32;  // k_block of the preprocessing
    if (blockIdx.x == gridDim.x - 1) return chain_wait();  // the CTA behind the rows
    const int lane = threadIdx.x & 31;
    const int l = lane % L;
    const unsigned gmask = group_mask<L>(lane);
    unsigned cta = blockIdx.x;
    if constexpr (kFirst) cta = after_chain(cta);
    const long long item0 = ((static_cast<long long>(cta) * kRowsCtaThreads + threadIdx.x) / L) * R;
    int row[R], begin[R], end[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        row[r] = -1;
        begin[r] = end[r] = 0;
        if (item0 + r < m2) row[r] = residue_r_ind != nullptr ? __ldg(residue_r_ind + item0 + r) : static_cast<int>(item0 + r);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (row[r] >= 0) {
            begin[r] = __ldg(row_offsets + row[r]);
            end[r] = __ldg(row_offsets + row[r] + 1);
        }
    // Lane l keeps nonzero l of a chunk of L; the pair is fetched one chunk ahead, so that the
    // fetch overlaps the gathers of the current chunk.
    int c_first[R];
    T v_first[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        // aligned length >= k_block: a block part exists and its last segment took the tail;
        // list form, no nonzero: the row stays as the caller zero-filled it (all rows: zeros are stored below)
        if (end[r] - begin[r] + (begin[r] % kAlign) >= kBlockK || (end[r] == begin[r] && residue_r_ind != nullptr)) row[r] = -1;
        c_first[r] = 0;
        v_first[r] = T(0);
        if (row[r] >= 0 && begin[r] + l < end[r]) {
            c_first[r] = ld_stream(column_indices + begin[r] + l);
            v_first[r] = ld_stream(values + begin[r] + l);
        }
    }
    // (this kernel keeps the 64-bit index form of the dense-row address: the 32 x 32 -> 64 bit form of
    // the other kernels measured 2.7 % slower here, stencil N = 64 0.692 -> 0.711 ms)
    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const size_t col_vec = static_cast<size_t>(blockIdx.y) * L * VPL + l;
    const V *b_lane = reinterpret_cast<const V *>(B) + col_vec;
    auto inside = [&](int v) { return !kRagged || col_vec + v * L < row_vecs; };
    // chunk staging in shared memory as in spmm_block (one region of L pairs per lane group; the
    // groups of a warp run rows of different lengths, so they synchronise by group)
    static_assert(L % U == 0 && U % 4 == 0, "whole batches, read as runs of four");
    __shared__ __align__(16) int s_col[2][kRowsCtaThreads];
    __shared__ __align__(16) T s_val[2][kRowsCtaThreads];
    const int stage_base = (threadIdx.x / L) * L;
    int stage_buf = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (row[r] < 0) continue;
        V acc[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v) acc[v] = vzero(static_cast<V *>(nullptr));
        int c_nxt = c_first[r];
        T v_nxt = v_first[r];
        for (int base = begin[r]; base < end[r]; base += L) {
            const int c = c_nxt;
            const T val = v_nxt;
            const int e = base + L + l;
            c_nxt = 0;
            v_nxt = T(0);
            if (e < end[r]) {
                c_nxt = ld_stream(column_indices + e);
                v_nxt = ld_stream(values + e);
            }
            const int cnt = min(L, end[r] - base);
            s_col[stage_buf][stage_base + l] = c;
            s_val[stage_buf][stage_base + l] = val;
            __syncwarp(gmask);
#pragma unroll
            for (int t0 = 0; t0 < L; t0 += U) {
                if (t0 >= cnt) break;
                int cc[U];
                T vv[U];
                V bb[U][VPL];
                ld_shared_run<U>(&s_col[stage_buf][stage_base + t0], cc);
                ld_shared_run<U>(&s_val[stage_buf][stage_base + t0], vv);
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        bb[u][v] = vzero(static_cast<V *>(nullptr));
                        if (t0 + u < cnt && inside(v))
                            bb[u][v] = ld_dense(b_lane + static_cast<size_t>(cc[u]) * row_vecs + v * L);
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int v = 0; v < VPL; ++v) vfma(acc[v], vv[u], bb[u][v]);
            }
            stage_buf ^= 1;
        }
#pragma unroll
        for (int v = 0; v < VPL; ++v)
            if (inside(v))
                st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row[r]) * row_vecs + col_vec + v * L, acc[v]);
    }
}

// ---------------------------------------------------------------------------------------
// The same rows, R per lane group one after the other, with all pairs of the warp's rows fetched at once: a load per row
// and array, coalesced over the row's nonzeros (fewer than 32), instead of one per chunk of L nonzeros of several rows.  That
// is three memory round trips before a warp only waits for dense rows, and a third fewer wavefronts for the pairs on the SM's
// load path, which bounds rows that share their columns (27-point stencil 128^3, us, one chunk after the other / staged: N = 16
// 353 / 286, N = 32 390 / 368, N = 64 673 / 628, N = 96 1179 / 1090, fp64 N = 32 792 / 665; 300,000 rows of 15 to 24 N = 64 116 / 97; 1,000,000 of 0
// to 12 N = 32 133 / 118, N = 64 267 / 226; Pareto 2^20 rows alone N = 64 434 / 358).
//
// It serves matrices without segments and lists of 2^19 rows and more.  Shorter lists beside a block grid keep spmm_rows_simple:
// there the rows are the smaller part, and their loads get in the way of the last segments (R-MAT 17 N = 64 51 / 54, the rows
// alone 25 / 22; Pareto 300,007 N = 32 87 / 93; but R-MAT 21 N = 64 697 / 679, Pareto 2^20 N = 64 1105 / 1064).
// (That is said of block grids that fill the GPU.  A handful of segments takes a short list off this kernel as well, for nothing: stencil
// 61^3 without / with one row of 600 nonzeros N = 64 84 / 90.)
//
// R = 2 where rows are not known to be long (rows alone, R = 1 / 2: R-MAT 21 N = 64 278 / 226, Pareto 2^20 N = 64 371 / 358; stencil N = 64
// 633 / 650; rows of 15 to 24 N = 32 56 / 58, N = 64 102 / 97); the 128-byte tile of fp64 has no room for two (8 rows x 32
// pairs are 3 KB per CTA; 1,000,000 rows of 0 to 12 N = 16 131 / 188) and leaves short rows to spmm_rows_simple (R-MAT 21 N = 16 456 /
// 466).
constexpr int kStagedRows = 1 << 19;
template <typename T, int VB, int L, int VPL, int R, bool kRagged, bool kFirst>
__global__ void __launch_bounds__(kRowsCtaThreads, 1024 / kRowsCtaThreads)  // 64 registers: 32 warps per SM
spmm_rows_simple_staged(int m2, int n, const T *__restrict__ values, const int *__restrict__ column_indices,
                 const int *__restrict__ row_offsets, const int *__restrict__ residue_r_ind,
                 const T *__restrict__ B, T *__restrict__ C) {
    using V = typename VecB<T, VB>::type;
    constexpr int kLen = VecB<T, VB>::kLen;
    constexpr int U = kLoadsInFlight * 16 / VB / VPL;  // dense rows per batch
    constexpr int G = 32 / L;                          // rows side by side
    constexpr int N = G * R;                           // rows of the warp
    constexpr int kAlign = 4;    // vec_len of the preprocessing
    constexpr int kBlockK = 32;  // k_block of the preprocessing
    constexpr unsigned kFull = 0xffffffffu;
    static_assert(U == 4 && N <= 32, "quadruples; a descriptor per lane");
    if (blockIdx.x == gridDim.x - 1) return chain_wait();  // the CTA behind the rows
    __shared__ __align__(16) int s_col[N * 32];
    __shared__ __align__(16) T s_val[N * 32];
    const int lane = threadIdx.x;
    const int g = lane / L, l = lane % L;
    unsigned cta = blockIdx.x;
    if constexpr (kFirst) cta = after_chain(cta);
    const long long item0 = static_cast<long long>(cta) * N;
    // lane j of the warp reads the descriptor of row item0 + j; group g takes rows g, G + g, ...
    int row = -1, begin = 0, len = 0;
    if (lane < N && item0 + lane < m2) {
        row = residue_r_ind != nullptr ? __ldg(residue_r_ind + item0 + lane) : static_cast<int>(item0) + lane;
        begin = __ldg(row_offsets + row);
        const int end = __ldg(row_offsets + row + 1);
        // aligned length >= k_block: a block part exists and its last segment took the tail;
        // list form, no nonzero: the row stays as the caller zero-filled it (all rows: zeros are stored below)
        if (end - begin + (begin % kAlign) >= kBlockK || (end == begin && residue_r_ind != nullptr))
            row = -1;
        else
            len = end - begin;
    }
    int c[N];
    T v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const int b = __shfl_sync(kFull, begin, r), e = __shfl_sync(kFull, len, r);
        c[r] = 0;
        v[r] = T(0);
        if (lane < e) {
            c[r] = ld_stream(column_indices + b + lane);
            v[r] = ld_stream(values + b + lane);
        }
    }
    // quadruple q of row r: rotated so that the lane groups read the same one of neighbouring rows from different banks
    auto at = [](int r, int q) { return r * 32 + ((q ^ (r & 7)) << 2); };
#pragma unroll
    for (int r = 0; r < N; ++r) {
        s_col[at(r, lane / 4) + lane % 4] = c[r];
        s_val[at(r, lane / 4) + lane % 4] = v[r];
    }
    __syncwarp();
    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const size_t col_vec = static_cast<size_t>(blockIdx.y) * L * VPL + l;
    const unsigned row_bytes = static_cast<unsigned>(n) * static_cast<unsigned>(sizeof(T));  // n < 2^21 elements
    const V *b_lane = reinterpret_cast<const V *>(B) + col_vec;
    auto inside = [&](int v) { return !kRagged || col_vec + v * L < row_vecs; };
#pragma unroll 1
    for (int i = 0; i < R; ++i) {
        const int row_i = __shfl_sync(kFull, row, i * G + g), len_i = __shfl_sync(kFull, len, i * G + g);
        const int longest = __reduce_max_sync(kFull, len_i);
        V acc[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v) acc[v] = vzero(static_cast<V *>(nullptr));
        for (int t0 = 0; t0 < longest; t0 += U) {
            int cc[U];
            T vv[U];
            V bb[U][VPL];
            ld_shared_run<U>(s_col + at(i * G + g, t0 / 4), cc);
            ld_shared_run<U>(s_val + at(i * G + g, t0 / 4), vv);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < VPL; ++v) {
                    bb[u][v] = vzero(static_cast<V *>(nullptr));
                    if (t0 + u < len_i && inside(v))
                        bb[u][v] = ld_dense(dense_row(b_lane + v * L, static_cast<unsigned>(cc[u]), row_bytes));
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < VPL; ++v) vfma(acc[v], vv[u], bb[u][v]);
        }
        if (row_i >= 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v)
                if (inside(v))
                    st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row_i) * row_vecs + col_vec + v * L, acc[v]);
        }
    }
}

// ---------------------------------------------------------------------------------------
// The same rows, one WARP per row: for residue lists too short to fill the GPU, where the
// time of the launch is the dependent chain of one row, not throughput.  The 32 lanes fetch
// the row's (fewer than 32) pairs in one coalesced load; the 32 / L lane groups then take
// every (32 / L)-th nonzero each, so that all gathers of the row are in flight at once (L
// per group), and a butterfly over the groups adds the partial rows.  Two dependent memory
// round trips after the row's bounds are known, against up to 32 / L in spmm_rows_simple.
template <typename T, int VB, int L, int VPL, bool kRagged>
__global__ void __launch_bounds__(32 * kSmallGridWarps, 1)
spmm_rows_wide(int m2, int n, const T *__restrict__ values, const int *__restrict__ column_indices,
               const int *__restrict__ row_offsets, const int *__restrict__ residue_r_ind,
               const T *__restrict__ B, T *__restrict__ C, bool first) {
    using V = typename VecB<T, VB>::type;
    constexpr int kLen = VecB<T, VB>::kLen;
    constexpr int G = 32 / L;    // lane groups; a group takes at most 32 / G = L nonzeros
    constexpr int kAlign = 4;    // vec_len of the preprocessing
    constexpr int kBlockK = 32;  // k_block of the preprocessing
    constexpr unsigned kFull = 0xffffffffu;
    if (blockIdx.x == gridDim.x - 1) return chain_wait();  // the CTA behind the rows
    const int cta = after_chain_if(first, blockIdx.x);
    const int item = cta * kSmallGridWarps + (threadIdx.x >> 5);
    if (item >= m2) return;
    const int lane = threadIdx.x & 31;
    const int g = lane / L, l = lane % L;

    const int row = residue_r_ind != nullptr ? __ldg(residue_r_ind + item) : item;
    const int begin = __ldg(row_offsets + row);
    const int end = __ldg(row_offsets + row + 1);
    if (end - begin + (begin % kAlign) >= kBlockK) return;  // the block part took this row's tail
    const int len = end - begin;                            // < 32
    if (len == 0 && residue_r_ind != nullptr) return;

    int c = 0;
    T val = T(0);
    if (lane < len) {
        c = ld_stream(column_indices + begin + lane);
        val = ld_stream(values + begin + lane);
    }
    const size_t row_vecs = static_cast<size_t>(n) / kLen;
    const unsigned row_bytes = static_cast<unsigned>(n) * static_cast<unsigned>(sizeof(T));  // n < 2^21 elements
    const size_t col_vec = static_cast<size_t>(blockIdx.y) * L * VPL + l;
    const V *b_lane = reinterpret_cast<const V *>(B) + col_vec;
    auto inside = [&](int v) { return !kRagged || col_vec + v * L < row_vecs; };
    if (len == 0) {  // (list form: stays as the caller zero-filled it, returned above)
        if (g == 0) {
#pragma unroll
            for (int v = 0; v < VPL; ++v)
                if (inside(v))
                    st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row) * row_vecs + col_vec + v * L,
                              vzero(static_cast<V *>(nullptr)));
        }
        return;
    }

    int cc[L];
    T vv[L];
    V bb[L][VPL];
#pragma unroll
    for (int t = 0; t < L; ++t) {  // nonzero t * G + g
        cc[t] = __shfl_sync(kFull, c, t * G + g);
        vv[t] = __shfl_sync(kFull, val, t * G + g);
    }
#pragma unroll
    for (int t = 0; t < L; ++t)
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
            bb[t][v] = vzero(static_cast<V *>(nullptr));
            if (t * G + g < len && inside(v)) bb[t][v] = ld_dense(dense_row(b_lane, static_cast<unsigned>(cc[t]), row_bytes) + v * L);
        }
    V acc[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        acc[v] = vzero(static_cast<V *>(nullptr));
#pragma unroll
        for (int t = 0; t < L; ++t) vfma(acc[v], vv[t], bb[t][v]);
#pragma unroll
        for (int d = L; d < 32; d <<= 1) vadd(acc[v], vshfl_xor(kFull, acc[v], d));
    }
    if (g == 0) {
#pragma unroll
        for (int v = 0; v < VPL; ++v)
            if (inside(v)) st_stream(reinterpret_cast<V *>(C) + static_cast<size_t>(row) * row_vecs + col_vec + v * L, acc[v]);
    }
}

// When an order of the segments pays (rode_order.cuh): from an operand beyond the L2 on, on skewed columns for the 256- and 512-byte
// tiles of float only.  Whole calls, row by row / ordered, us.
//
// What it gives is a matter of how much of the columns a segment spans.  N = 64, 2^20 columns (256 MB): Zipf of mean 16 (segments
// span 0.46 of the columns on average) 598 / 395, log-normal lengths of sigma 3 (0.70) 640 / 494, Pareto of mean 32 (0.86) 1063 / 912, of
// mean 16 603 / 546; 2^21 columns: log-normal of sigma 1 (0.96), mean 16 and 32, 1273 / 1538 and 2435 / 3018, Pareto of shape 2
// (0.95) 2401 / 2986.  Segments that are rows of one length (span 0.99; three segments: 0.33): rows of 256, 400, 500 N = 128
// 662 / 678, 523 / 540, 478 / 505, N = 256 1395 / 1428, 1136 / 1181, 980 / 1083, N = 32 401 / 415, 388 / 396, 370 / 380, rows of
// 1500 N = 128 523 / 371.  So wide segments keep the order of the rows, except short ones in grids that are not too large (up
// to 2^17 of less than 192 nonzeros: rows of 160 N = 128 803 / 802, of 96 824 / 828, log-normal of sigma 2 1212 / 1203); narrow ones
// are ordered from 8192 on (Pareto of shape 0.8 and mean 4, 11,607 segments, N = 128 418 / 406; rows of 600, 13,980 segments, 250 /
// 172), and those between them where there are more segments and references per column (Pareto of mean 8, 31,336 segments,
// N = 128 673 / 675, 2^22 of mean 8 N = 32 1023 / 1039, N = 128 2841 / 2820).
//
// In the 256-byte tile of float the ordered form is the faster one whatever the segments
// span, up to 2^17 of them and from 4 references per column on (rows of 256, 400, 500 N = 64 323 / 308, 275 / 264, 273 / 258, Pareto of
// mean 4 and 8 243 / 230, 366 / 344, of mean 4 N = 48 232 / 224; of 2 references per column rows of 96, 160 N = 64 73 / 77, 74 / 77).
//
// Skewed columns, against the popularity hints at N = 128 and 256 and without at 64: R-MAT 23, 22, 21, 20 N = 64 3136 / 2764, 1441 / 1326,
// 693 / 668, 355 / 334, but N = 32 863 / 876 (22), fp64 N = 32 785 / 832 (21); N = 128, calls one by one 5072 / 4900, 2275 / 2224, 1081 / 1064,
// 531 / 522 (19: 271 / 275), back to back under the power cap 5879 / 5799, 2743 / 2677, 1266 / 1253, 605 / 581, between GEMMs 5800 / 5671, 2643 /
// 2595, 1221 / 1222, 581 / 570; with rows and columns in random order 5132 / 5019, 2284 / 2225, 1070 / 1045, 532 / 503; of 32 per row (21)
// 1900 / 1807, 20 of 64 1635 / 1543, N = 256 (22) 4837 / 4560; 22 of 6 per row 1119 / 1136, which the references per column leave out.
// Columns skewed by themselves (Pareto 2^21 of mean 16, columns repeat 13, 81, 334 times as often as uniform ones) N = 64 1124 /
// 1097, 977 / 947, 781 / 742, but N = 128 2074 / 2087, 1681 / 1721, 1134 / 1201: there hints are better from some fifteen calls on,
// for an ordered first call needs no bitmap (0.5 to 2 ms).
bool order_pays(int verdict, long long m1, long long k, long long n, long long nnz, int elem_size) {
    if (verdict < 0 || m1 < kOrderMinSegments || k * n * elem_size < 160ll << 20) return false;
    const int kind = verdict & kOrderKind;
    const long long row_bytes = n * elem_size;
    const bool moderate = m1 <= 1 << 17 && row_bytes > 128;
    const bool narrow_tile = moderate && elem_size == 4 && row_bytes <= 256 && kind == kOrderHelps && nnz >= 4 * k;
    if ((verdict & kOrderWide) != 0 && !narrow_tile && !(moderate && nnz < 192 * m1)) return false;
    const bool narrow = (verdict & kOrderNarrow) != 0 && kind == kOrderHelps;
    if (!narrow && !narrow_tile && (m1 < 1 << 15 || nnz < 12 * k)) return false;
    return kind == kOrderHelps || (kind == kOrderSkewed && elem_size == 4 && (n == 64 || n % 128 == 0));
}

template <typename T, int VB, int L, int VPL, bool kRagged>
int launch_rows(int m2, int n, const T *values, const int *col, const int *row_offsets, const int *residue_r_ind,
                const T *B, T *C, int *counters, bool chained, bool counters_clear, int m1, long long nnz,
                cudaStream_t s2);

// Block kernel of one shape and residue-row kernel of another; each walks the columns in tiles of its own.
template <typename T, typename Block, typename Rows, bool kRagged = false, bool kRowsRagged = kRagged>
int launch_shape(int m1, int m2, int k, int n, const T *values, const int *col, const int *row_offsets,
                 const int *block_r_ind, const int *residue_r_ind, const int *st_off, const T *B, T *C,
                 T *partial, int *counters, const unsigned *hot, long long nnz, const Ordering *ord, cudaStream_t s1,
                 cudaStream_t s2) {
    constexpr int VB = Block::VB, L = Block::L, VPL = Block::VPL;
    constexpr int kTileWidth = L * VPL * VecB<T, VB>::kLen;
    constexpr int U = kLoadsInFlight * 16 / VB / VPL;            // rows per batch
    // ragged widths: the last tile is partly empty
    const unsigned tiles = static_cast<unsigned>(kRagged ? (n + kTileWidth - 1) / kTileWidth : n / kTileWidth);
    const bool chained = s1 == s2 && m1 > 0;
    bool rows_done = false;
    bool counters_clear = false;  // the residue kernel's claim counters have been zeroed already
    if (m1 > 0) {
        // fewer warps than two full waves of 32 per SM: no hints, no claims
        const bool small_grid = static_cast<long long>(m1) * tiles <= 2LL * 32 * sm_count();
        // large grids: one resident wave of CTAs whose warps claim segments from counters at the end of the workspace,
        // zeroed on the stream before the launch
        const int ctas_needed = (m1 + kCtaWarps - 1) / kCtaWarps;
        const int resident = kPersistentCtasPerSm * sm_count();
        const int resident_per_tile = resident / static_cast<int>(tiles <= kClaimTiles ? tiles : 1);
        const bool claims = counters != nullptr && claims_work<T>(n, tiles);
        const bool persistent = claims && !small_grid && ctas_needed > kPersistentMinWaves * resident_per_tile;
        // in a chain the residue kernel's counters are zeroed here too: nothing may stand between two of its grids.  On a stream
        // of its own it may be at work already, and zeroes them itself
        counters_clear = claims && chained && m2 > 32LL * kPersistentMinWaves * resident_per_tile;
        if (persistent || counters_clear)
            RODE_CUDA_TRY(cudaMemsetAsync(counters, 0, (counters_clear ? 2 : 1) * kClaimTiles * sizeof(int), s1));
        int *claim = persistent ? counters : nullptr;
        dim3 grid(persistent ? (resident + tiles - 1) / tiles : ctas_needed, tiles);
        bool launched = false;  // one of the special forms
        if (ord != nullptr) {  // segments in the order of their columns
            if (int rc = launch_order<0>(*ord, m1, row_offsets, col, block_r_ind, st_off, s1)) return rc;
            RODE_CUDA_TRY(launch_chained(spmm_block<T, VB, L, VPL, U, kCtaWarps, 1, false, true, kRagged, true>, grid,
                                         dim3(kCtaThreads), s1, true, m1, n, values, col, row_offsets, block_r_ind, st_off, B, C,
                                         partial, nullptr, 0, claim, ord->list<0>()));
            launched = true;
        }
        // Popularity hints: block kernel of the 512-byte tile only.  In the residue-row kernel
        // the marks saved DRAM bytes (5.36 -> 4.79 GB on R-MAT scale 23) but the extra registers
        // cost more time than that returned (1.41 -> 1.52 ms).
        if constexpr (L * VPL * VB == 512 && !kRagged) {
            if (!launched && hot && !small_grid) {
                RODE_CUDA_TRY(launch_chained(spmm_block<T, VB, L, VPL, U, kCtaWarps, 1, true, true, false>, grid, dim3(kCtaThreads), s1, true,
                    m1, n, values, col, row_offsets, block_r_ind, st_off, B, C, partial, hot, (k + 31) / 32, claim, nullptr));
                launched = true;
            }
        }
        // Up to 40 MB of gathers the host's launches are what a call waits for: one for segments and rows.  (Beyond
        // that the separate kernels win back their launch: R-MAT 13 N = 128, 64 MB, 16.7 us with them, 18.7 in one.)
        const bool one_launch = !launched && chained && nnz >= 0 && nnz * n * static_cast<long long>(sizeof(T)) <= 40LL << 20 &&
                                small_grid && static_cast<long long>(m2) * tiles <= 2LL * 32 * sm_count();
        if (one_launch) {
            constexpr int UOne = 2 * U <= L ? 2 * U : L;
            const int seg_ctas = (m1 + kOneLaunchWarps - 1) / kOneLaunchWarps;
            const int row_ctas = (m2 + kOneLaunchWarps - 1) / kOneLaunchWarps;
            RODE_CUDA_TRY(launch_chained(spmm_one_launch<T, VB, L, VPL, UOne, kRagged>, dim3(seg_ctas + row_ctas, tiles),
                                         dim3(32 * kOneLaunchWarps), s1, true, m1, seg_ctas, m2, n, values, col, row_offsets,
                                         block_r_ind, st_off, residue_r_ind, B, C, partial));
            rows_done = launched = true;
        }
        const long long warps = static_cast<long long>(m1) * tiles;
        if (!launched && warps <= kSplit4WarpsPerSm * sm_count()) {
            RODE_CUDA_TRY(launch_chained(spmm_block<T, VB, L, VPL, U, 4, 4, false, false, kRagged>, dim3(m1, tiles), dim3(4 * 32), s1,
                                         true, m1, n, values, col, row_offsets, block_r_ind, st_off, B, C, partial, nullptr, 0,
                                         nullptr, nullptr));
        } else if (!launched && warps <= kSplit2WarpsPerSm * sm_count()) {
            RODE_CUDA_TRY(launch_chained(spmm_block<T, VB, L, VPL, U, 2, 2, false, false, kRagged>, dim3(m1, tiles), dim3(2 * 32), s1,
                                         true, m1, n, values, col, row_offsets, block_r_ind, st_off, B, C, partial, nullptr, 0,
                                         nullptr, nullptr));
        } else if (!launched) {
            RODE_CUDA_TRY(launch_chained(spmm_block<T, VB, L, VPL, U, kCtaWarps, 1, false, true, kRagged>, grid, dim3(kCtaThreads), s1,
                                         true, m1, n, values, col, row_offsets, block_r_ind, st_off, B, C, partial, nullptr, 0,
                                         claim, nullptr));
        }
        RODE_CHECK_LAUNCH("rode::spmm_block");
    }
    // Rows: on the block kernel's own stream they are chained behind it (see chain_begin), on another one
    // they are a plain launch.
    if (m2 > 0 && !rows_done) {
        if (int rc = launch_rows<T, Rows::VB, Rows::L, Rows::VPL, kRowsRagged>(m2, n, values, col, row_offsets, residue_r_ind, B, C, counters,
                                                            chained, counters_clear, m1, nnz, s2))
            return rc;
    }
    if (m1 > 1) {  // (a row that was cut has two segments at least)
        // fix-up last, chained behind the block grid (and the rows): its launch latency and its
        // metadata prologue overlap the tail of those grids
        int per = (m1 / (4 * sm_count()) + 31) / 32 * 32;  // segments per CTA: about four CTAs per SM
        per = per < 32 ? 32 : (per > kFixupThreads ? kFixupThreads : per);
        const T *partial_in = partial;
        RODE_CUDA_TRY(launch_chained(spmm_fixup<T>, dim3((m1 + per - 1) / per), dim3(kFixupThreads), s1, true, m1, per, n,
                                     row_offsets, block_r_ind, st_off, partial_in, C));
        RODE_CHECK_LAUNCH("rode::spmm_fixup");
    }
    return RODE_OK;
}

template <typename T, int VB, int L, int VPL, bool kRagged>
int launch_rows(int m2, int n, const T *values, const int *col, const int *row_offsets, const int *residue_r_ind,
                const T *B, T *C, int *counters, bool chained, bool counters_clear, int m1, long long nnz,
                cudaStream_t s2) {
    constexpr int kTileWidth = L * VPL * VecB<T, VB>::kLen;
    const unsigned tiles = static_cast<unsigned>(kRagged ? (n + kTileWidth - 1) / kTileWidth : n / kTileWidth);
    if constexpr (VB == 16 && L == 32 && VPL == 1) {
        // 32 rows per warp when the list is long; fewer (shorter dependent chains, more
        // warps) when the warps would not fill the GPU twice over
        const long long slots = 2LL * 28 * sm_count() * (kCtaThreads / 32);
        int per_group = static_cast<int>((m2 + slots - 1) / slots);
        per_group = per_group < 4 ? 4 : (per_group > 32 ? 32 : per_group);
        const long long groups = (static_cast<long long>(m2) + per_group - 1) / per_group;
        constexpr int kGroupsPerCta = kCtaThreads / 32;
        const long long ctas_needed = (groups + kGroupsPerCta - 1) / kGroupsPerCta;
        const long long resident = static_cast<long long>(kPersistentCtasPerSm) * sm_count();
        const bool persistent = counters != nullptr && claims_work<T>(n, tiles) && (!chained || counters_clear) &&
                                ctas_needed > kPersistentMinWaves * (resident / tiles);
        int *claim = nullptr;
        if (persistent) {
            claim = counters + kClaimTiles;
            if (!counters_clear) RODE_CUDA_TRY(cudaMemsetAsync(claim, 0, kClaimTiles * sizeof(int), s2));
        }
        const dim3 grid(static_cast<unsigned>(persistent ? (resident + tiles - 1) / tiles : ctas_needed), tiles);
        RODE_CUDA_TRY(launch_chained(spmm_rows<T, 32, kRagged>, grid, dim3(kCtaThreads), s2, true, m2, per_group, n, values,
                                     col, row_offsets, residue_r_ind, B, C, claim, !chained));
    } else if (static_cast<long long>(m2) * tiles <= kWideRowsWaves * 32 * sm_count()) {
        const dim3 grid((m2 + kSmallGridWarps - 1) / kSmallGridWarps + 1, tiles);
        RODE_CUDA_TRY(launch_chained(spmm_rows_wide<T, VB, L, VPL, kRagged>, grid, dim3(32 * kSmallGridWarps), s2, true, m2,
                                     n, values, col, row_offsets, residue_r_ind, B, C, !chained));
    } else {
        // (first grid of the call: an early start is worth a microsecond, and a wait in each of half a million CTAs costs
        // more than that: stencil 128^3 N = 64 +1.7 %)
        auto launch = [&](auto plain, auto first, int rows_per_group) {
            const int rows_per_cta = rows_per_group * kRowsCtaThreads / L;
            const dim3 grid(static_cast<unsigned>((static_cast<long long>(m2) + rows_per_cta - 1) / rows_per_cta + 1), tiles);
            const bool early = !chained && grid.x <= 64u * 32u * sm_count();
            return launch_chained(early ? first : plain, grid, dim3(kRowsCtaThreads), s2, chained || early, m2, n, values, col,
                                  row_offsets, residue_r_ind, B, C);
        };
        constexpr int kTileBytes = VB * L * VPL;
        constexpr bool kRoomForTwo = sizeof(T) == 4 || kTileBytes > 128;
        const bool shorts = short_rows(nnz, m1, m2, kTileBytes);
        const bool staged = (m1 == 0 || m2 >= kStagedRows) && (kRoomForTwo || !shorts);
        if constexpr (kRoomForTwo) {
            if (staged && !rows_hold(nnz, m1, m2, kTileBytes == 128 ? 10 : 20)) {
                RODE_CUDA_TRY(launch(spmm_rows_simple_staged<T, VB, L, VPL, 2, kRagged, false>,
                                     spmm_rows_simple_staged<T, VB, L, VPL, 2, kRagged, true>, 2));
                RODE_CHECK_LAUNCH("rode::spmm_rows");
                return RODE_OK;
            }
        }
        if (staged) {
            RODE_CUDA_TRY(launch(spmm_rows_simple_staged<T, VB, L, VPL, 1, kRagged, false>,
                                 spmm_rows_simple_staged<T, VB, L, VPL, 1, kRagged, true>, 1));
        } else if (shorts) {
            // Two rows per lane group where rows are short: both rows' bounds and first columns are then fetched together, and
            // a short row's life is that chain of loads; long even rows lose it again to the longer life of a warp.
            RODE_CUDA_TRY(launch(spmm_rows_simple<T, VB, L, VPL, 2, kRagged, false>,
                                 spmm_rows_simple<T, VB, L, VPL, 2, kRagged, true>, 2));
        } else {
            RODE_CUDA_TRY(launch(spmm_rows_simple<T, VB, L, VPL, 1, kRagged, false>,
                                 spmm_rows_simple<T, VB, L, VPL, 1, kRagged, true>, 1));
        }
    }
    RODE_CHECK_LAUNCH("rode::spmm_rows");
    return RODE_OK;
}

template <typename T>
int spmm(int m1, int m2, int k, int n, const T *values, const int *col, const int *row_offsets,
         const int *block_r_ind, const int *residue_r_ind, const int *st_off, const T *B, T *C, void *workspace,
         size_t workspace_bytes, const unsigned *hot, rode_stream_t stream1, rode_stream_t stream2,
         bool all_rows = false, long long nnz = -1, bool ordered = false) {
    constexpr int kLen = Vec16<T>::kLen;
    if (m1 < 0 || m2 < 0 || n <= 0) return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: m1, m2 >= 0 and n > 0 required");
    if (hot != nullptr && k <= 0)
        return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: k (the number of columns the bitmap covers) must be positive "
                                               "when hot_columns is given");
    if (n % 4 != 0) return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: n = %d is not a multiple of 4", n);
    if (m1 == 0 && m2 == 0) return RODE_OK;
    const bool may_be_empty = all_rows && m1 == 0;  // rows of zeros only: nothing of the three arrays is read
    if (!row_offsets || !C || (!may_be_empty && (!values || !col || !B))) return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: null array");
    if (m1 > 0 && (!block_r_ind || !st_off)) return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: null block metadata");
    if (m2 > 0 && !residue_r_ind && !all_rows) return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: null residue metadata");
    if (!aligned_to(B, 16) || !aligned_to(C, 16))
        return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: B and C must be 16-byte aligned");
    if ((n + 8 * kLen - 1) / (8 * kLen) > 65535)
        return fail(RODE_ERR_INVALID_ARGUMENT, "spmm: n = %d exceeds the supported width (%d)", n, 65535 * 8 * kLen);
    size_t need = 0;
    rode_spmm_workspace_bytes(m1, n, static_cast<int>(sizeof(T)), &need);
    // Without block segments the workspace holds the claim counters only and may be left out (the
    // residue kernel then runs one CTA per bundle of rows).
    if (m1 > 0 || workspace != nullptr) {
        if (workspace == nullptr || workspace_bytes < need)
            return fail(RODE_ERR_WORKSPACE, "spmm: workspace of %zu bytes needed, %zu given", need,
                        workspace ? workspace_bytes : static_cast<size_t>(0));
        if (!aligned_to(workspace, 16)) return fail(RODE_ERR_WORKSPACE, "spmm: workspace must be 16-byte aligned");
    }
    Ordering ordering = {}, *ord = nullptr;
    if (ordered && m1 > 0 && m1 < kWholeMaxSegments && k > 0) {
        const size_t more = ordering_bytes<0>(m1, 0);
        if (workspace_bytes < need + more)
            return fail(RODE_ERR_WORKSPACE, "spmm: workspace of %zu bytes needed, %zu given", need + more, workspace_bytes);
        ordering = {reinterpret_cast<OrderHead *>(static_cast<char *>(workspace) + need), m1, k};
        ord = &ordering;
    }
    T *partial = static_cast<T *>(workspace);
    // the claim counters of the persistent block kernel sit behind the partial rows
    int *counters = workspace != nullptr
                        ? reinterpret_cast<int *>(static_cast<char *>(workspace) + need - kCounterBytes) : nullptr;
    // Widest tile (32, 16 or 8 vectors of 16 bytes) that divides the row.
#define RODE_LAUNCH(...)                                                                                             \
    launch_shape<T, __VA_ARGS__>(m1, m2, k, n, values, col, row_offsets, block_r_ind, residue_r_ind, st_off, B, C, partial, \
                                 counters, hot, nnz, ord, stream1, stream2)
    const bool aligned32 = aligned_to(B, 32) && aligned_to(C, 32) && aligned_to(workspace, 32);
    const int vecs = n / kLen;
    // Widths of whole lines that the 512-byte tile does not divide (N = 96, 160, 192, 224 ...): 512-byte tiles with a
    // partly idle last one all the same, instead of up to seven passes over the sparse matrix with narrow ones.  us, narrow ->
    // wide: R-MAT 21 N = 96 1411 -> 954, N = 160 2627 -> 1948, N = 224 3701 -> 2449; Pareto 2^20 N = 96 2309 -> 1756, N = 224
    // 5897 -> 4493; Bernoulli 4096^2 N = 96 20.7 -> 12.5; Zipf 65536 N = 160 70 -> 74.  fp64 only where it is one tile instead
    // of three passes (R-MAT 20 692 -> 517, 30,000 rows of 25 41 -> 31, Zipf 300,007 of mean 40 369 -> 373): several tiles lose what
    // the narrow ones' passes over a slice of the operand keep in the L2 (Zipf of mean 40 N = 112 848 -> 917, N = 144 1092 ->
    // 1356, Pareto 300,007 N = 80 496 -> 566).
    //
    // The residue rows take wide tiles too unless they are long (narrow / wide, us): of 2 (0 to 4) N = 96 61 / 52, N = 160 100 /
    // 100, N = 224 138 / 117; of 4 82 / 72, 133 / 143, 184 / 163; of 7 102 / 101, 166 / 197, 233 / 226; of 10 (8 to 12) 112 / 123,
    // 183 / 250, 259 / 286; of 19.5 190 / 210, 312 / 422, 455 / 489; uneven ones of 5.9 (R-MAT 18) 152 / 138, 280 / 253, 330 / 266, of
    // 11.5 (Pareto 2^20) 1806 / 1718, 3218 / 3211, 4611 / 4286.  So the line lies at 6 where the tiles are three quarters full or
    // more, and at 2 for N = 160.  Beyond a mean of 20 over all rows the narrow form is taken, which loses less on even rows
    // (30,000 rows of 25 N = 96 27 / 31, N = 160 44 / 53) than it gives away on uneven ones (Zipf of mean 40 412 / 376);
    // in fp64, where it gives away more, only if there are fewer segments than one for 20 rows (30,000 rows of 21 27 / 30) or
    // more than one for 8 (rows of 25 31 / 33), else not (Zipf of mean 40 415 / 373, Pareto 300,007 306 / 294).
    if (vecs % 8 == 0 && vecs > 16 && vecs % 32 != 0 && (sizeof(T) == 4 || vecs < 32)) {
        const int full = 4 * vecs >= 3 * 32 * ((vecs + 31) / 32) ? 6 : 2;
        const bool wide_rows = nnz >= 0 && !rows_hold(nnz, m1, m2, full) &&
                               (nnz < 20LL * m2 || (sizeof(T) == 8 && 20LL * m1 >= m2 && 8LL * m1 <= m2));
        hot = nullptr;  // (no popularity hints here)
        if (wide_rows) return RODE_LAUNCH(Tile512, Tile512, true, true);
        if (vecs % 16 == 0) return RODE_LAUNCH(Tile512, Tile256, true, false);
        if (aligned_to(B, 32) && aligned_to(C, 32)) return RODE_LAUNCH(Tile512, Aligned128, true, false);
        return RODE_LAUNCH(Tile512, Rows128, true, false);
    }
    // Matrices without segments whose rows are not short take the 256-byte tile's row kernel, in two or more passes, in the place of
    // the stream of spmm_rows: the passes read the pairs again, but four rows run side by side and wait for dense rows only.  us,
    // stream / 256-byte tiles, N = 128: stencil 128^3 1415 / 1257, 61^3 193 / 156, rows of 15 to 24 271 / 198, of 0 to 27 211 / 177, of 4 to 8
    // 223 / 186, of 4 to 6 195 / 172, of 2 to 6 165 / 160, of 0 to 4 231 / 246; fp64 N = 64 stencil 128^3 1705 / 1351, rows of 15 to 24
    // 308 / 220, of 0 to 4 231 / 258.  Ragged widths idle lanes in the last tile of either, and need longer rows: stencil 61^3
    // N = 68 191 / 139, N = 100 197 / 163, N = 132 340 / 217, N = 200 344 / 297; rows of 0 to 27 145 / 162, 180 / 211, 349 / 305, 426 / 403.
    // (With segments beside them those passes lose, R-MAT 21 N = 128 1109 / 1291; that a few segments do no harm this line does not know:
    // stencil 61^3 without / with one row of 600 nonzeros N = 128 160 / 194, N = 132 224 / 369.)
    const bool long_rows_only = m1 == 0 && rows_hold(nnz, 0, m2, vecs % 32 == 0 ? 5 : 20);
    // Widths the tiles do not divide (any other multiple of 4 columns; the reference has none of them): the narrowest
    // shape that covers the row, or 512-byte tiles with a partly empty last one.  No popularity hints.
    if (vecs % 8 != 0) {
        if (vecs < 8) return RODE_LAUNCH(Block128, Rows128, true);
        if (vecs < 16) return RODE_LAUNCH(Tile256, Tile256, true);
        if (long_rows_only) return RODE_LAUNCH(Tile512, Tile256, true);
        return RODE_LAUNCH(Tile512, Tile512, true);
    }
    // (32-byte loads measured no faster than 16-byte ones in the wider tiles: the gathers are bound by bytes through L1 and L2)
    if (vecs % 32 == 0 && long_rows_only) return RODE_LAUNCH(Tile512, Tile256);
    if (vecs % 32 == 0) return RODE_LAUNCH(Tile512, Tile512);
    if (vecs % 16 == 0) return RODE_LAUNCH(Tile256, Tile256);
    if (aligned32) return RODE_LAUNCH(Aligned128, Aligned128);
    return RODE_LAUNCH(Block128, Rows128);
#undef RODE_LAUNCH
}

}  // namespace

}  // namespace rode

extern "C" {

int rode_spmm_workspace_bytes(int m1, int n, int elem_size, size_t *bytes) {
    if (bytes == nullptr || m1 < 0 || n < 0 || (elem_size != 4 && elem_size != 8))
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "spmm_workspace_bytes: bad argument");
    // one partial row per block segment, rounded up to 256 bytes, then the claim counters
    const size_t rows = static_cast<size_t>(m1) * static_cast<size_t>(n) * static_cast<size_t>(elem_size);
    *bytes = (rows + 255) / 256 * 256 + rode::kCounterBytes;
    return RODE_OK;
}

int rode_spmm_f32(int m1, int m2, int k, int n, const float *values, const int *column_indices,
                  const int *row_offsets, const int *block_r_ind, const int *residue_r_ind, const int *st_off,
                  const float *B, float *C, void *workspace, size_t workspace_bytes, rode_stream_t stream1,
                  rode_stream_t stream2) {
    return rode::spmm<float>(m1, m2, k, n, values, column_indices, row_offsets, block_r_ind, residue_r_ind,
                             st_off, B, C, workspace, workspace_bytes, nullptr, stream1, stream2);
}

int rode_spmm_f32_hot(int m1, int m2, int k, int n, const float *values, const int *column_indices,
                      const int *row_offsets, const int *block_r_ind, const int *residue_r_ind, const int *st_off,
                      const float *B, float *C, void *workspace, size_t workspace_bytes,
                      const unsigned *hot_columns, rode_stream_t stream1, rode_stream_t stream2) {
    return rode::spmm<float>(m1, m2, k, n, values, column_indices, row_offsets, block_r_ind, residue_r_ind,
                             st_off, B, C, workspace, workspace_bytes, hot_columns, stream1, stream2);
}

int rode_spmm_f64(int m1, int m2, int k, int n, const double *values, const int *column_indices,
                  const int *row_offsets, const int *block_r_ind, const int *residue_r_ind, const int *st_off,
                  const double *B, double *C, void *workspace, size_t workspace_bytes, rode_stream_t stream1,
                  rode_stream_t stream2) {
    return rode::spmm<double>(m1, m2, k, n, values, column_indices, row_offsets, block_r_ind, residue_r_ind,
                              st_off, B, C, workspace, workspace_bytes, nullptr, stream1, stream2);
}

int rode_spmm_f64_hot(int m1, int m2, int k, int n, const double *values, const int *column_indices,
                      const int *row_offsets, const int *block_r_ind, const int *residue_r_ind, const int *st_off,
                      const double *B, double *C, void *workspace, size_t workspace_bytes,
                      const unsigned *hot_columns, rode_stream_t stream1, rode_stream_t stream2) {
    return rode::spmm<double>(m1, m2, k, n, values, column_indices, row_offsets, block_r_ind, residue_r_ind,
                              st_off, B, C, workspace, workspace_bytes, hot_columns, stream1, stream2);
}

int rode_spmm_f32_all(int M, int m1, int k, int n, long long nnz, const float *values, const int *column_indices,
                      const int *row_offsets, const int *block_r_ind, const int *st_off, const float *B, float *C,
                      void *workspace, size_t workspace_bytes, const unsigned *hot_columns, rode_stream_t stream1,
                      rode_stream_t stream2) {
    return rode::spmm<float>(m1, M, k, n, values, column_indices, row_offsets, block_r_ind, nullptr, st_off, B, C,
                             workspace, workspace_bytes, hot_columns, stream1, stream2, /*all_rows=*/true, nnz);
}

int rode_spmm_f64_all(int M, int m1, int k, int n, long long nnz, const double *values, const int *column_indices,
                      const int *row_offsets, const int *block_r_ind, const int *st_off, const double *B, double *C,
                      void *workspace, size_t workspace_bytes, const unsigned *hot_columns, rode_stream_t stream1,
                      rode_stream_t stream2) {
    return rode::spmm<double>(m1, M, k, n, values, column_indices, row_offsets, block_r_ind, nullptr, st_off, B, C,
                              workspace, workspace_bytes, hot_columns, stream1, stream2, /*all_rows=*/true, nnz);
}

int rode_spmm_order_pays(int verdict, int m1, int k, int n, long long nnz, int elem_size) {
    return rode::order_pays(verdict, m1, k, n, nnz, elem_size) ? 1 : 0;
}

int rode_spmm_ordered_workspace_bytes(int m1, int n, int elem_size, size_t *bytes) {
    if (int rc = rode_spmm_workspace_bytes(m1, n, elem_size, bytes)) return rc;
    *bytes += rode::ordering_bytes<0>(m1, 0);
    return RODE_OK;
}

int rode_spmm_f32_ordered(int M, int m1, int k, int n, long long nnz, const float *values, const int *column_indices,
                          const int *row_offsets, const int *block_r_ind, const int *st_off, const float *B, float *C,
                          void *workspace, size_t workspace_bytes, rode_stream_t stream1, rode_stream_t stream2) {
    return rode::spmm<float>(m1, M, k, n, values, column_indices, row_offsets, block_r_ind, nullptr, st_off, B, C,
                             workspace, workspace_bytes, nullptr, stream1, stream2, /*all_rows=*/true, nnz, /*ordered=*/true);
}

int rode_spmm_f64_ordered(int M, int m1, int k, int n, long long nnz, const double *values, const int *column_indices,
                          const int *row_offsets, const int *block_r_ind, const int *st_off, const double *B, double *C,
                          void *workspace, size_t workspace_bytes, rode_stream_t stream1, rode_stream_t stream2) {
    return rode::spmm<double>(m1, M, k, n, values, column_indices, row_offsets, block_r_ind, nullptr, st_off, B, C,
                              workspace, workspace_bytes, nullptr, stream1, stream2, /*all_rows=*/true, nnz, /*ordered=*/true);
}

}  // extern "C"
