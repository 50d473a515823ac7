// RoDe SDDMM for sm_100a:  out[e] = values[e] * dot(lhs[row(e), :], rhs[col(e), :]).
//
// Stands in for the reference's SDDMMKernel4Block / SDDMMKernel4Residue
// (RoDe_SDDMM/RoDeSddmm.cu:15-203, :206-494) and their launchers (:496-545).  The work
// split follows the reference's metadata (block segments, residue rows).  sddmm_items serves the residue rows of
// every K and the 32-long segments that go with K = 128; sddmm_block the long segments:
//
//  * A warp takes up to 32 consecutive ITEMS (block segments, or residue rows that have no
//    block part): lane j reads the descriptor of item j, so the dependent chain row index ->
//    row pointer -> column -> dense row is paid once per 32 items.  The nonzeros of the items,
//    concatenated, form one entry stream.  The last segment of a row also covers the row's
//    tail (shorter than 32) that the reference leaves to its residue kernel.
//  * A dense row of length K is covered by a lane group of L lanes, VPL 16-byte loads per
//    lane (K = 4 * L * VPL).  The G = 32/L groups of the warp split the stream into G equal
//    contiguous parts (equal in nonzeros, not in items), so all groups run the same number of
//    iterations and a group walks through its items in order; it keeps the lhs row slice of
//    its current item in registers and prefetches the next item's.
//  * Nonzeros are handled in chunks of L per group (lane l fetches column and value of
//    nonzero l, two chunks ahead) and, inside a chunk, in batches of 8: 8 * VPL independent
//    LDG.128 per lane (8 loads in all: fewer nonzeros where a lane has several), one partial dot product per
//    nonzero, then a shuffle reduce that halves
//    the number of live partials at every step (4 + 2 + 1 exchanges, then a butterfly over
//    the remaining lanes).  The finished dot products land in the lanes that hold the
//    matching values, so results are stored coalesced.
//  * Row mode of the residue-row kernel: a warp whose rows are long enough (6 nonzeros on average, 16 where the stream has
//    one lane group) and, in short lists and wide rows, about equally long does not form a stream; its lane groups
//    take the rows one each, neighbouring rows side by side (sddmm_rows_one_by_one).  The warp decides from the row lengths it has just loaded (27-point stencil, K = 64:
//    1.26 -> 0.81 ms, rhs rows shared by neighbouring rows now hit in L1; power-law rows,
//    K = 64: 0.51 -> 0.44 ms; graphs with many empty rows keep the stream).
//  * The column indices of a chunk reach the lanes that gather with them through a small
//    double-buffered shared-memory tile (stored once per chunk, read as 16-byte broadcast runs)
//    instead of one shuffle per nonzero: shuffles share the SM's load/store data path with the
//    gathers (block kernel K = 64 on an R-MAT graph 2.29 -> 2.16 ms, power-law residue rows
//    K = 32 0.33 -> 0.26 ms).
//  * sddmm_block: where segments are long (every K but 128: up to 543 nonzeros) a segment gets a
//    warp of its own; chunk loads are then plain coalesced loads without any search and the
//    lhs slice never changes (power-law K = 32: 370 us against 744 us through sddmm_items).
//    Small grids run segments and rows in one launch.
//  * sddmm_pieces: the segments of large operands, cut into pieces that are sorted by their columns (rode_order.cuh).
//  * One-warp CTAs: a CTA's slot is held until its slowest warp finishes.
//
// Per nonzero: 12 B of CSR data/output plus 4*K bytes of rhs (L1/L2/HBM by reuse); per item
// 4*K bytes of lhs per group that touches it.  No atomics, no workspace in global memory.
#include <climits>
#include <mutex>
#include <type_traits>

#include "rode_common.cuh"
#include "rode_order.cuh"

namespace rode {
namespace {

// Mean number of nonzeros per row from which a warp of the residue-row kernel takes its rows one by one, where the stream
// has several lane groups and where it has one.
constexpr int kRowModeMin = 6;
constexpr int kRowModeMin32 = 16;
constexpr int kLoadsInFlight = 8;  // 16-byte loads per lane per batch
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float dot4(const float4 &a, const float4 &b, float acc) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// Where the dense row of a column starts, seen from a lane's base pointer.  Widths known at compile time: shifts and adds.
// Ragged ones: one 32 x 32 -> 64 bit multiply by the row's bytes.  (A signed column times an unsigned row length was a
// 64-bit multiply per gather: R-MAT 21 residue rows K = 96 540 -> 433 us, Pareto 131,072 rows K = 200 297 -> 195.  With four vectors
// per lane, one multiply per four loads, the row mode is faster with the 64-bit form: stencil 64^3 K = 256 400 against 439 us.)
template <bool kMultiply>
__device__ __forceinline__ const float4 *rhs_row(const float4 *lane_base, int c, size_t row_vecs) {
    if constexpr (kMultiply)
        return dense_row(lane_base, static_cast<unsigned>(c), static_cast<unsigned>(row_vecs) * 16u);
    else
        return lane_base + static_cast<size_t>(c) * row_vecs;
}

// p[u] = this lane's share of the dot product of nonzero u of the batch (u = 0..NB-1).
// Returns the complete dot product of nonzero l / (L / NB) - the same value in the L / NB
// lanes that share those bits.  All L lanes of the group named by gmask take part.
template <int L, int NB>
__device__ __forceinline__ float reduce_batch(float (&p)[NB], int l, unsigned gmask) {
    static_assert(NB <= L, "a batch cannot hold more nonzeros than the group has lanes");
#pragma unroll
    for (int keep = NB / 2, w = L / 2; keep >= 1; keep >>= 1, w >>= 1) {
        const bool upper = (l & w) != 0;
#pragma unroll
        for (int i = 0; i < keep; ++i) {
            const float send = upper ? p[i] : p[i + keep];
            const float mine = upper ? p[i + keep] : p[i];
            p[i] = mine + __shfl_xor_sync(gmask, send, w, L);
        }
    }
    float r = p[0];
#pragma unroll
    for (int w = L / (2 * NB); w >= 1; w >>= 1) r += __shfl_xor_sync(gmask, r, w, L);
    return r;
}

// The rows of up to 32 items one by one, 32 / L neighbouring ones side by side, a lane group (L lanes x VPL loads per lane)
// each.  Lane j of the warp holds bounds and row of item j (len = 0: nothing to do); all lanes call.  The columns and values of a
// round's rows, fewer than 32 each, are fetched by one coalesced load per row and array, a round ahead; the columns
// reach the groups, and the dot products the lanes that hold the values, through shared memory.
// `stage` = 2 x 32 / L x 32 words of shared memory.  (Chunks of L nonzeros fetched by each group for itself, and the results
// stored from the lanes of the group, took more wavefronts on the SM's load path, which bounds rows that share columns, and
// more round trips: calls, us, before / after: stencil 128^3 K = 32 524 / 506, K = 64 761 / 727, K = 96 1217 / 1195; 300,000 rows of 0 to 28 K =
// 64 138 / 127; rows of Pareto 2^20 K = 64 431 / 402, of R-MAT 21 K = 200 1181 / 1078.)
// kRagged: the dense rows hold row_vecs_arg <= L * VPL vectors, the rest of the lanes idle.
template <int L, int VPL, int kBatch, bool kRagged>
__device__ __forceinline__ void sddmm_rows_one_by_one(int n_items, int row, int begin, int len, int lane, int row_vecs_arg,
                                                      const int *__restrict__ column_indices,
                                                      const float *__restrict__ values, const float *__restrict__ lhs,
                                                      const float *__restrict__ rhs, float *__restrict__ out, int *stage) {
    constexpr int G = 32 / L;
    const size_t row_vecs = kRagged ? static_cast<unsigned>(row_vecs_arg) : L * VPL;
    const int g = lane / L, l = lane % L;
    const float4 *rhs_lane = reinterpret_cast<const float4 *>(rhs) + l;
    auto inside = [&](int v) { return !kRagged || static_cast<size_t>(l + v * L) < row_vecs; };
    int *s_col = stage;
    float *s_dot = reinterpret_cast<float *>(stage + G * 32);
    // quadruple q of row r, rotated so that the groups read the same one of neighbouring rows from different banks
    auto at = [](int r, int q) { return r * 32 + ((q ^ (r & 7)) << 2); };
    int c_nxt[G];
    float v_nxt[G];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const int b = __shfl_sync(kFull, begin, (j0 + r) & 31), n = __shfl_sync(kFull, len, (j0 + r) & 31);
            c_nxt[r] = 0;
            v_nxt[r] = 0.f;
            if (j0 + r < n_items && lane < n) {
                c_nxt[r] = ld_stream(column_indices + b + lane);
                v_nxt[r] = ld_stream(values + b + lane);
            }
        }
    };
    fetch(0);
#pragma unroll 1
    for (int j0 = 0; j0 < n_items; j0 += G) {
        const int j = (j0 + g) & 31;
        const int my_row = __shfl_sync(kFull, row, j);
        int my_len = __shfl_sync(kFull, len, j);
        if (j0 + g >= n_items) my_len = 0;
        const int longest = __reduce_max_sync(kFull, my_len);
        float val[G];
#pragma unroll
        for (int r = 0; r < G; ++r) {
            s_col[at(r, lane / 4) + lane % 4] = c_nxt[r];
            val[r] = v_nxt[r];
        }
        __syncwarp();
        if (j0 + G < n_items) fetch(j0 + G);
        float4 a[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v)
            a[v] = my_len > 0 && inside(v) ? __ldg(reinterpret_cast<const float4 *>(lhs) + static_cast<size_t>(my_row) * row_vecs + v * L + l)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        constexpr int kQuad = kBatch < 4 ? 4 : kBatch;  // columns read at a time
#pragma unroll 1
        for (int t0 = 0; t0 < longest; t0 += kQuad) {
            int cc[kQuad];
#pragma unroll
            for (int x = 0; x < kQuad; x += 4) {
                int quad[4];
                ld_shared_run<4>(s_col + at(g, (t0 + x) / 4), quad);
#pragma unroll
                for (int u = 0; u < 4; ++u) cc[x + u] = quad[u];
            }
#pragma unroll
            for (int x = 0; x < kQuad; x += kBatch) {
                if (x > 0 && t0 + x >= longest) break;  // warp-uniform
                float4 bb[kBatch][VPL];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        bb[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (t0 + x + u < my_len && inside(v))
                            bb[u][v] = ld_dense(rhs_row<kRagged && VPL < 4>(rhs_lane, cc[x + u], row_vecs) + v * L);
                    }
                }
                float p[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    float d = 0.f;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) d = dot4(a[v], bb[u][v], d);
                    p[u] = d;
                }
                // nonzero u of the batch sits in lanes u * (L / kBatch) ..
                const float r = reduce_batch<L, kBatch>(p, l, kFull);
                if (l % (L / kBatch) == 0) s_dot[g * 32 + t0 + x + l / (L / kBatch)] = r;
            }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const int b = __shfl_sync(kFull, begin, (j0 + r) & 31), n = __shfl_sync(kFull, len, (j0 + r) & 31);
            if (j0 + r < n_items && lane < n) st_stream(out + b + lane, val[r] * s_dot[r * 32 + lane]);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------
// One warp per block segment (used where segments are long, K other than 128: up to 543
// nonzeros).  Chunks of 32 nonzeros are plain coalesced loads without any search, the G groups take every G-th
// nonzero of a chunk, and the lhs slice stays in registers.
//
// Few lanes per dense row with several loads each keep the instruction count low: the reduction over the
// lanes, its selects and shuffles, is paid once per L lanes, the FMAs and loads are the same in every shape.
// A full chunk takes a form without bounds (no predicate and no zero-fill per load).  (Block grids, us: Zipf
// 100003 x 50021 K = 96, 32 lanes x 1 85, 8 x 3 54; Zipf 65536 K = 64, 16 x 1 27, 8 x 2 23; R-MAT 21 K = 96 900 and 700.)
//
// kClaim (grids of one resident wave): a warp starts with the segment of its own index and
// claims further ones from *next_segment; the claim is issued before the segment's work and
// read after it.  One-warp CTAs of one segment each live a few microseconds, and a fifth of the
// warp slots stood empty waiting for the next CTA to be launched into them.
template <int L, int VPL, int U, bool kClaim, bool kRagged>
__device__ __forceinline__ void block_segments(int m1, const int *__restrict__ block_r_ind, const int *__restrict__ st_off,
            const int *__restrict__ row_offsets, const int *__restrict__ column_indices,
            const float *__restrict__ values, const float *__restrict__ lhs, const float *__restrict__ rhs,
            float *__restrict__ out, int *__restrict__ next_segment, int row_vecs_arg, int seg) {
    constexpr int G = 32 / L;
    static_assert(L % U == 0 && U >= 2, "a chunk is a whole number of batches");
    const unsigned row_vecs = kRagged ? static_cast<unsigned>(row_vecs_arg) : L * VPL;
    const unsigned row_bytes = row_vecs * 16u;
    __shared__ __align__(16) int s_col[2][32];  // column indices of the current chunk, two buffers
    int stage_buf = 0;
    const int lane = threadIdx.x;
    const int g = lane / L, l = lane % L;
    // (with four vectors per lane a second form only spills; L = 16 is the form of the large grids)
    constexpr bool kFullPath = VPL <= 3 && L == 8;
    const int pos = l * G + g;  // this lane's nonzero of a chunk: group g holds positions g, g + G, ...
    while (seg < m1) {
    int claimed = INT_MAX;  // never used in arithmetic: the loop test compares it with m1 as it is
    if constexpr (kClaim) {
        if (lane == 0) claimed = static_cast<int>(gridDim.x) + atomicAdd(next_segment, 1);
    }

    const int row = __ldg(block_r_ind + seg);
    const int off = __ldg(st_off + seg);
    const int next = (seg + 1 < m1) ? __ldg(st_off + seg + 1) : INT_MAX;
    const int end = min(__ldg(row_offsets + row + 1), next);

    const float4 *rhs_lane = reinterpret_cast<const float4 *>(rhs) + l;
    auto inside = [&](int v) { return !kRagged || static_cast<unsigned>(l + v * L) < row_vecs; };
    float4 a[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v)
        a[v] = inside(v)
                   ? __ldg(reinterpret_cast<const float4 *>(lhs) + static_cast<size_t>(row) * row_vecs + v * L + l)
                   : make_float4(0.f, 0.f, 0.f, 0.f);

    int c_cur = 0, c_nxt = 0;
    float v_cur = 0.f, v_nxt = 0.f;
    if (off + pos < end) {
        c_cur = ld_stream(column_indices + off + pos);
        v_cur = ld_stream(values + off + pos);
    }
    if (off + 32 + pos < end) {
        c_nxt = ld_stream(column_indices + off + 32 + pos);
        v_nxt = ld_stream(values + off + 32 + pos);
    }
    for (int base = off; base < end; base += 32) {
        int c_pre = 0;
        float v_pre = 0.f;
        if (base + 64 + pos < end) {  // pairs of the chunk after next
            c_pre = ld_stream(column_indices + base + 64 + pos);
            v_pre = ld_stream(values + base + 64 + pos);
        }
        const int cnt = min(32, end - base);
        float mine = 0.f;
        s_col[stage_buf][lane] = c_cur;
        __syncwarp();
        const int *my_cols = &s_col[stage_buf][g * L];
        auto chunk = [&](auto full_tag) {
            constexpr bool kFullChunk = decltype(full_tag)::value;
#pragma unroll
            for (int b = 0; b < L / U; ++b) {
                if (!kFullChunk && b * U * G >= cnt) break;  // warp-uniform
                float4 bb[U][VPL];
                int cc[U];
                ld_shared_run<U>(my_cols + b * U, cc);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float4 *src = dense_row(rhs_lane, static_cast<unsigned>(cc[u]), row_bytes);
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        if constexpr (kFullChunk && !kRagged) {
                            bb[u][v] = ld_dense(src + v * L);
                        } else {
                            bb[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
                            if ((kFullChunk || (b * U + u) * G + g < cnt) && inside(v)) bb[u][v] = ld_dense(src + v * L);
                        }
                    }
                }
                float p[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float d = 0.f;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) d = dot4(a[v], bb[u][v], d);
                    p[u] = d;
                }
                const float r = reduce_batch<L, U>(p, l, kFull);
                // nonzero u of the batch sits in lanes u * (L / U) ..; lane b * U + u of the group wants it
                const float got = (L == U) ? r : __shfl_sync(kFull, r, (l & (U - 1)) * (L / U), L);
                if ((l / U) == b) mine = got;
            }
        };
        if (kFullPath && cnt == 32)
            chunk(std::true_type{});
        else
            chunk(std::false_type{});
        if (pos < cnt) st_stream(out + base + pos, v_cur * mine);
        c_cur = c_nxt;
        v_cur = v_nxt;
        c_nxt = c_pre;
        v_nxt = v_pre;
        stage_buf ^= 1;
    }
    seg = kClaim ? __shfl_sync(kFull, claimed, 0) : INT_MAX;
    }  // segments of this warp
}
// One-warp CTAs per SM: 64 registers while a lane holds two vectors per dense row, 72 beyond.
constexpr int block_ctas(int vpl) { return vpl <= 2 ? 32 : 28; }
template <int L, int VPL, int U, bool kClaim, bool kRagged>
__global__ void __launch_bounds__(32, block_ctas(VPL))
sddmm_block(int m1, const int *__restrict__ block_r_ind, const int *__restrict__ st_off,
            const int *__restrict__ row_offsets, const int *__restrict__ column_indices,
            const float *__restrict__ values, const float *__restrict__ lhs, const float *__restrict__ rhs,
            float *__restrict__ out, int *__restrict__ next_segment, int row_vecs) {
    const int seg = after_chain(blockIdx.x);  // (the first grid of the call)
    chain_begin();
    block_segments<L, VPL, U, kClaim, kRagged>(m1, block_r_ind, st_off, row_offsets, column_indices, values, lhs, rhs, out,
                                               next_segment, row_vecs, seg);
}

// ---------------------------------------------------------------------------------------
// Items as an entry stream, or rows one by one.
//
// kSegments: items are block segments (block_r_ind / st_off); otherwise residue rows
// (residue_r_ind) without a block part.
//
// kRagged: the dense rows hold row_vecs_arg <= L * VPL vectors (any K that is a multiple of 4
// up to 4 * L * VPL); vectors beyond the row's end are not loaded and count as zeros.
//
// LB > 0 (residue rows only): a warp whose rows hold at least row_mode_min nonzeros on average, and are even enough (below),
// does not form a stream; its 32 / LB lane groups (LB lanes x VPLB loads) take the rows one
// each, neighbouring rows side by side.  Long even rows need no balancing over the groups,
// and rows that share columns (stencils, meshes) then find each other's rhs rows in L1; short
// and empty rows (graphs) are better served by the stream, which splits the warp's nonzeros
// evenly.  The warp decides from the row lengths it has just loaded, so no statistic of the
// matrix has to be passed in.
//
// BL > 0 (residue rows only): segments and rows in one launch, for grids so small that the second launch is
// what costs: the first m1 CTAs take a segment each, the others a bundle of rows (Bernoulli 4096^2, K = 32,
// back to back 10.6 -> 8.6 us).
// One-warp CTAs per SM the register allocation must allow: 28 (72 registers).  Left to itself the
// compiler takes 78-80 registers for K = 64 once the chunk staging is in, and the four warps per
// SM that costs outweigh what the staging gains; 64 registers (32 CTAs) spill.
constexpr int kItemsCtas = 28;
template <int L, int VPL, bool kSegments, bool kRagged, int LB, int VPLB, int UB, int BL = 0, int BVPL = 1, int BU = 1>
__global__ void __launch_bounds__(32, (VPL > 1 || BL > 0) ? 24 : kItemsCtas)
sddmm_items(int n_items, int items_per_warp, const int *__restrict__ item_rows, const int *__restrict__ st_off,
            const int *__restrict__ row_offsets, const int *__restrict__ column_indices,
            const float *__restrict__ values, const float *__restrict__ lhs, const float *__restrict__ rhs,
            float *__restrict__ out, int row_vecs_arg, int row_mode_min, int m1, const int *__restrict__ seg_rows, bool first) {
    constexpr int G = 32 / L;
    constexpr int kBatch = kLoadsInFlight / VPL;  // nonzeros per batch
    const size_t row_vecs = kRagged ? static_cast<size_t>(row_vecs_arg) : L * VPL;  // float4 per dense row (K / 4)
    constexpr int kAlign = 4;             // vec_len of the preprocessing
    constexpr int kBlockK = 32;           // k_block of the preprocessing
    // the stream's tables, or the row mode's columns and dot products
    constexpr int kRowWords = LB > 0 ? 2 * 32 / (LB > 0 ? LB : 1) * 32 : 0;
    __shared__ __align__(16) int s_words[kRowWords > 128 ? kRowWords : 128];
    int *const s_end = s_words;           // stream position where item j ends
    int *const s_row = s_words + 32;      // row of item j
    int *const s_col = s_words + 64;      // column indices of the current chunk, two buffers
    int stage_buf = 0;
    const int lane = threadIdx.x;
    const int g = lane / L, l = lane % L;
    const unsigned gmask = group_mask<L>(lane);
    int bundle = kSegments || BL > 0 ? after_chain(blockIdx.x) : after_chain_if(first, blockIdx.x);
    chain_begin();
    if constexpr (BL > 0) {
        if (bundle < m1)
            return block_segments<BL, BVPL, BU, false, kRagged>(m1, seg_rows, st_off, row_offsets, column_indices, values, lhs,
                                                                rhs, out, nullptr, row_vecs_arg, bundle);
        bundle -= m1;
    }
    const long long item0 = static_cast<long long>(bundle) * items_per_warp;
    if (item0 >= n_items) return chain_wait();  // the CTA behind the items

    // ---- descriptors: lane j owns item item0 + j --------------------------------------------
    int row = 0, begin = 0, len = 0;
    if (lane < items_per_warp && item0 + lane < n_items) {
        const int item = static_cast<int>(item0) + lane;
        row = __ldg(item_rows + item);
        if (kSegments) {
            begin = __ldg(st_off + item);
            const int next = (item + 1 < n_items) ? __ldg(st_off + item + 1) : INT_MAX;
            len = min(__ldg(row_offsets + row + 1), next) - begin;
        } else {
            begin = __ldg(row_offsets + row);
            const int end = __ldg(row_offsets + row + 1);
            if (end - begin + (begin % kAlign) < kBlockK) len = end - begin;
        }
    }
    int start = len;  // exclusive prefix sum of len
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(kFull, start, d);
        if (lane >= d) start += up;
    }
    const int total = __shfl_sync(kFull, start, 31);
    const int stop = start;  // inclusive sum = end position
    start -= len;
    if (total == 0) return;
    if constexpr (LB > 0 && !kSegments) {
        static_assert(LB * VPLB == L * VPL || kRagged, "both lane-group shapes must cover the same dense row");
        bool one_by_one = BL > 0;
        if (BL == 0 && total >= row_mode_min * items_per_warp) {  // warp-uniform
            if constexpr (L == 32) {
                // The stream has one lane group and leaves no lane idle.  Row by row a round lasts as long as its longest row
                // (in batches of UB nonzeros), and the lane groups of shorter rows, or of none, wait: taken where the lanes'
                // time stays within a quarter of the stream's.  us, rows only, without / with this test (and 16 x 2 lanes
                // for 8 x 4, which spilled): R-MAT 16 of 43 per row K = 128 26 / 21, Pareto 131,072 rows 80 / 72, 300,000 rows of 0 to 31
                // 296 / 254, stencil 64^3 227 / 203.
                int longest = (len + UB - 1) & ~(UB - 1);
#pragma unroll
                for (int d = 1; d < 32 / LB; d <<= 1) longest = max(longest, __shfl_xor_sync(kFull, longest, d));
                one_by_one = __reduce_add_sync(kFull, longest) * (4 * LB * VPLB) <= total * (5 * L * VPL);
            } else {
                // Short lists give a warp few rows, and there the stream's even split of the nonzeros shortens the
                // dependent chain: then only rows of about equal length are taken one by one (none longer than twice the
                // mean; 27-point stencil of 48^3 rows, us: K = 32 42 -> 33, K = 64 66 -> 50; Zipf 100003 x 50021 K = 64 would go
                // 40 -> 43, R-MAT 17 K = 64 46 -> 48).
                one_by_one = items_per_warp == 32 ||
                             (items_per_warp >= 32 / LB && __reduce_max_sync(kFull, len) * items_per_warp <= 2 * total);
            }
        }
        if (one_by_one)
            return sddmm_rows_one_by_one<LB, VPLB, UB, kRagged>(items_per_warp, row, begin, len, lane, row_vecs_arg, column_indices,
                                                                values, lhs, rhs, out, s_words);
    }
    s_end[lane] = stop;
    s_row[lane] = row;
    const unsigned nonempty = __ballot_sync(kFull, len > 0);
    __syncwarp();

    // ---- this group's contiguous part of the stream: [p0, p1) ----------------------------------
    const int per = (((total + G - 1) / G) + kBatch - 1) & ~(kBatch - 1);
    const int p0 = g * per;
    const int p1 = min(p0 + per, total);
    const int n_chunks = (per + L - 1) / L;  // same for every group

    // stream position p -> (nonzero index, column, value); every lane of the warp calls
    auto fetch = [&](int p, int &e, int &c, float &v) {
        int lo = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const int s = __shfl_sync(kFull, start, lo + step);
            if (s <= p) lo += step;
        }
        const int b0 = __shfl_sync(kFull, begin, lo);
        const int s0 = __shfl_sync(kFull, start, lo);
        e = -1;
        c = 0;
        v = 0.f;
        if (p < p1) {
            e = b0 + (p - s0);
            c = ld_stream(column_indices + e);
            v = ld_stream(values + e);
        }
    };

    const float4 *lhs_lane = reinterpret_cast<const float4 *>(lhs) + l;
    const float4 *rhs_lane = reinterpret_cast<const float4 *>(rhs) + l;
    // vector v of this lane lies inside the dense row
    auto inside = [&](int v) { return !kRagged || static_cast<size_t>(l + v * L) < row_vecs; };
    auto load_lhs = [&](int item, int v) {
        return inside(v) ? __ldg(lhs_lane + static_cast<size_t>(s_row[item]) * row_vecs + v * L)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    };

    // ---- item the group is in, its lhs slice, and the next item's (prefetched) --------------------
    // first item whose end lies beyond p0 = number of items that end at or before p0
    int cur = 0;
#pragma unroll
    for (int gg = 0; gg < G; ++gg) {
        const int cnt = __popc(__ballot_sync(kFull, s_end[lane] <= gg * per));
        if (g == gg) cur = cnt;
    }
    cur = min(cur, 31);
    auto next_nonempty = [&](int after) {  // first non-empty item with index > after, or -1
        const unsigned rest = (after >= 31) ? 0u : (nonempty & (kFull << (after + 1)));
        return __ffs(rest) - 1;
    };
    int cur_end = s_end[cur];
    int nxt = next_nonempty(cur);
    float4 a_cur[VPL], a_nxt[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
        a_cur[v] = load_lhs(cur, v);
        a_nxt[v] = a_cur[v];
        if (nxt >= 0) a_nxt[v] = load_lhs(nxt, v);
    }

    int e_cur, c_cur, e_nxt, c_nxt;
    float v_cur, v_nxt;
    fetch(p0 + l, e_cur, c_cur, v_cur);
    fetch(p0 + L + l, e_nxt, c_nxt, v_nxt);
    int pos = p0;  // stream position of the next nonzero this group multiplies
    for (int ch = 0; ch < n_chunks; ++ch) {
        int e_pre, c_pre;
        float v_pre;
        fetch(p0 + (ch + 2) * L + l, e_pre, c_pre, v_pre);
        const int cnt = min(L, p1 - (p0 + ch * L));  // valid nonzeros of this chunk (may be <= 0)
        float mine = 0.f;
        int *my_stage = s_col + stage_buf * 32 + lane - l;  // this group's region of the chunk buffer
        my_stage[l] = c_cur;
        __syncwarp();  // every group runs the same number of chunks
        stage_buf ^= 1;
#pragma unroll
        for (int b = 0; b < L / kBatch; ++b) {
            if (b * kBatch < cnt) {  // uniform inside the group; no warp-wide shuffles inside
                float4 bb[kBatch][VPL];
                int cc[kBatch];
                ld_shared_run<kBatch>(my_stage + b * kBatch, cc);
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int t = b * kBatch + u;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        bb[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (t < cnt && inside(v))
                            bb[u][v] = ld_dense(rhs_row<kRagged>(rhs_lane, cc[u], row_vecs) + v * L);
                    }
                }
                float p[kBatch];
                if (cur_end - pos >= kBatch) {  // the whole batch lies inside the current item
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        float d = 0.f;
#pragma unroll
                        for (int v = 0; v < VPL; ++v) d = dot4(a_cur[v], bb[u][v], d);
                        p[u] = d;
                    }
                    pos += kBatch;
                } else {
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    if (pos == cur_end && nxt >= 0) {  // the group enters its next item
                        cur = nxt;
                        cur_end = s_end[cur];
                        nxt = next_nonempty(cur);
#pragma unroll
                        for (int v = 0; v < VPL; ++v) {
                            a_cur[v] = a_nxt[v];
                            if (nxt >= 0) a_nxt[v] = load_lhs(nxt, v);
                        }
                    }
                    float d = 0.f;
#pragma unroll
                    for (int v = 0; v < VPL; ++v) d = dot4(a_cur[v], bb[u][v], d);
                    p[u] = d;
                    ++pos;
                }
                }
                const float r = reduce_batch<L, kBatch>(p, l, gmask);
                // nonzero u of the batch sits in lanes u * (L / kBatch) ..; lane b * kBatch + u wants it
                const float got = (L == kBatch) ? r : __shfl_sync(gmask, r, (l & (kBatch - 1)) * (L / kBatch), L);
                if ((l / kBatch) == b) mine = got;
            }
        }
        if (e_cur >= 0) st_stream(out + e_cur, v_cur * mine);
        e_cur = e_nxt;
        c_cur = c_nxt;
        v_cur = v_nxt;
        e_nxt = e_pre;
        c_nxt = c_pre;
        v_nxt = v_pre;
    }
}

// ---------------------------------------------------------------------------------------
// The pieces of the block segments in the order of their columns (rode_order.cuh), a warp per piece, its G lane groups taking
// every G-th nonzero.  One resident wave; a warp claims kPieceRounds pieces at a time, so that the pieces on the GPU are
// neighbours in the list, and has the next piece's first columns and the one after's list entry on their way.
//
// What bounds it: latency (28 to 32 warps of 4 KB in flight each, every batch of 8 loads waiting for its slowest), and from 16 TB/s on the L2.
// Pieces of 64 up to K = 64, of 32 beyond: Pareto 2^20 K = 128, order and pieces, us: P = 16 986, 32 959, against 1612 row by row; K = 64
// P = 32 513, 64 513, 128 564, against 702; R-MAT 23 K = 64 32 2106, 64 1934, 128 2008, against 1972.  (A lane group per
// piece: K = 128 P = 16 929 and R-MAT 21 959 against 876; spilled registers cost 10 to 40 %, so no shape here spills.)
constexpr int kPieceRounds = 4;
constexpr int piece_ctas(int vpl) { return vpl == 1 ? 32 : 28; }
template <int L, int VPL, int U, bool kRagged>
__global__ void __launch_bounds__(32, piece_ctas(VPL))
sddmm_pieces(OrderHead *head, const unsigned long long *__restrict__ list, int capacity,
             const int *__restrict__ column_indices, const float *__restrict__ values, const float *__restrict__ lhs,
             const float *__restrict__ rhs, float *__restrict__ out, int row_vecs_arg) {
    constexpr int G = 32 / L;
    const unsigned row_vecs = kRagged ? static_cast<unsigned>(row_vecs_arg) : L * VPL;
    const unsigned row_bytes = row_vecs * 16u;
    const int lane = threadIdx.x;
    const int g = lane / L, l = lane % L;
    const int pos = l * G + g;  // this lane's nonzero of a chunk
    __shared__ __align__(16) int s_col[2][32];
    int stage_buf = 0;
    chain_begin();
    // position of the piece two ahead: round `r2` of bundle `b2`.  Behind the wait, as is whatever is claimed from the head: the
    // list is not read before it is complete.
    int b2 = after_chain(blockIdx.x), r2 = 0;
    int total = 0;
#pragma unroll
    for (int i = 0; i < kOrderBuckets / 32; ++i) total += ld_behind_wait(&head->counts[lane + 32 * i]);
    total = min(__reduce_add_sync(kFull, total), capacity);
    const int bundles = (total + kPieceRounds - 1) / kPieceRounds;
    const float4 *lhs_lane = reinterpret_cast<const float4 *>(lhs) + l;
    const float4 *rhs_lane = reinterpret_cast<const float4 *>(rhs) + l;
    auto inside = [&](int v) { return !kRagged || static_cast<unsigned>(l + v * L) < row_vecs; };
    auto entry = [&](int bundle, int round) {
        const long long i = static_cast<long long>(bundle) * kPieceRounds + round;
        return bundle < bundles && i < total ? __ldcg(list + i) : 0ull;
    };
    if (b2 >= bundles) return;
    int claimed = INT_MAX;
    auto claim = [&]() {
        if (lane == 0) claimed = static_cast<int>(gridDim.x) + atomicAdd(&head->claim, 1);
    };
    claim();
    auto next_entry = [&]() {
        const unsigned long long e = entry(b2, r2);
        if (++r2 == kPieceRounds) {
            r2 = 0;
            b2 = __shfl_sync(kFull, claimed, 0);
            claim();
        }
        return e;
    };
    auto fetch = [&](const Piece &p, int at, int &c, float &v) {
        c = 0;
        v = 0.f;
        if (at < p.len) {
            c = ld_stream(column_indices + p.off + at);
            v = ld_stream(values + p.off + at);
        }
    };
    Piece p = unpack_piece(next_entry());
    unsigned long long e1 = next_entry();
    int c_nxt;
    float v_nxt;
    fetch(p, pos, c_nxt, v_nxt);
    while (true) {
        if (p.len == 0) return;  // behind the end of the list
        float4 a[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v)
            a[v] = inside(v) ? __ldg(lhs_lane + static_cast<size_t>(p.row) * row_vecs + v * L) : make_float4(0.f, 0.f, 0.f, 0.f);
        const Piece q = unpack_piece(e1);
        int c_q;
        float v_q;
        fetch(q, pos, c_q, v_q);
        e1 = next_entry();
        for (int base = 0; base < p.len; base += 32) {
            const int c = c_nxt;
            const float val = v_nxt;
            fetch(p, base + 32 + pos, c_nxt, v_nxt);
            const int cnt = p.len - base;  // of this chunk, at most 32 count
            float mine = 0.f;
            s_col[stage_buf][lane] = c;
            __syncwarp();
            const int *my_cols = &s_col[stage_buf][g * L];
            stage_buf ^= 1;
#pragma unroll
            for (int b = 0; b < L / U; ++b) {
                if (b * U * G >= cnt) break;  // warp-uniform
                float4 bb[U][VPL];
                int cc[U];
                ld_shared_run<U>(my_cols + b * U, cc);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float4 *src = dense_row(rhs_lane, static_cast<unsigned>(cc[u]), row_bytes);
#pragma unroll
                    for (int v = 0; v < VPL; ++v) {
                        bb[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if ((b * U + u) * G + g < cnt && inside(v)) bb[u][v] = ld_dense(src + v * L);
                    }
                }
                float d[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    // (two vectors per lane are added as two lanes with one each would: the same bits as the kernel without order)
                    d[u] = dot4(a[0], bb[u][0], 0.f);
#pragma unroll
                    for (int v = 1; v < VPL; ++v) d[u] += dot4(a[v], bb[u][v], 0.f);
                }
                const float r = reduce_batch<L, U>(d, l, kFull);
                const float got = (L == U) ? r : __shfl_sync(kFull, r, (l & (U - 1)) * (L / U), L);
                if ((l / U) == b) mine = got;
            }
            if (pos < cnt) st_stream(out + p.off + base + pos, val * mine);
        }
        p = q;
        c_nxt = c_q;
        v_nxt = v_q;
    }
}

// ---------------------------------------------------------------------------------------
// Claim counter of the persistent block grid.  The SDDMM entry points carry no workspace, so the
// counters live in a fixed array of the library's device image: kClaimSlots slots of 64 ints
// (32 KB on every GPU that loads the library).  A slot belongs to one (device, stream1, stream2)
// for the life of the process: calls on the same streams are ordered by them and may share
// their counter, calls on other streams get other slots; when all slots are taken a call simply
// runs one CTA per segment.  Nothing is allocated.  What keeps two kernels off one counter:
//   * streams are told apart by number, not by handle (stream_id): a destroyed stream's handle is given to a new one
//     while its last kernels may still run;
//   * the reset and the kernel that follows it are enqueued under one lock (ClaimCounter holds it), so that host
//     threads that share a stream cannot come between them;
//   * a call that is being captured gets no counter: its graph may be replayed on any stream, next to graphs
//     captured on the same one.
constexpr int kClaimSlots = 128;
constexpr int kClaimInts = 64;
static __device__ __align__(256) int g_claim_counters[kClaimSlots * kClaimInts];
std::mutex g_claim_mutex;

struct ClaimCounter {
    int *ptr = nullptr;  // null: run one CTA per segment
    std::unique_lock<std::mutex> enqueue;

    int acquire(cudaStream_t s1, cudaStream_t s2) {
        struct Key {
            int dev;
            unsigned long long id1, id2;
        };
        static Key keys[kClaimSlots];
        static int n_keys = 0;
        static int *base[64] = {nullptr};  // device address of the array, per device
        if (is_capturing(s1) || is_capturing(s2)) return RODE_OK;
        Key key = {0, stream_id(s1), stream_id(s2)};
        RODE_CUDA_TRY(cudaGetDevice(&key.dev));
        if (key.dev < 0 || key.dev >= 64) return RODE_OK;
        enqueue = std::unique_lock<std::mutex>(g_claim_mutex);
        if (base[key.dev] == nullptr) {
            void *p = nullptr;
            RODE_CUDA_TRY(cudaGetSymbolAddress(&p, g_claim_counters));
            base[key.dev] = static_cast<int *>(p);
        }
        int slot = -1;
        for (int i = 0; i < n_keys; ++i)
            if (keys[i].dev == key.dev && keys[i].id1 == key.id1 && keys[i].id2 == key.id2) slot = i;
        if (slot < 0 && n_keys < kClaimSlots) {
            slot = n_keys++;
            keys[slot] = key;
        }
        if (slot >= 0) ptr = base[key.dev] + slot * kClaimInts;
        return RODE_OK;
    }
};

// Items per warp: up to `cap` when that still gives every SM `waves` waves of warps, fewer otherwise.  Rows whose warp
// holds several lane groups want two waves, because a warp then brings its own balance (us with four waves -> two: Zipf 65536
// K = 32 22.8 -> 18.8, K = 64 28.9 -> 25.6, Zipf 100003 x 50021 K = 64 42.5 -> 39.7);
// a warp of one group wants four (R-MAT 17 K = 96 95 us with two, 92 with four; K = 128 90 and 85).
int items_per_warp(int n_items, int cap, int waves) {
    const long long slots = waves * 24LL * sm_count();
    long long per = (n_items + slots - 1) / slots;
    per = per < 1 ? 1 : (per > cap ? cap : per);
    return static_cast<int>(per);
}

// A lane group of L lanes x VPL vectors, with U nonzeros per batch.
template <int L_, int VPL_, int U_>
struct Shape {
    static constexpr int L = L_, VPL = VPL_, U = U_;
};
// Lengths of the pieces (rode_order.cuh) by the number of vectors of a dense row.
constexpr int piece_len(int row_vecs) { return row_vecs <= 16 ? 64 : 32; }
// When an order pays: an rhs beyond the L2, enough segments to pay for it, and columns that it helps (rode_order.cuh).  With wide
// rows the pieces are also the better form for the segments of skewed matrices (whole calls, row by row / ordered, us: R-MAT 21
// K = 128 1240 / 1189, K = 256 3106 / 2760, R-MAT 20 of 64 per row K = 128 1961 / 1910; K = 64 671 / 720, K = 96 1088 / 1229).
// Uniform columns, us: K = 32 512 MB Pareto of mean 16 1912 / 1495, 128 MB 347 / 345 and of mean 8 228 / 241; K = 64 256 MB 1090 / 919
// (mean 32), 364 / 368 (mean 8, 31,336 segments); Zipf 671,008 x 929,297 of mean 40 K = 64 800 / 517, K = 128 1797 / 942; K = 128 128 MB
// Pareto 394 / 355; 10,953 segments Zipf of mean 16 K = 64 159 / 156, K = 96 265 / 241.  Bands: 1M rows of 60 in 3000 columns K = 128 1775 / 1921.
//
// An order also needs references to bring together (rows of one length, uniform columns, references per column, row by row / ordered): K = 32
// 2 80 / 95 (rows of 64), 78 / 85 (of 128), 4 214 / 174, 145 / 136; K = 64 2 69 / 83 and 77 / 89 (of 40), 3 98 / 116 and 129 / 130, 4 129 /
// 148 and 171 / 159, 6 207 / 212 (of 64), 8 248 / 214 (of 128); K = 96 2 128 / 138 (of 40), in long rows (of 2000; 8388 and 12,580
// segments) 4 158 / 171, K = 80 4 150 / 169, 6 205 / 212, but Zipf of mean 4 and 8, K = 96, 370 / 349 and 581 / 445; K = 128 1 80 / 85 and 79 / 89 (of 64 and
// 128), 2 157 / 139 (of 96); Pareto 2^21 K = 32 of mean 4 323 / 339, of 8 480 / 474, 2^20 K = 128 of mean 2 234 / 245, of 4 403 / 398.
bool order_pays(int verdict, long long M, long long m1, long long n, int k, long long nnz) {
    const bool enough = m1 >= 1 << 15 || (k > 64 && m1 >= kOrderMinSegments && nnz >= kOrderLongRows * m1);
    const bool shared = k > 96 ? nnz >= 2 * n : m1 < 1 << 15 ? nnz >= 6 * n : 2 * nnz >= 7 * n;
    return verdict >= 0 && M < kPieceMaxRows && enough && shared && n * k * 4 >= (k > 96 ? 128ll << 20 : 160ll << 20) &&
           ((verdict & kOrderKind) == kOrderHelps || ((verdict & kOrderKind) == kOrderSkewed && k > 96));
}
// The block segments through sddmm_pieces.
template <int L, int VPL, int U>
int launch_pieces(const Ordering &ord, int row_vecs, const int *col, const float *values, const float *lhs,
                  const float *rhs, float *out, cudaStream_t s) {
    const dim3 resident(piece_ctas(VPL) * sm_count());
    const auto kernel = row_vecs == L * VPL ? sddmm_pieces<L, VPL, U, false> : sddmm_pieces<L, VPL, U, true>;
    RODE_CUDA_TRY(launch_chained(kernel, resident, dim3(32), s, true, ord.head, ord.list<64>(), ord.capacity, col, values, lhs, rhs,
                                 out, row_vecs));
    RODE_CHECK_LAUNCH("rode::sddmm_pieces");
    return RODE_OK;
}
// L lanes x VPL vectors for the streams; shapes of the segments (a warp each: kLongSegments, else up to 32 segments per warp
// run as a stream, and Block serves the small grids) and of the row mode of the residue kernel; Claimed: of the persistent
// grids of segments.
template <int L, int VPL, typename Block, typename Rows, bool kRagged, bool kLongSegments, typename Claimed = Block>
int launch_k(int m1, int m2, int k, const int *block_r_ind, const int *residue_r_ind,
             const int *st_off, const int *row_offsets, const int *col, const float *values, const float *lhs,
             const float *rhs, float *out, cudaStream_t s1, cudaStream_t s2, const Ordering *ord) {
    constexpr int BL = Block::L, BVPL = Block::VPL, BU = Block::U;
    constexpr int RL = Rows::L, RVPL = Rows::VPL, RU = Rows::U;
    const int row_vecs = k / 4;
    // nonzeros per row from which a warp takes its rows one by one: where the stream form has one lane group only
    // it balances nothing, but short rows still lose more to the idle lane groups of the row form (R-MAT 21,
    // K = 96: 0.56 ms as a stream, 0.65 to 0.68 ms row by row; stencil, K = 128: 1.78 against 1.57 ms)
    const int row_mode_min = L == 32 ? kRowModeMin32 : kRowModeMin;
    {
        // (a row per lane group of the segments' shape: on such matrices most residue rows have had their tail taken by a
        // segment.  16 x 2 lanes for the rows of K = 100: Zipf 16384 28.0 -> 28.8 us, R-MAT 15, which then takes two launches,
        // 32.8 -> 39.1)
        constexpr int kRowU = BL == RL && BVPL == RVPL ? RU : BU;
        const int per = 32 / BL;
        const long long ctas = static_cast<long long>(m1) + (m2 + per - 1) / per;
        // (a warp per 32-long segment, K = 128, pays while they all fit at once: Bernoulli 4096^2 13.5 us with the two
        // kernels, 14.7 in one; 2000^2 12.3 and 10.3)
        if (ord == nullptr && m1 > 0 && m2 > 0 && s1 == s2 && ctas <= (kLongSegments ? 4LL : 1LL) * 24 * sm_count()) {
            RODE_CUDA_TRY(launch_chained(sddmm_items<L, VPL, false, kRagged, BL, BVPL, kRowU, BL, BVPL, BU>,
                                         dim3(static_cast<unsigned>(ctas)), dim3(32), s1, true, m2, per, residue_r_ind, st_off,
                                         row_offsets, col, values, lhs, rhs, out, row_vecs, row_mode_min, m1, block_r_ind, true));
            RODE_CHECK_LAUNCH("rode::sddmm_items<segments and rows>");
            return RODE_OK;
        }
    }
    if (ord != nullptr) {
        const auto order = piece_len(row_vecs) == 64 ? launch_order<64> : launch_order<32>;
        if (int rc = order(*ord, m1, row_offsets, col, block_r_ind, st_off, s1)) return rc;
        const auto pieces = row_vecs <= 8 ? launch_pieces<8, 1, 8> : row_vecs <= 16 ? launch_pieces<16, 1, 8>
                            : row_vecs <= 24 ? launch_pieces<8, 3, 2> : row_vecs <= 32 ? launch_pieces<16, 2, 4>
                                                                                       : launch_pieces<32, 2, 4>;
        if (int rc = pieces(*ord, row_vecs, col, values, lhs, rhs, out, s1)) return rc;
    } else if (m1 > 0) {
        if constexpr (kLongSegments) {
            const int resident = block_ctas(Claimed::VPL) * sm_count();
            ClaimCounter claim;  // holds its lock until the kernel is enqueued
            if (m1 > 16 * resident) {  // from about 16 segments per warp on it pays
                if (int rc = claim.acquire(s1, s2)) return rc;
            }
            if (claim.ptr != nullptr) {
                RODE_CUDA_TRY(cudaMemsetAsync(claim.ptr, 0, sizeof(int), s1));
                RODE_CUDA_TRY(launch_chained(sddmm_block<Claimed::L, Claimed::VPL, Claimed::U, true, kRagged>, dim3(resident), dim3(32),
                                             s1, true, m1, block_r_ind, st_off, row_offsets, col, values, lhs, rhs, out, claim.ptr,
                                             row_vecs));
            } else {
                RODE_CUDA_TRY(launch_chained(sddmm_block<BL, BVPL, BU, false, kRagged>, dim3(m1), dim3(32), s1, true, m1, block_r_ind,
                                             st_off, row_offsets, col, values, lhs, rhs, out, nullptr, row_vecs));
            }
            RODE_CHECK_LAUNCH("rode::sddmm_block");
        } else {
            const int per = items_per_warp(m1, 32, 4);
            RODE_CUDA_TRY(launch_chained(sddmm_items<L, VPL, true, kRagged, 0, 1, 1>, dim3((m1 + per - 1) / per), dim3(32), s1, true,
                                         m1, per, block_r_ind, st_off, row_offsets, col, values, lhs, rhs, out, row_vecs, 0, 0,
                                         nullptr, true));
            RODE_CHECK_LAUNCH("rode::sddmm_items<segments>");
        }
    }
    if (m2 > 0) {
        int per = items_per_warp(m2, 32, L < 32 ? 2 : 4);
        // whole rounds of the row mode (30,000 rows of 25, 3 -> 4 rows per warp: K = 128 28.6 -> 25.3 us, K = 96 28.8 -> 22.6)
        if (L == 32 && per > 1) per = (per + 32 / RL - 1) / (32 / RL) * (32 / RL);
        RODE_CUDA_TRY(launch_chained(sddmm_items<L, VPL, false, kRagged, RL, RVPL, RU>, dim3((m2 + per - 1) / per + 1), dim3(32), s2,
                                     true, m2, per, residue_r_ind, nullptr, row_offsets, col, values, lhs, rhs, out, row_vecs,
                                     row_mode_min, 0, nullptr, !(m1 > 0 && s1 == s2)));
        RODE_CHECK_LAUNCH("rode::sddmm_items<rows>");
    }
    return RODE_OK;
}

int sddmm(int m1, int m2, int k, const int *block_r_ind, const int *residue_r_ind, const int *st_off, const int *row_offsets,
          const int *column_indices, const float *values, const float *lhs, const float *rhs, float *out, cudaStream_t stream1,
          cudaStream_t stream2, const Ordering *ord) {
    if (m1 < 0 || m2 < 0) return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: m1, m2 must be >= 0");
    if (k <= 0 || k % 4 != 0 || k > 256)
        return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: k = %d unsupported (a multiple of 4, at most 256)", k);
    if (m1 == 0 && m2 == 0) return RODE_OK;
    if (!row_offsets || !column_indices || !values || !lhs || !rhs || !out)
        return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: null array");
    if (m1 > 0 && (!block_r_ind || !st_off)) return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: null block metadata");
    if (m2 > 0 && !residue_r_ind) return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: null residue metadata");
    if (!aligned_to(lhs, 16) || !aligned_to(rhs, 16))
        return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: lhs and rhs must be 16-byte aligned");
#define RODE_SDDMM_LAUNCH(...)                                                                                   \
    launch_k<__VA_ARGS__>(m1, m2, k, block_r_ind, residue_r_ind, st_off, row_offsets, column_indices, values, lhs, rhs, \
                          out, stream1, stream2, ord)
    // The narrowest lane group that covers the dense row; where it does not fit exactly the lanes beyond the
    // row's end idle (ragged).  (One form of 32 lanes x 2 vectors for all of those widths took 0.209 ms on
    // the 100003 x 50021 Zipf matrix at K = 96, the 32 x 1 form 0.117 ms.)  The decomposition that goes with
    // K = 128 has 32-long segments, all others 512-long ones.
    const int vecs = k / 4;
    // (K = 64: 8 x 2 takes fewer instructions, Pareto 2^18 block grid 119 -> 103 us, Zipf 65536 29 -> 23 us; matrices of
    // millions of rows lose 4 % with it, each of its loads asking for half of the row, R-MAT 23 3.16 -> 3.29 ms: persistent
    // grids keep 16 x 1 in the form without a separate full chunk.)
    if (vecs == 8) return RODE_SDDMM_LAUNCH(8, 1, Shape<8, 1, 8>, Shape<8, 1, 8>, false, true);
    if (vecs == 16) return RODE_SDDMM_LAUNCH(16, 1, Shape<8, 2, 4>, Shape<8, 2, 4>, false, true, Shape<16, 1, 8>);
    if (vecs == 32) return RODE_SDDMM_LAUNCH(32, 1, Shape<8, 4, 2>, Shape<16, 2, 4>, false, false);
    if (vecs < 8) return RODE_SDDMM_LAUNCH(8, 1, Shape<8, 1, 8>, Shape<8, 1, 8>, true, true);
    if (vecs < 16) return RODE_SDDMM_LAUNCH(16, 1, Shape<8, 2, 4>, Shape<8, 2, 4>, true, true);
    if (vecs <= 24) return RODE_SDDMM_LAUNCH(32, 1, Shape<8, 3, 4>, Shape<8, 3, 2>, true, true);
    if (vecs < 32) return RODE_SDDMM_LAUNCH(32, 1, Shape<8, 4, 2>, Shape<16, 2, 4>, true, true);
    return RODE_SDDMM_LAUNCH(32, 2, Shape<16, 4, 2>, Shape<16, 4, 2>, true, true);
#undef RODE_SDDMM_LAUNCH
}

// The verdict of rode_order_verdict (rode_order.cuh says what its values mean).
constexpr int kJudgeThreads = 1024;
constexpr int kJudgeSamples = 4 * kJudgeThreads;
constexpr int kJudgeSlots = 2 * kJudgeSamples;
__global__ void __launch_bounds__(kJudgeThreads)
judge_columns(int m1, int n_cols, long long nnz, const int *__restrict__ row_offsets,
              const int *__restrict__ column_indices, const int *__restrict__ block_r_ind, int *__restrict__ verdict) {
    __shared__ int s_slot[kJudgeSlots];
    __shared__ int s_repeats;
    __shared__ float s_span[kJudgeThreads / 32], s_seg_span[kJudgeThreads / 32];
    const int t = threadIdx.x;
    int c[kJudgeSamples / kJudgeThreads];
    const int seg = static_cast<int>(static_cast<long long>(t) * m1 / kJudgeThreads);
    const int row = __ldg(block_r_ind + seg);
    // segments of the row, up to two on either side of this one: from five on it is narrow enough
    int segs = 1;
#pragma unroll
    for (int d = -2; d <= 2; ++d)
        if (d != 0 && seg + d >= 0 && seg + d < m1 && __ldg(block_r_ind + seg + d) == row) ++segs;
    const int begin = __ldg(row_offsets + row), end = __ldg(row_offsets + row + 1);
#pragma unroll
    for (int i = 0; i < kJudgeSamples / kJudgeThreads; ++i) {
        const unsigned at = static_cast<unsigned>(i * kJudgeThreads + t);
        // (somewhere in the sample's share of the nonzeros: at even distances rows of equal length would be asked at the
        // same place, where ascending columns repeat without being popular)
        const unsigned within = (at * 2654435761u) >> 16;
        c[i] = __ldg(column_indices + ((static_cast<long long>(at) << 16) + within) * nnz /
                                          (static_cast<long long>(kJudgeSamples) << 16));
    }
    float span = 0.f;
    if (end > begin) span = fabsf(static_cast<float>(__ldg(column_indices + end - 1)) - static_cast<float>(__ldg(column_indices + begin)));
    for (int i = t; i < kJudgeSlots; i += kJudgeThreads) s_slot[i] = -1;
    if (t == 0) s_repeats = 0;
    __syncthreads();
    int repeats = 0;
#pragma unroll
    for (int i = 0; i < kJudgeSamples / kJudgeThreads; ++i) {
        int at = static_cast<int>(static_cast<unsigned>(c[i]) * 2654435761u / (0x100000000ull / kJudgeSlots));
        while (true) {  // ends: there are fewer samples than slots
            const int old = atomicCAS(&s_slot[at], -1, c[i]);
            if (old == -1) break;
            if (old == c[i]) {
                ++repeats;
                break;
            }
            at = (at + 1) % kJudgeSlots;
        }
    }
    repeats = __reduce_add_sync(0xffffffffu, repeats);
    float seg_span = span / static_cast<float>(segs);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        span += __shfl_xor_sync(0xffffffffu, span, d);
        seg_span += __shfl_xor_sync(0xffffffffu, seg_span, d);
    }
    if (t % 32 == 0) {
        atomicAdd(&s_repeats, repeats);
        s_span[t / 32] = span;
        s_seg_span[t / 32] = seg_span;
    }
    __syncthreads();
    if (t == 0) {
        float sum = 0.f, seg_sum = 0.f;
        for (int w = 0; w < kJudgeThreads / 32; ++w) {
            sum += s_span[w];
            seg_sum += s_seg_span[w];
        }
        const float of_columns = seg_sum / (static_cast<float>(kJudgeThreads) * n_cols);
        const float uniform = 0.5f * kJudgeSamples * kJudgeSamples / n_cols;
        const bool skewed = s_repeats > 8.f * uniform + 16.f;
        const bool local = sum / kJudgeThreads < n_cols / 32.f;
        *verdict = (local ? kOrderLocal : skewed ? kOrderSkewed : kOrderHelps) |
                   (of_columns < 0.75f ? kOrderNarrow : of_columns > 0.9f ? kOrderWide : 0);
    }
}

size_t piece_bytes(long long m1, long long nnz, int row_vecs) {
    return piece_len(row_vecs) == 64 ? ordering_bytes<64>(m1, nnz) : ordering_bytes<32>(m1, nnz);
}

}  // namespace
}  // namespace rode

extern "C" {

int rode_sddmm_f32(int m1, int m2, int n, int k, const int *block_r_ind, const int *residue_r_ind, const int *st_off,
                   const int *row_offsets, const int *column_indices, const float *values, const float *lhs, const float *rhs,
                   float *out, rode_stream_t stream1, rode_stream_t stream2) {
    (void)n;
    return rode::sddmm(m1, m2, k, block_r_ind, residue_r_ind, st_off, row_offsets, column_indices, values, lhs, rhs, out, stream1,
                       stream2, nullptr);
}

int rode_order_verdict(int m1, int n_cols, long long nnz, const int *row_offsets, const int *column_indices,
                       const int *block_r_ind, int *in_range, int *verdict, rode_stream_t stream) {
    using namespace rode;
    if (in_range == nullptr || m1 < 0 || n_cols < 0 || nnz < 0)
        return fail(RODE_ERR_INVALID_ARGUMENT, "order_verdict: bad argument");
    *in_range = nnz > 0 && m1 >= kOrderMinSegments && n_cols >= kOrderMinColumns ? 1 : 0;
    if (*in_range == 0 || verdict == nullptr) return RODE_OK;
    if (!row_offsets || !column_indices || !block_r_ind) return fail(RODE_ERR_INVALID_ARGUMENT, "order_verdict: null array");
    judge_columns<<<1, kJudgeThreads, 0, stream>>>(m1, n_cols, nnz, row_offsets, column_indices, block_r_ind, verdict);
    RODE_CHECK_LAUNCH("rode::judge_columns");
    return RODE_OK;
}

int rode_sddmm_order_pays(int verdict, int M, int m1, int n, int k, long long nnz) {
    return rode::order_pays(verdict, M, m1, n, k, nnz) ? 1 : 0;
}

int rode_sddmm_workspace_bytes(int m1, int k, long long nnz, size_t *bytes) {
    using namespace rode;
    if (bytes == nullptr || m1 < 0 || k <= 0 || nnz < 0)
        return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm_workspace_bytes: bad argument");
    *bytes = piece_bytes(m1, nnz, (k + 3) / 4);
    return RODE_OK;
}

int rode_sddmm_f32_ordered(int M, int m1, int m2, int n, int k, long long nnz, const int *block_r_ind, const int *residue_r_ind,
                           const int *st_off, const int *row_offsets, const int *column_indices, const float *values,
                           const float *lhs, const float *rhs, float *out, void *workspace, size_t workspace_bytes,
                           rode_stream_t stream1, rode_stream_t stream2) {
    using namespace rode;
    if (M < 0 || nnz < 0) return fail(RODE_ERR_INVALID_ARGUMENT, "sddmm: M, nnz must be >= 0");
    Ordering ord = {};
    // (the cuts of a segment are multiples of up to 64 beyond its ends)
    const bool ordered = workspace != nullptr && m1 > 0 && n > 0 && k > 0 && nnz > 0 && nnz < INT_MAX - 256 && M < kPieceMaxRows;
    if (ordered) {
        const size_t need = piece_bytes(m1, nnz, (k + 3) / 4);
        if (workspace_bytes < need)
            return fail(RODE_ERR_WORKSPACE, "sddmm: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
        if (!aligned_to(workspace, 16)) return fail(RODE_ERR_WORKSPACE, "sddmm: workspace must be 16-byte aligned");
        ord.head = static_cast<OrderHead *>(workspace);
        ord.capacity = static_cast<int>(max_pieces(m1, nnz, piece_len((k + 3) / 4)));
        ord.n_cols = n;
    }
    return rode::sddmm(m1, m2, k, block_r_ind, residue_r_ind, st_off, row_offsets, column_indices, values, lhs, rhs, out, stream1,
                       stream2, ordered ? &ord : nullptr);
}

}  // extern "C"
