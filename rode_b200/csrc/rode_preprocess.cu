// RoDe row-decomposition preprocessing on the GPU, plus its host twin.
//
// Specification: the single-thread loop RoDe_preprocess_cpu of the reference
// (Preprocess_opt/_preprocess.cu:340-373).  For row i with pad = row_ptr[i] % vec_len and
// aligned length A = len + pad:
//     A >  seg_len : segments (i, row_ptr[i]), (i, row_ptr[i] - pad + j*seg_len), j = 1, 2, ...
//     last piece   : one more segment if it is >= k_block long; residue row if it is not a
//                    multiple of k_block.
// The reference's device version (count kernel _preprocess.cu:244-274, two CUB scans
// :330-334, fill kernel :275-322) keeps its prefix sums in the output arrays and overwrites
// them in place across thread blocks.  Here the prefix sums live in a separate scratch
// array, the totals of each tile of rows: count_tiles writes them, fill_tiles adds up those before its
// tile and writes the outputs; a matrix of a few tiles needs fill_tiles only.
#include <climits>
#include <mutex>

#include <cooperative_groups.h>

#include "rode_common.cuh"

namespace rode {
namespace {

constexpr int kThreads = 256;
constexpr int kTile = 2048;    // rows per CTA
constexpr int kWarps = kThreads / 32;
constexpr int kShortRow = 8;   // rows of up to so many segments are written by one thread, others by a warp
// Scratch: running sums of the tiles, one int2 each.

// The three parameters of the decomposition.  kPow2 = all of them are powers of two (every
// parameter set the reference uses: (512, 32, 4) and (32, 32, 4)): quotients and remainders
// are then shifts and masks.  With run-time divisors the five integer divisions per row made
// the count and fill kernels instruction-bound (about 150 instructions per row).
struct Params {
    int seg_len, k_block, vec_len;
    int seg_shift;  // log2(seg_len) when kPow2
};
template <bool kPow2>
__device__ __forceinline__ int mod_vec(int x, const Params &p) {
    return kPow2 ? (x & (p.vec_len - 1)) : (x % p.vec_len);
}
template <bool kPow2>
__device__ __forceinline__ int mod_block(int x, const Params &p) {
    return kPow2 ? (x & (p.k_block - 1)) : (x % p.k_block);
}

// Number of block segments and residue flag of one row (closed form of the spec loop;
// valid because seg_len % k_block == 0).
template <bool kPow2>
__device__ __forceinline__ void row_counts(int off, int next, const Params &p, int &bn, int &rn) {
    const int a = next - off + mod_vec<kPow2>(off, p);
    if constexpr (kPow2) {
        // one form for both cases of the spec loop: with a <= seg_len the quotient is 0 and the
        // remainder is a itself, except a == seg_len, where quotient 1 + remainder 0 gives the same
        // single segment; and (a % seg_len) % k_block == a % k_block because k_block divides seg_len
        // (a / seg_len, plus one where the remainder reaches k_block = one division of a sum)
        bn = static_cast<int>((static_cast<unsigned>(a) + (p.seg_len - p.k_block)) >> p.seg_shift);
        rn = (a & (p.k_block - 1)) != 0 ? 1 : 0;
    } else if (a > p.seg_len) {
        const int rest = a % p.seg_len;
        bn = a / p.seg_len + (rest >= p.k_block ? 1 : 0);
        rn = rest % p.k_block != 0 ? 1 : 0;
    } else {
        bn = a >= p.k_block ? 1 : 0;
        rn = a % p.k_block != 0 ? 1 : 0;
    }
}

// M == 0: no tile, only the counts and the sentinel.
__global__ void empty_matrix(const int *__restrict__ row_ptr, int *__restrict__ st_off, int *__restrict__ n_blk,
                             int *__restrict__ n_res, bool write_sentinel) {
    n_blk[0] = 0;
    n_res[0] = 0;
    if (write_sentinel) st_off[0] = row_ptr[0];
}

// Segments of one row: j = first, first + step, ...
template <bool kPow2>
__device__ __forceinline__ void write_row(const Params &p, int first, int step, int row, int off, int cnt,
                                          int *__restrict__ dst_row, int *__restrict__ dst_off) {
    const int aligned = off - mod_vec<kPow2>(off, p);
    for (int j = first; j < cnt; j += step) {
        dst_row[j] = row;
        dst_off[j] = j == 0 ? off : aligned + j * p.seg_len;
    }
}

// The rows of one warp: kVecs x 128 of them, unit i of a lane being rows row0 + 128 i .. + 3, in registers
// from 16-byte loads that are all in flight together.
constexpr int kUnit = 128;
constexpr int kVecs = kTile / kThreads / 4;
constexpr int kWarpRows = kUnit * kVecs;
template <bool kPow2>
struct WarpRows {
    int o[kVecs][4];
    int after;  // offset of the row behind the last one
    int row0;
    bool wide;  // warp-uniform: all rows exist and the row pointer is 16-byte aligned

    __device__ __forceinline__ void load(int M, const int *__restrict__ row_ptr, int warp_row0, int lane) {
        row0 = warp_row0 + lane * 4;
        wide = reinterpret_cast<size_t>(row_ptr) % 16 == 0 && warp_row0 + kWarpRows <= M;
        if (wide) {
#pragma unroll
            for (int i = 0; i < kVecs; ++i) {
                const int4 v = __ldg(reinterpret_cast<const int4 *>(row_ptr + row0 + kUnit * i));
                o[i][0] = v.x;
                o[i][1] = v.y;
                o[i][2] = v.z;
                o[i][3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kVecs; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k) o[i][k] = __ldg(row_ptr + min(row0 + kUnit * i + k, M));
        }
        after = __ldg(row_ptr + min(warp_row0 + kWarpRows, M));
    }
    int packed[kVecs][4];  // 2 * segments + residue flag of each row, set by sums()
    // The four rows of unit i; rows at or beyond M count as nothing.
    __device__ __forceinline__ void count(const Params &p, int M, int lane, int i) {
        const int behind = i + 1 < kVecs ? o[i + 1 < kVecs ? i + 1 : i][0] : after;
        const int next = __shfl_sync(0xffffffffu, lane == 0 ? behind : o[i][0], (lane + 1) & 31);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            int bn, rn;
            row_counts<kPow2>(o[i][k], k < 3 ? o[i][k < 3 ? k + 1 : k] : next, p, bn, rn);
            packed[i][k] = !wide && row0 + kUnit * i + k >= M ? 0 : 2 * bn + rn;
        }
    }
    __device__ __forceinline__ void sums(const Params &p, int M, int lane, int &b, int &r) {  // of the warp
        b = r = 0;
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            count(p, M, lane, i);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                b += packed[i][k] >> 1;
                r += packed[i][k] & 1;
            }
        }
        b = __reduce_add_sync(0xffffffffu, b);
        r = __reduce_add_sync(0xffffffffu, r);
    }
};

// Counts of `group` tiles (1, or a multiple of kGroup) per CTA: sums[t] = segments and residue rows from the first row
// of the group to the end of tile t, so the last tile of a group holds the group's total.
constexpr int kGroup = 8;
template <bool kPow2>
__global__ void __launch_bounds__(kThreads, 4)
count_tiles(Params p, int M, int n_tiles, int group, const int *__restrict__ row_ptr, int2 *__restrict__ sums) {
    __shared__ int2 s_warp[kGroup][kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cta = static_cast<int>(after_chain(blockIdx.x));
    int carry_b = 0, carry_r = 0;
    for (int t0 = 0; t0 < group; t0 += kGroup) {
        const int tile0 = cta * group + t0;
        if (tile0 >= n_tiles) break;
#pragma unroll 4
        for (int t = 0; t < kGroup; ++t) {
            int b = 0, r = 0;
            if (tile0 + t < n_tiles && t < group) {
                WarpRows<kPow2> rows;
                rows.load(M, row_ptr, (tile0 + t) * kTile + warp * kWarpRows, lane);
                rows.sums(p, M, lane, b, r);
            }
            if (lane == 0) s_warp[t][warp] = make_int2(b, r);
        }
        __syncthreads();
        if (warp == 0) {
            int b = 0, r = 0;
            if (lane < kGroup) {
#pragma unroll
                for (int w = 0; w < kWarps; ++w) {
                    b += s_warp[lane][w].x;
                    r += s_warp[lane][w].y;
                }
            }
#pragma unroll
            for (int d = 1; d < kGroup; d <<= 1) {
                const int ub = __shfl_up_sync(0xffffffffu, b, d), ur = __shfl_up_sync(0xffffffffu, r, d);
                if (lane >= d) {
                    b += ub;
                    r += ur;
                }
            }
            b += carry_b;
            r += carry_r;
            if (lane < min(group, kGroup) && tile0 + lane < n_tiles) sums[tile0 + lane] = make_int2(b, r);
            carry_b = __shfl_sync(0xffffffffu, b, kGroup - 1);
            carry_r = __shfl_sync(0xffffffffu, r, kGroup - 1);
        }
        __syncthreads();
    }
    // the fill grid may start once every CTA of this grid has come this far (released at the start of the CTAs
    // instead, its CTAs take slots from this grid)
    chain_begin();
}

// The listed long rows, taken by the CTA's warps in turn.  The next row's list entry and bounds are
// fetched before the current row is written, so that chain of dependent loads is off the critical path.
template <bool kPow2>
__device__ __forceinline__ void write_long_rows(const Params &p, int lane, int warp, int total, const int *list_row,
                                                const int *list_dst, const int *__restrict__ row_ptr,
                                                int *__restrict__ out_row, int *__restrict__ out_off) {
    int s = warp;
    if (s >= total) return;
    int row = list_row[s], dst = list_dst[s];
    int off = __ldg(row_ptr + row), next = __ldg(row_ptr + row + 1);
    while (true) {
        const int s2 = s + kWarps;
        int row2 = 0, dst2 = 0, off2 = 0, next2 = 0;
        if (s2 < total) {
            row2 = list_row[s2];
            dst2 = list_dst[s2];
            off2 = __ldg(row_ptr + row2);
            next2 = __ldg(row_ptr + row2 + 1);
        }
        int cnt, unused;
        row_counts<kPow2>(off, next, p, cnt, unused);
        write_row<kPow2>(p, lane, 32, row, off, cnt, out_row + dst, out_off + dst);
        if (s2 >= total) return;
        s = s2;
        row = row2;
        dst = dst2;
        off = off2;
        next = next2;
    }
}

// The outputs of every tile.  Its place comes from the group totals before it, added up by the tile's own CTA, and
// the places inside it from one warp scan per 128 rows over the thread's (segments, residue rows), packed into
// one word.  A row's first segment is written by its thread, and so are a few further ones; rows of more than
// kShortRow segments are listed and written by the CTA's warps in turn (on graphs they cluster in the first tile).
//
// What bounds the decomposition: the latency of its phases, the instructions per row (19 + 60 warp instructions
// per 32 rows in the two kernels) and the tile with the longest rows; of the bytes 33 MB are read (the second time
// from the L2) and 38 MB written at 8.4 M rows (11 us at the copy bandwidth).  us per call, segments of 512 / 32,
// with a memset, a count kernel that scans in its last CTA and a fill kernel that orders through shared
// memory -> now: R-MAT scale 23 41.2 / 67.6 -> 34.9 / 59.7, R-MAT 21 16.9 / 39.7 -> 14.2 / 34.8, Pareto 2^22 rows
// 26.7 / 34.9 -> 22.6 / 32.7, 131,072 rows 10.1 / 10.6 -> 7.4 / 8.2, 1000 rows 8.3 / 9.6 -> 5.0 / 6.2.  Measured and dropped:
// one kernel with a look-back over the tiles' states (the CTAs that poll the same few lines hold up those that
// publish: 54 to 78 us), one row per lane with ballots (98 instructions per 32 rows), one segment per lane by a
// search in the warp's prefix (a chain of shuffles, 5 us per CTA), larger tiles (4096 rows 50, 8192 96 us).
//
// in_cluster: no count grid; this grid is one cluster of at most kClusterTiles CTAs and the totals travel
// through distributed shared memory.
constexpr int kClusterTiles = 8;
template <bool kPow2>
__global__ void __launch_bounds__(kThreads, 4)
fill_tiles(Params p, int M, int group, const int *__restrict__ row_ptr, const int2 *__restrict__ sums,
           int *__restrict__ block_r_ind, int *__restrict__ st_off, int *__restrict__ residue_r_ind,
           int *__restrict__ n_blk, int *__restrict__ n_res, bool write_sentinel, bool in_cluster) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ int2 s_warp[kWarps], s_before[kWarps];
    __shared__ int2 s_total;
    __shared__ int s_long_row[kTile], s_long_dst[kTile];
    __shared__ int n_long;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = static_cast<int>(after_chain_if(in_cluster, blockIdx.x));
    if (in_cluster) chain_begin();  // (large grids: the next call's waiting CTAs would take their slots, R-MAT 23 37.4 -> 38.2 us)
    if (threadIdx.x == 0) n_long = 0;
    const int warp_row0 = tile * kTile + warp * kWarpRows;
    WarpRows<kPow2> rows;
    rows.load(M, row_ptr, warp_row0, lane);
    const int row0 = rows.row0;
    const auto &o = rows.o;
    if (!in_cluster) {
        chain_wait();  // the count grid's sums
        int b = 0, r = 0;
        const int groups = tile / group;
#pragma unroll 4
        for (int g = threadIdx.x; g < groups; g += kThreads) {
            const int2 v = ld_behind_wait(sums + (static_cast<size_t>(g) + 1) * group - 1);
            b += v.x;
            r += v.y;
        }
        if (threadIdx.x == 0 && tile % group != 0) {
            const int2 v = ld_behind_wait(sums + tile - 1);
            b += v.x;
            r += v.y;
        }
        b = __reduce_add_sync(kFull, b);
        r = __reduce_add_sync(kFull, r);
        if (lane == 0) s_before[warp] = make_int2(b, r);
    }
    int bsum, rsum;
    rows.sums(p, M, lane, bsum, rsum);
    if (lane == 0) s_warp[warp] = make_int2(bsum, rsum);
    __syncthreads();
    // lane w < kWarps: warp w's sums; then the sums of the warps before this one
    int2 mine = make_int2(0, 0);
    if (lane < kWarps) mine = s_warp[lane];
    int base_b = __reduce_add_sync(kFull, lane < warp ? mine.x : 0), base_r = __reduce_add_sync(kFull, lane < warp ? mine.y : 0);
    const bool last = tile == static_cast<int>(gridDim.x) - 1;
    int place_b = 0, place_r = 0;
    if (in_cluster) {
        const auto cluster = cooperative_groups::this_cluster();
        const int total_b = __reduce_add_sync(kFull, mine.x), total_r = __reduce_add_sync(kFull, mine.y);
        if (threadIdx.x == 0) s_total = make_int2(total_b, total_r);
        cluster.sync();
        for (int t = 0; t < tile; ++t) {
            const int2 v = *cluster.map_shared_rank(&s_total, t);
            place_b += v.x;
            place_r += v.y;
        }
        cluster.sync();  // nobody leaves while its totals are being read
    } else {
        int2 before = make_int2(0, 0);
        if (lane < kWarps) before = s_before[lane];
        place_b = __reduce_add_sync(kFull, before.x);
        place_r = __reduce_add_sync(kFull, before.y);
    }
    if (last && warp == 0) {  // the last rows of the matrix
        const int n_b = place_b + __reduce_add_sync(kFull, mine.x), n_r = place_r + __reduce_add_sync(kFull, mine.y);
        if (lane == 0) {
            n_blk[0] = n_b;
            n_res[0] = n_r;
            if (write_sentinel) st_off[n_b] = __ldg(row_ptr + M);
        }
    }
    base_b += place_b;
    base_r += place_r;

    // ---- outputs --------------------------------------------------------------------------------------
    auto inclusive = [&](int x) {  // prefix sum over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int up = __shfl_up_sync(kFull, x, d);
            if (lane >= d) x += up;
        }
        return x;
    };
    constexpr int kResBits = 8;  // at most 128 residue rows per unit
    const bool packs = bsum < (1 << (31 - kResBits));
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
        int bn[4], rn[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            bn[k] = rows.packed[i][k] >> 1;
            rn[k] = rows.packed[i][k] & 1;
        }
        const int b4 = bn[0] + bn[1] + bn[2] + bn[3], r4 = rn[0] + rn[1] + rn[2] + rn[3];
        int b_incl, r_incl;
        if (packs) {
            const int x = inclusive((b4 << kResBits) | r4);
            b_incl = x >> kResBits;
            r_incl = x & ((1 << kResBits) - 1);
        } else {
            b_incl = inclusive(b4);
            r_incl = inclusive(r4);
        }
        const int row = row0 + kUnit * i;
        int at_r = base_r + r_incl - r4;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (rn[k]) residue_r_ind[at_r] = row + k;
            at_r += rn[k];
        }
        base_r += __shfl_sync(kFull, r_incl, 31);
        const int unit_b = __shfl_sync(kFull, b_incl, 31);
        if (unit_b == 0) continue;
        int at = base_b + b_incl - b4;
        base_b += unit_b;
        const bool several = __any_sync(kFull, (bn[0] > 1) | (bn[1] > 1) | (bn[2] > 1) | (bn[3] > 1));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (bn[k]) {
                block_r_ind[at] = row + k;
                st_off[at] = o[i][k];
            }
            if (several) {  // warp-uniform
                if (bn[k] > 1 && bn[k] <= kShortRow)
                    write_row<kPow2>(p, 1, 1, row + k, o[i][k], bn[k], block_r_ind + at, st_off + at);
                if (bn[k] > kShortRow) {
                    const int slot = atomicAdd(&n_long, 1);
                    s_long_row[slot] = row + k;
                    s_long_dst[slot] = at;
                }
            }
            at += bn[k];
        }
    }
    __syncthreads();
    write_long_rows<kPow2>(p, lane, warp, n_long, s_long_row, s_long_dst, row_ptr, block_r_ind, st_off);
}

int check_params(int seg_len, int k_block, int vec_len, int M, const void *row_ptr) {
    if (seg_len <= 0 || k_block <= 0 || vec_len <= 0)
        return fail(RODE_ERR_INVALID_ARGUMENT, "preprocess: seg_len, k_block, vec_len must be positive");
    if (seg_len % k_block != 0 || k_block % vec_len != 0)
        return fail(RODE_ERR_INVALID_ARGUMENT,
                    "preprocess: need seg_len %% k_block == 0 and k_block %% vec_len == 0 (got %d, %d, %d)",
                    seg_len, k_block, vec_len);
    if (M < 0 || M > INT_MAX - kTile)
        return fail(RODE_ERR_INVALID_ARGUMENT, "preprocess: M = %d outside [0, %d]", M, INT_MAX - kTile);
    if (row_ptr == nullptr) return fail(RODE_ERR_INVALID_ARGUMENT, "preprocess: row_ptr is null");
    return RODE_OK;
}

}  // namespace

int preprocess_tiles(int M) { return (M + kTile - 1) / kTile; }
constexpr int kMaxGroups = 2048;

// `sums` holds one entry per tile.  write_sentinel: also store st_off[n_blk] = row_ptr[M] (the C ABI's
// contract; the reference's device version does not, and its callers size st_off without room for it).
template <bool kPow2>
int launch_preprocess_kernels(const Params &p, int M, const int *row_ptr, int *block_r_ind, int *st_off,
                              int *residue_r_ind, int *n_blk, int *n_res, int2 *sums, cudaStream_t stream,
                              bool write_sentinel) {
    // What one portable cluster holds takes one launch; otherwise count, then fill as a programmatic dependent.
    const int n_tiles = preprocess_tiles(M);
    const bool in_cluster = n_tiles <= kClusterTiles;
    // tiles per count CTA: one while a fill CTA can add up all of them quickly (131,072 rows 10.2 us with eight),
    // then so many that it adds up at most kMaxGroups sums
    int group = n_tiles <= 1024 ? 1 : kGroup;
    while (n_tiles / group > kMaxGroups) group *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    if (in_cluster) {
        cfg.numAttrs = 2;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = n_tiles;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
    } else {
        RODE_CUDA_TRY(launch_chained(count_tiles<kPow2>, dim3((n_tiles + group - 1) / group), dim3(kThreads), stream, true, p, M,
                                     n_tiles, group, row_ptr, sums));
        RODE_CHECK_LAUNCH("rode::count_tiles");
    }
    const int2 *sums_in = sums;
    RODE_CUDA_TRY(cudaLaunchKernelEx(&cfg, fill_tiles<kPow2>, p, M, group, row_ptr, sums_in, block_r_ind, st_off,
                                     residue_r_ind, n_blk, n_res, write_sentinel, in_cluster));
    RODE_CHECK_LAUNCH("rode::fill_tiles");
    return RODE_OK;
}

int launch_preprocess(int seg_len, int k_block, int vec_len, int M, const int *row_ptr, int *block_r_ind,
                      int *st_off, int *residue_r_ind, int *n_blk, int *n_res, int2 *tile_scratch,
                      cudaStream_t stream, bool write_sentinel = true) {
    auto pow2 = [](int x) { return (x & (x - 1)) == 0; };
    const bool all_pow2 = pow2(seg_len) && pow2(k_block) && pow2(vec_len);
    Params p = {seg_len, k_block, vec_len, 0};
    while (all_pow2 && (1 << p.seg_shift) < seg_len) ++p.seg_shift;
    if (M == 0) {
        empty_matrix<<<1, 1, 0, stream>>>(row_ptr, st_off, n_blk, n_res, write_sentinel);
        RODE_CHECK_LAUNCH("rode::empty_matrix");
        return RODE_OK;
    }
    if (all_pow2)
        return launch_preprocess_kernels<true>(p, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk, n_res,
                                               tile_scratch, stream, write_sentinel);
    return launch_preprocess_kernels<false>(p, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk, n_res,
                                            tile_scratch, stream, write_sentinel);
}

// Body of the reference-signature entry point RoDe_preprocess (Preprocess_opt/_preprocess.cu:323-339):
// default stream, and nothing is written beyond the n_blk segments and n_res residue rows -- the
// reference's callers allocate nnz / seg_len + M entries for st_off (_preprocess.cu:426-430),
// which has no room for an end sentinel when every row is a whole number of segments.
int preprocess_reference_signature(int seg_len, int k_block, int vec_len, int M, const int *row_ptr,
                                   int *block_r_ind, int *st_off, int *residue_r_ind, int *n_blk, int *n_res,
                                   void *tile_scratch) {
    if (int rc = check_params(seg_len, k_block, vec_len, M, row_ptr)) return rc;
    if (!block_r_ind || !st_off || !residue_r_ind || !n_blk || !n_res)
        return fail(RODE_ERR_INVALID_ARGUMENT, "RoDe_preprocess: an output pointer is null");
    return launch_preprocess(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind, n_blk, n_res,
                             static_cast<int2 *>(tile_scratch), nullptr, /*write_sentinel=*/false);
}

// ---------------------------------------------------------------------------------------
// Scratch of rode_preprocess_noalloc: one int2 per tile for up to kNoAllocMaxRows rows,
// resident in every GPU that loads the library (64 KB) until the process exits.  In host
// code this name is only a handle; the device address comes from cudaGetSymbolAddress.
constexpr int kNoAllocMaxRows = 1 << 24;
constexpr int kNoAllocTiles = kNoAllocMaxRows / kTile;
static __device__ __align__(256) int2 g_noalloc_tile_scratch[kNoAllocTiles];

// Device address of the scratch array on the current device, looked up once per device.
int noalloc_scratch(int2 **out) {
    static int2 *address[64] = {nullptr};
    static std::mutex lock;
    int dev = 0;
    RODE_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(RODE_ERR_NO_DEVICE, "device index %d out of range", dev);
    std::lock_guard<std::mutex> guard(lock);
    if (address[dev] == nullptr) {
        void *p = nullptr;
        RODE_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_tile_scratch));
        address[dev] = static_cast<int2 *>(p);
    }
    *out = address[dev];
    return RODE_OK;
}

}  // namespace rode

extern "C" {

int rode_preprocess_workspace_bytes(int M, size_t *bytes) {
    if (bytes == nullptr || M < 0)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "preprocess_workspace_bytes: bad argument");
    const size_t tiles = static_cast<size_t>(rode::preprocess_tiles(M));
    *bytes = (tiles + 1) * sizeof(int2);  // one entry spare, so that no matrix needs an empty buffer
    return RODE_OK;
}

int rode_preprocess_capacity(int seg_len, int vec_len, int M, long long nnz, long long *max_blocks) {
    if (max_blocks == nullptr || seg_len <= 0 || vec_len <= 0 || M < 0 || nnz < 0)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "preprocess_capacity: bad argument");
    *max_blocks = (nnz + static_cast<long long>(vec_len - 1) * M) / seg_len + M;
    return RODE_OK;
}

int rode_preprocess(int seg_len, int k_block, int vec_len, int M, const int *row_ptr, int *block_r_ind,
                    int *st_off, int *residue_r_ind, int *n_blk, int *n_res, void *workspace,
                    size_t workspace_bytes, rode_stream_t stream) {
    if (int rc = rode::check_params(seg_len, k_block, vec_len, M, row_ptr)) return rc;
    if (!block_r_ind || !st_off || !residue_r_ind || !n_blk || !n_res)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "preprocess: an output pointer is null");
    size_t need = 0;
    rode_preprocess_workspace_bytes(M, &need);
    if (workspace == nullptr || workspace_bytes < need)
        return rode::fail(RODE_ERR_WORKSPACE, "preprocess: workspace of %zu bytes needed, %zu given", need,
                          workspace ? workspace_bytes : static_cast<size_t>(0));
    if (!rode::aligned_to(workspace, 8))
        return rode::fail(RODE_ERR_WORKSPACE, "preprocess: workspace must be 8-byte aligned");
    return rode::launch_preprocess(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind,
                                   n_blk, n_res, static_cast<int2 *>(workspace), stream);
}

int rode_preprocess_noalloc(int seg_len, int k_block, int vec_len, int M, const int *row_ptr, int *block_r_ind,
                            int *st_off, int *residue_r_ind, int *n_blk, int *n_res, rode_stream_t stream) {
    if (int rc = rode::check_params(seg_len, k_block, vec_len, M, row_ptr)) return rc;
    if (!block_r_ind || !st_off || !residue_r_ind || !n_blk || !n_res)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "preprocess_noalloc: an output pointer is null");
    if (M > rode::kNoAllocMaxRows)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT,
                          "preprocess_noalloc: M = %d exceeds the built-in scratch (at most %d rows); use "
                          "rode_preprocess with a caller-provided workspace",
                          M, rode::kNoAllocMaxRows);
    int2 *scratch = nullptr;
    if (int rc = rode::noalloc_scratch(&scratch)) return rc;
    return rode::launch_preprocess(seg_len, k_block, vec_len, M, row_ptr, block_r_ind, st_off, residue_r_ind,
                                   n_blk, n_res, scratch, stream);
}

int rode_preprocess_cpu(int seg_len, int k_block, int vec_len, int M, const int *row_ptr, int *block_r_ind,
                        int *st_off, int *residue_r_ind, int *n_blk, int *n_res) {
    if (int rc = rode::check_params(seg_len, k_block, vec_len, M, row_ptr)) return rc;
    if (!block_r_ind || !st_off || !residue_r_ind || !n_blk || !n_res)
        return rode::fail(RODE_ERR_INVALID_ARGUMENT, "preprocess_cpu: an output pointer is null");
    int nb = 0, nr = 0;
    for (int row = 0; row < M; ++row) {
        const int off = row_ptr[row];
        const int pad = off % vec_len;
        int left = row_ptr[row + 1] - off + pad;  // aligned length still to place
        int pos = off;                            // where the next segment starts
        while (left > seg_len) {
            block_r_ind[nb] = row;
            st_off[nb++] = pos;
            pos = (pos == off) ? off - pad + seg_len : pos + seg_len;
            left -= seg_len;
        }
        if (left >= k_block) {
            block_r_ind[nb] = row;
            st_off[nb++] = pos;
        }
        if (left % k_block != 0) residue_r_ind[nr++] = row;
    }
    st_off[nb] = row_ptr[M];
    *n_blk = nb;
    *n_res = nr;
    return RODE_OK;
}

}  // extern "C"
