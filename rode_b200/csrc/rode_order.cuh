// Block segments in the order of the columns that they gather from.
//
// A row's columns ascend, so a piece of a long row gathers from a narrow band of the dense operand.  Row by row, the warps on
// the GPU work on bands all over it at the same time, and an operand larger than the L2 comes from DRAM once per gather.
// With the pieces sorted by their first column into 256 buckets, the warps move through the operand together: a band is
// read once, and the other pieces that need it find it in the L2.  Nothing but the order of the work depends on the columns,
// so rows in any order of columns give the same results.  (An LRU model of a 100 MB cache: Pareto 2^20 K = 128, gathers that miss,
// row by row 82 %, pieces of 32 31 %, of 16 18 %; R-MAT scale 23 K = 64 35 %, of 128 22 %, of 32 13 %.)
//
// The order costs two passes over the segments' descriptors and one column per piece: 24 to 30 us for 300,000 pieces, 70 to 76 for
// 0.7 to 1.4 million, 77 to 205 for 1 to 7 million (R-MAT 23), bound by the chain descriptor -> row pointer -> column -> count.
#pragma once

#include <climits>

#include "rode_common.cuh"

namespace rode {

// Below so many segments an order does not pay for itself, below so many columns the dense operand fits the L2 at any width in
// use (1 KB per row: 160 MB).
constexpr int kOrderMinSegments = 1 << 13;
constexpr int kOrderLongRows = 330;  // SDDMM: nonzeros of the matrix per segment, most are in rows of many (512-long) segments
constexpr int kOrderMinColumns = 160 << 10;
constexpr int kOrderBuckets = 256;   // one per thread of an ordering CTA
constexpr int kOrderThreads = kOrderBuckets;
constexpr int kOrderPerThread = 8;   // pieces a thread holds per round (1 where a segment is one)
// Head of the ordering's part of a workspace, zeroed before the call's first kernel; the list follows it.
struct OrderHead {
    int counts[kOrderBuckets];  // pieces per bucket
    int used[kOrderBuckets];    // of them already placed in the list
    int claim;                  // claim counter of the kernel that works through the list
    int unused[63];             // (the list starts on a 256-byte boundary of the head)
};

// A piece: some consecutive nonzeros of one row, packed into 64 bits.
constexpr int kPieceOffBits = 31, kPieceLenBits = 7;  // P = 64: up to 126 nonzeros
constexpr int kPieceMaxRows = 1 << (64 - kPieceOffBits - kPieceLenBits);
__host__ __device__ constexpr unsigned long long pack_piece(int row, int off, int len) {
    return static_cast<unsigned long long>(row) << (kPieceOffBits + kPieceLenBits) |
           static_cast<unsigned long long>(len) << kPieceOffBits | static_cast<unsigned>(off);
}
struct Piece {
    int row, off, len;
};
__host__ __device__ inline Piece unpack_piece(unsigned long long p) {
    return {static_cast<int>(p >> (kPieceOffBits + kPieceLenBits)), static_cast<int>(p & 0x7fffffffu),
            static_cast<int>((p >> kPieceOffBits) & ((1 << kPieceLenBits) - 1))};
}

// Segment [off, end) cut at multiples of P, without pieces shorter than P / 2 at its ends: P / 2 <= length <= 2 P - 2
// (or the whole segment, where that is shorter).
template <int P>
struct Cuts {
    int off, end, first, last;  // first and last inner cut; last < first: one piece
    __host__ __device__ Cuts(int off_, int end_) : off(off_), end(end_) {
        first = (off / P + 1) * P;
        if (first - off < P / 2) first += P;
        last = end / P * P;
        if (end - last < P / 2) last -= P;
    }
    __host__ __device__ int count() const { return end <= off ? 0 : last < first ? 1 : (last - first) / P + 2; }
    __host__ __device__ int begin(int j) const { return j == 0 ? off : first + (j - 1) * P; }
    __host__ __device__ int stop(int j) const { return j == count() - 1 ? end : first + j * P; }
};
// At most so many pieces in m1 segments that hold nnz nonzeros together.
inline long long max_pieces(long long m1, long long nnz, int P) { return nnz / P + m1; }

// P = 0: whole segments.  number: of the segment; last bit of `bits`: it is all of its row.
struct __align__(16) WholeSegment {
    int row, off, end, bits;
    __host__ __device__ int number() const { return bits >> 1; }
    __host__ __device__ bool whole_row() const { return (bits & 1) != 0; }
};
constexpr int kWholeMaxSegments = 1 << 30;
template <int P>
struct Entry {
    using type = unsigned long long;
};
template <>
struct Entry<0> {
    using type = WholeSegment;
};

// Bytes of an ordering workspace.
template <int P>
size_t ordering_bytes(long long m1, long long nnz) {
    return sizeof(OrderHead) + static_cast<size_t>(P > 0 ? max_pieces(m1, nnz, P > 0 ? P : 1) : m1) * sizeof(typename Entry<P>::type);
}

#ifdef __CUDACC__
// What keeps an order by columns from helping, judged from 4096 samples of the nonzeros.  kOrderLocal: rows are narrow bands already
// (1024 rows span less than a thirtieth of the columns on average).  kOrderSkewed: a few columns get most of the references, and
// their rows stay in the L2 in any order (R-MAT 21 K = 64 block 457 us row by row, 486 ordered); the samples then repeat
// columns far more often than the S^2 / 2n times of uniform ones, on R-MAT graphs of scale 18 to 21 50 to 150 times as often,
// whatever the numbering of the columns.
//
// How much of the columns a segment spans (a row's span over the number of its segments, 1024 samples) is what whole segments in
// order depend on, and goes with it: kOrderNarrow: less than three quarters on average; kOrderWide: more than nine tenths.
enum { kOrderHelps = 0, kOrderSkewed = 1, kOrderLocal = 2, kOrderKind = 3, kOrderNarrow = 4, kOrderWide = 8 };

// One CTA takes 256 consecutive segments, their pieces in rounds of 2048.  kPlace = false counts the pieces of each bucket,
// kPlace = true puts them into the list, bucket after bucket; inside a bucket they stand in any order.  capacity: entries that the
// list has room for; max_pieces() of the true nnz and m1 is always enough.
template <int P, bool kPlace>
__global__ void __launch_bounds__(kOrderThreads)
order_pieces(int m1, int n_cols, const int *__restrict__ row_offsets, const int *__restrict__ column_indices,
             const int *__restrict__ block_r_ind, const int *__restrict__ st_off, OrderHead *head,
             typename Entry<P>::type *__restrict__ list, int capacity) {
    using E = typename Entry<P>::type;
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ int s_row[kOrderThreads], s_off[kOrderThreads], s_end[kOrderThreads], s_stop[kOrderThreads];
    __shared__ int s_whole[P == 0 ? kOrderThreads : 1];
    __shared__ int s_warp[kOrderThreads / 32], s_hist[kOrderBuckets], s_base[kOrderBuckets];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    chain_begin();
    const int seg = blockIdx.x * kOrderThreads + t;
    int row = 0, off = 0, end = 0, n = 0;
    if (seg < m1) {
        row = __ldg(block_r_ind + seg);
        off = __ldg(st_off + seg);
        const int next = seg + 1 < m1 ? __ldg(st_off + seg + 1) : INT_MAX;
        const int row_end = __ldg(row_offsets + row + 1);
        end = min(row_end, next);
        if constexpr (P == 0) s_whole[t] = off == __ldg(row_offsets + row) && next >= row_end ? 1 : 0;
        if constexpr (P > 0)
            n = Cuts<P>(off, end).count();
        else
            n = 1;
    }
    // exclusive prefix sum over the CTA
    auto scan = [&](int x, int &total) {
        int incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int up = __shfl_up_sync(kFull, incl, d);
            if (lane >= d) incl += up;
        }
        __syncthreads();
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = 0;
        total = 0;
#pragma unroll
        for (int w = 0; w < kOrderThreads / 32; ++w) {
            if (w < warp) before += s_warp[w];
            total += s_warp[w];
        }
        return before + incl - x;
    };
    int total, unused;
    const int start = scan(n, total);
    s_row[t] = row;
    s_off[t] = off;
    s_end[t] = end;
    s_stop[t] = start + n;  // pieces up to and with this segment
    s_hist[t] = 0;
    int my_start = 0;       // where bucket t starts in the list
    if constexpr (kPlace) {
        chain_wait();  // the counts
        my_start = scan(ld_behind_wait(&head->counts[t]), unused);
    }
    __syncthreads();
    constexpr int N = P > 0 ? kOrderPerThread : 1;
    for (int base = 0; base < total; base += kOrderThreads * N) {
        E piece[N];
        int key[N], rank[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int q = base + i * kOrderThreads + t;
            key[i] = -1;
            if (q < total) {
                int lo = 0;  // segments that end at or before q
#pragma unroll
                for (int step = kOrderThreads / 2; step >= 1; step >>= 1)
                    if (s_stop[lo + step - 1] <= q) lo += step;
                int b;
                if constexpr (P > 0) {
                    const Cuts<P> cuts(s_off[lo], s_end[lo]);
                    const int j = q - (lo > 0 ? s_stop[lo - 1] : 0);
                    b = cuts.begin(j);
                    piece[i] = pack_piece(s_row[lo], b, cuts.stop(j) - b);
                } else {
                    b = s_off[lo];
                    piece[i] = {s_row[lo], b, s_end[lo], (static_cast<int>(blockIdx.x) * kOrderThreads + lo) << 1 | s_whole[lo]};
                }
                const unsigned c = static_cast<unsigned>(__ldg(column_indices + b));
                key[i] = static_cast<int>(min(static_cast<unsigned long long>(c) * kOrderBuckets / static_cast<unsigned>(n_cols),
                                              kOrderBuckets - 1ull));
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (key[i] >= 0) rank[i] = atomicAdd(&s_hist[key[i]], 1);
        if constexpr (kPlace) {
            __syncthreads();
            const int mine = s_hist[t];
            if (mine > 0) s_base[t] = my_start + atomicAdd(&head->used[t], mine);
            s_hist[t] = 0;
            __syncthreads();
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (key[i] >= 0 && s_base[key[i]] + rank[i] < capacity) list[s_base[key[i]] + rank[i]] = piece[i];
            __syncthreads();
        }
    }
    if constexpr (!kPlace) {
        __syncthreads();
        if (s_hist[t] > 0) atomicAdd(&head->counts[t], s_hist[t]);
    }
}
// What a call with an ordering workspace has: the head, the list behind it, and the number of columns.
struct Ordering {
    OrderHead *head;
    int capacity, n_cols;
    template <int P>
    typename Entry<P>::type *list() const {
        return reinterpret_cast<typename Entry<P>::type *>(head + 1);
    }
};
// The order of the segments' pieces, on s.  The kernel that works through the list is launched chained behind it.
template <int P>
int launch_order(const Ordering &ord, int m1, const int *row_offsets, const int *col, const int *block_r_ind, const int *st_off,
                 cudaStream_t s) {
    const dim3 grid((m1 + kOrderThreads - 1) / kOrderThreads), block(kOrderThreads);
    RODE_CUDA_TRY(cudaMemsetAsync(ord.head, 0, sizeof(OrderHead), s));
    order_pieces<P, false><<<grid, block, 0, s>>>(m1, ord.n_cols, row_offsets, col, block_r_ind, st_off, ord.head, ord.list<P>(),
                                                  ord.capacity);
    RODE_CUDA_TRY(launch_chained(order_pieces<P, true>, grid, block, s, true, m1, ord.n_cols, row_offsets, col, block_r_ind,
                                 st_off, ord.head, ord.list<P>(), ord.capacity));
    RODE_CHECK_LAUNCH("rode::order_pieces");
    return RODE_OK;
}
#endif  // __CUDACC__

}  // namespace rode
