// The emission fold of a multiply with one 4-byte word per value: all levels'
// emissions in one launch, gathered from shared memory.
//
// What bounds a fold of 4-byte values out of global memory is the L1: a warp
// instruction that gathers 32 words from 32 lines takes 32 tag cycles, about
// 300 G gathers/s on the whole GPU while the values fit L2, whatever the load
// path.  Shared memory serves the same random words at 2000 G/s.  So the value
// space (terminals, then arena slots) is cut into chunks that fill one block's
// shared memory, and the emissions are kept once more in (chunk, row, source)
// order, 4 bytes each: the source's place in the chunk and the row's in its
// block of 65,536 rows, 16 bits each (half the 8 bytes of the level order).
// Each block takes an equal share of that list, loads the few chunks it spans
// with coalesced reads and reduces every row's run in registers, a warp 128
// emissions at a time; each run within those 128 is one reduction into Y.
//
// With the gathers out of the way the instruction rate bounds it: a first form
// with one emission per lane and a shuffle scan over the 32 rows of every warp
// step issued 96 instructions per 32 emissions.  Here a lane folds four
// consecutive emissions by itself and only the run at its edges goes through
// shuffles, and the list is padded with zeroes so that a warp's 128 emissions
// never cross a (chunk, block of rows): no bounds are checked inside.
#pragma once

#include <cstdint>

#include "device_util.cuh"

namespace gmr {

constexpr int kWordChunk = 57344;   // words of values per chunk: 224 KB of a block's 227 KB, and 16-bit places
constexpr int kWordThreads = 1024;  // one block per SM
constexpr int kWordGroup = 128;     // emissions per warp step: four per lane
// Where the fold pays (one multiply as a graph, level by level -> in one launch).
// It takes the emissions off every level's launch and pays a launch and the loads
// of the chunks for it, so the levels have to be many: grammars of mosaics mostly
// have 14 to 23, of copy graphs 6 to 13.  Right product:
//   mosaics          levels  emissions  per chunk and row   (+,x) us      (OR,AND) us
//   1,500 x 800        19      0.10 M      67                -            36.9 ->  34.8
//   5,000 x 2,000      20      0.75 M      50                -            44.1 ->  45.0
//   9,000 x 3,000      21      1.9 M       30                -            53.3 ->  49.3
//   40,000 x 1,000     19      2.5 M        7.7          47.2 ->  47.8    52.6 ->  47.1
//   20,000 x 5,000     23      6.5 M       15            69.6 ->  65.2    74.1 ->  62.6
//   600,000 x 300      17      8.9 M        0.67         75.8 ->  72.7    79.9 ->  67.0
//   1,500,000 x 150    14     10.4 M        0.30         84.1 ->  87.2    87.8 ->  77.9
//   400,000 x 1,000     -     20.6 M        0.99        139.7 -> 113.9   144.4 -> 109.2
//   98,160 x 7,210      -     40.7 M        3.6         239.5 -> 151.8   240.2 -> 146.1
//   200,000 x 10,000    -    109 M          1.9           625 -> 322         -
//   copy graphs (nodes, degree, share copied)
//   20,000, 48, 0.7     7      0.54 M       9.0              -            20.5 ->  26.6
//   200,000, 16, 0.8    9      1.4 M        0.58             -            32.7 ->  36.9
//   100,000, 48, 0.5    6      3.7 M        3.7          30.6 ->  32.8    32.8 ->  32.8
//   300,000, 32, 0.8   11      4.2 M        0.47         51.0 ->  57.4    53.3 ->  55.1
//   500,000, 24, 0.6    7      8.1 M        0.48         63.2 ->  71.9    65.6 ->  67.5
//   200,000, 100, 0.7   9     11.4 M        1.09         82.8 ->  82.2    85.2 ->  77.8
//   300,000, 100, 0.7   9     17.1 M        0.74        113.1 -> 123.0   115.4 -> 117.6
// (min,+) is within 3 % of (OR,AND).  (+,x) lost below 2 M (a mosaic of 1.4 M: 40.8
// -> 43.4), and is within 1 % from there to 4 M.  Below 0.25 per chunk and row not
// measured.
constexpr int kWordMinDepth = 14;
constexpr double kWordMinPerRow = 0.25;
constexpr int64_t kWordMinEmissions = 1 << 16, kWordMinEmissionsPlus = 2 << 20;
// The left product, (+,x) only: two launches more, and every down value is read
// and written once more.  The same depth, and emissions per chunk of x and target
// (rules and terminals).  One product, edge lists alone -> rows' edges at once:
//   20,000 x 5,000     6.5 M  4.7  100 -> 115 us    50,000 x 5,000    15.3 M  5.6  164 -> 155
//   80,001 x 1,500     7.0 M  2.7  101 -> 117       100,000 x 4,000   22.9 M  2.9  207 -> 185
//   25,000 x 5,000     8.0 M  5.0  118 -> 123       98,160 x 7,210    40.7 M  3.1  295 -> 245
//   30,000 x 5,000     9.6 M  5.4  120 -> 117       200,000 x 10,000  109 M   1.6  664 -> 647
//   35,000 x 5,000    11.0 M  5.5  139 -> 126       1,500,000 x 150   10.4 M  0.3  111 -> 144
//   160,001 x 1,500   13.1 M  1.9  146 -> 141       graph 300,000 x 100  17 M  0.7  143 -> 197
// The idempotent semirings, whose atomics on down values are slower, lose on most:
// (OR,AND) 11.0 M 129 -> 123, 15.3 M 151 -> 173, 40.7 M 279 -> 290, 109 M 627 -> 703.
constexpr int64_t kLeftWordMinEmissions = 9 << 20;
constexpr double kLeftWordMinPerTarget = 1.5;
// Chunks per copy of Y: a row gets an addition per chunk that emits into it, more
// where its run there is longer than a warp step (n / 128 + 1 for n emissions),
// and the error of that chain grows with its length.  Long runs shorten it: the
// per-level fold they replace adds once per 32 to 128 emissions too, in every
// level.  Error against 64 bits, worst row over the largest value, per-level
// default before -> one launch: 41 rows x 400,000 (2.2 M emissions) 3.2e-6 ->
// 2.5e-6, 8 x 2,000,000 (2.6 M) 1.8e-6 -> 0.9e-6.
constexpr int kWordChunksPerCopy = 16, kWordMaxCopies = 16;

// Where the arena starts in the value space: a whole number of 256-byte lines.
inline int64_t word_t_span(int64_t n_terms) { return (n_terms + 63) / 64 * 64; }

// Place of the zero value: after the largest chunk.
inline int word_zero_at(int64_t n_terms, int64_t n_ops) {
    const int64_t total = word_t_span(n_terms) + n_ops;
    return (int)(total < kWordChunk ? total : kWordChunk);
}

struct WordFoldArgs {
    const uint4* entries;      // groups of 128; an entry: place in the chunk << 16 | row in its block of rows
    const uint32_t* seg;       // first group of (chunk, block of rows), then the group count
    int n_seg, n_blk;          // chunks x blocks of 65,536 rows; blocks
    int64_t n_groups;
    const void* T;             // n_terms words
    const void* arena;         // n_ops words
    int64_t n_terms, t_span, n_ops;  // t_span: n_terms rounded up, where the arena starts
    int zero_at;               // place of a zero value, after the largest chunk
    void* Y;                   // [copies][rows]: chunk c adds into copy c % copies
    int64_t rows;
    int copies;
    // Left product: the targets are the rules' and then, from block of rows
    // term_blk on, the terminals' down values.  nullptr: rows of Y throughout.
    void* Yterm;
    int term_blk;
};

// Chunk `chunk` of the value space into shared memory, 16 bytes per load (both
// arrays start on 256 bytes, chunks and t_span are multiples of 4 words).
template <class T>
__device__ __forceinline__ void load_word_chunk(const WordFoldArgs& a, int chunk, T* vals) {
    const int64_t v0 = (int64_t)chunk * kWordChunk, v1 = min(v0 + kWordChunk, a.t_span + a.n_ops);
    const int n = (int)(v1 - v0);
#pragma unroll 4
    for (int i = threadIdx.x * 4; i < n; i += kWordThreads * 4) {
        const int64_t v = v0 + i;
        const bool term = v < a.t_span;
        const T* p = term ? static_cast<const T*>(a.T) + v : static_cast<const T*>(a.arena) + (v - a.t_span);
        const int64_t left = term ? a.n_terms - v : a.n_ops - (v - a.t_span);  // words of that array from here
        if (left >= 4) {
            *reinterpret_cast<uint4*>(vals + i) = *reinterpret_cast<const uint4*>(p);
        } else {
            for (int j = 0; j < left; ++j) vals[i + j] = p[j];
        }
    }
}

// One warp step of a segmented fold: lane l holds items 4l .. 4l+3 of 128,
// items with equal keys are contiguous, and flush(key, sum) is called once per
// run.  A lane folds its own four; a run that crosses lanes is carried from
// the lane before (a scan over the lanes that are one run throughout, as many
// steps as the longest such stretch needs).
template <class S, int VEC, class Flush>
__device__ __forceinline__ void fold_runs(const int4 k, const Vec<typename S::T, VEC> (&v)[4], int lane, Flush&& flush) {
    using V = Vec<typename S::T, VEC>;
    constexpr unsigned kAll = 0xffffffffu;
    auto shfl_up = [](const V& x, int d) {
        V o;
#pragma unroll
        for (int j = 0; j < VEC; ++j) o.v[j] = __shfl_up_sync(kAll, x.v[j], d);
        return o;
    };
    const bool c1 = k.y == k.x, c2 = k.z == k.y, c3 = k.w == k.z;
    const V a1 = c1 ? voplus<S, VEC>(v[0], v[1]) : v[1], a2 = c2 ? voplus<S, VEC>(a1, v[2]) : v[2];
    V last = c3 ? voplus<S, VEC>(a2, v[3]) : v[3];  // the run this lane ends with
    const int32_t key_before = __shfl_up_sync(kAll, k.w, 1), key_after = __shfl_down_sync(kAll, k.x, 1);
    const bool joined = lane > 0 && key_before == k.x;  // the first run goes on from the lane before
    const bool open = lane == 31 || key_after != k.w;   // the last run ends here
    bool through = joined && c1 && c2 && c3;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        if (!__any_sync(kAll, through)) break;
        const V o = shfl_up(last, d);
        const bool t = __shfl_up_sync(kAll, (int)through, d);
        if (through) {
            last = voplus<S, VEC>(o, last);
            through = lane >= d && t;
        }
    }
    const V before = shfl_up(last, 1);
    const V in = joined ? before : vzero<S, VEC>();
    if (!c1) flush(k.x, voplus<S, VEC>(v[0], in));
    if (!c2) flush(k.y, c1 ? voplus<S, VEC>(a1, in) : a1);
    if (!c3) flush(k.z, c1 && c2 ? voplus<S, VEC>(a2, in) : a2);
    if (open) flush(k.w, last);
}

// The same with one item per lane: the sum of its run in the run's first lane.
template <class S, int VEC>
__device__ __forceinline__ Vec<typename S::T, VEC> fold_lanes(int32_t key, Vec<typename S::T, VEC> v, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    const int32_t before = __shfl_up_sync(kAll, key, 1);
    const unsigned heads = __ballot_sync(kAll, lane == 0 || before != key);
    const unsigned above = heads & (0xfffffffeu << lane);
    const int last = above ? __ffs(above) - 2 : 31;  // last lane of this lane's run
    unsigned m = ~heads;  // step d is needed while some run is longer than d: d lanes in a row that start none
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        if (m == 0) break;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const typename S::T o = __shfl_down_sync(kAll, v.v[j], d);
            if (lane + d <= last) v.v[j] = S::oplus(v.v[j], o);
        }
        m &= m >> d;
    }
    return v;
}

template <class S>
__device__ __forceinline__ void fold_word_group(const uint4 q, const typename S::T* vals, typename S::T* Y, int lane) {
    using T = typename S::T;
    const int4 row = make_int4(q.x & 0xffff, q.y & 0xffff, q.z & 0xffff, q.w & 0xffff);
    const Vec<T, 1> v[4] = {{vals[q.x >> 16]}, {vals[q.y >> 16]}, {vals[q.z >> 16]}, {vals[q.w >> 16]}};
    fold_runs<S, 1>(row, v, lane, [&](int32_t r, const Vec<T, 1>& sum) { S::red(Y + r, sum.v[0]); });
}

template <class S>
__global__ void __launch_bounds__(kWordThreads, 1) k_word_fold(WordFoldArgs a) {
    using T = typename S::T;
    extern __shared__ __align__(16) unsigned char word_smem[];
    T* vals = reinterpret_cast<T*>(word_smem);
    dependents_may_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t per = (a.n_groups + gridDim.x - 1) / gridDim.x;
    int64_t at = (int64_t)blockIdx.x * per;
    const int64_t end = min(at + per, a.n_groups);
    int s = 0;  // the last (chunk, block of rows) that starts at or before group `at`
    for (int lo = 0, hi = a.n_seg; lo < hi;) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)__ldg(a.seg + mid) <= at) {
            s = mid;
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    if (threadIdx.x == 0) vals[a.zero_at] = S::zero();
    wait_for_previous_kernel();
    int loaded = -1;
    for (; at < end && s < a.n_seg; ++s) {
        const int64_t to = min((int64_t)__ldg(a.seg + s + 1), end);
        if (to <= at) continue;
        const int chunk = s / a.n_blk;
        const int blk = s - chunk * a.n_blk;
        T* Y = a.Yterm && blk >= a.term_blk ? static_cast<T*>(a.Yterm) + ((int64_t)(blk - a.term_blk) << 16)
                                            : static_cast<T*>(a.Y) + (chunk % a.copies) * a.rows + ((int64_t)blk << 16);
        if (chunk != loaded) {
            __syncthreads();  // the chunk before is no longer read
            load_word_chunk<T>(a, chunk, vals);
            __syncthreads();
            loaded = chunk;
        }
        constexpr int kWarps = kWordThreads / 32;
        // the loads of the next two groups are in flight while two are folded (left
        // product, 50,000 x 5,000: 184 us without, 157 with; no difference where the
        // list streams from HBM at 200,000 x 10,000)
        const uint4* mine = a.entries + lane;
        int64_t g = at + warp;
        uint4 q0 = g < to ? __ldg(mine + g * 32) : make_uint4(0, 0, 0, 0);
        uint4 q1 = g + kWarps < to ? __ldg(mine + (g + kWarps) * 32) : q0;
        for (; g < to; g += 2 * kWarps) {
            const bool two = g + kWarps < to, three = g + 2 * kWarps < to, four = g + 3 * kWarps < to;
            const uint4 p0 = three ? __ldg(mine + (g + 2 * kWarps) * 32) : q0;
            const uint4 p1 = four ? __ldg(mine + (g + 3 * kWarps) * 32) : q0;
            fold_word_group<S>(q0, vals, Y, lane);
            if (two) fold_word_group<S>(q1, vals, Y, lane);
            q0 = p0;
            q1 = p1;
        }
        at = to;
    }
}

// Y from its copies, which the fold before writes (plain loads, no __restrict__).
template <class S>
__global__ void __launch_bounds__(256) k_word_sum(const typename S::T* parts, typename S::T* Y, int64_t rows, int copies) {
    dependents_may_launch();
    wait_for_previous_kernel();
    for (int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x; r < rows; r += (int64_t)gridDim.x * 256) {
        typename S::T v = parts[r];
        for (int c = 1; c < copies; ++c) v = S::oplus(v, parts[c * rows + r]);
        Y[r] = v;
    }
}

// Sort keys of the emissions: source in chunk << 48 | chunk << row_bits | row,
// to be sorted by the bits below 48.  left: rows are gathered (the value space
// is x) and the targets are rules, then terminals from left_terms on.
static __global__ void __launch_bounds__(256) k_word_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ row,
                                                          int64_t n, int64_t t_span, int row_bits, bool left,
                                                          int64_t left_terms, uint64_t* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int32_t c = src[i];
        const int64_t v = left ? (int64_t)row[i] : c >= 0 ? t_span + c : -(int64_t)c - 1;
        const int64_t to = !left ? (int64_t)row[i] : c >= 0 ? (int64_t)c : left_terms - (int64_t)c - 1;
        const int64_t chunk = v / kWordChunk;
        key[i] = (uint64_t)(v - chunk * kWordChunk) << 48 | (uint64_t)chunk << row_bits | (uint64_t)to;
    }
}

// first[s]: the first sorted emission whose (chunk, block of rows) is s or later.
static __global__ void __launch_bounds__(256) k_word_segments(const uint64_t* __restrict__ key, int64_t n, int row_bits,
                                                              int n_blk, int n_seg, uint32_t* __restrict__ first) {
    const uint64_t low = (1ull << 48) - 1;
    for (int s = blockIdx.x * 256 + threadIdx.x; s <= n_seg; s += gridDim.x * 256) {
        const uint64_t want = (uint64_t)(s / n_blk) << row_bits | (uint64_t)(s % n_blk) << 16;
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((key[mid] & low) < want) lo = mid + 1;
            else hi = mid;
        }
        first[s] = (uint32_t)lo;
    }
}

// The entries in whole groups per (chunk, block of rows): one warp per group;
// past the last emission of its segment an entry is the zero value in the
// segment's last row.
static __global__ void __launch_bounds__(256) k_word_entries(const uint64_t* __restrict__ key,
                                                             const uint32_t* __restrict__ first,
                                                             const uint32_t* __restrict__ seg, int n_seg, int64_t n_groups,
                                                             uint32_t zero_at, uint32_t* __restrict__ entries) {
    const int64_t warps = (int64_t)gridDim.x * 8;
    for (int64_t g = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); g < n_groups; g += warps) {
        int lo = 0, hi = n_seg;  // the last segment that starts at or before g (empty ones start with the next)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((int64_t)seg[mid] <= g) lo = mid;
            else hi = mid;
        }
        const uint32_t f0 = first[lo], f1 = first[lo + 1];
        for (int j = threadIdx.x & 31; j < kWordGroup; j += 32) {
            const int64_t i = (int64_t)f0 + (g - seg[lo]) * kWordGroup + j;
            const uint64_t k = key[i < f1 ? i : (int64_t)f1 - 1];
            entries[g * kWordGroup + j] = (i < f1 ? (uint32_t)(k >> 48) : zero_at) << 16 | (uint32_t)(k & 0xffffu);
        }
    }
}

}  // namespace gmr
