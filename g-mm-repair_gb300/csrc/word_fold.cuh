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
// with coalesced reads, reduces every row's run in registers and issues one
// reduction per (chunk, row) into Y.  Rows ascend along a warp, so those
// reductions touch few sectors.  It pays when runs are long enough, that is
// when a chunk holds about one emission per row or more (kWordMinPerRow).
#pragma once

#include <cstdint>

#include "device_util.cuh"

namespace gmr {

constexpr int kWordChunk = 57344;       // words of values per chunk: 224 KB of a block's 227 KB
constexpr int kWordThreads = 1024;      // one block per SM
constexpr int kWordBatch = 8;           // emissions in flight per lane
constexpr int64_t kWordTermAlign = 64;  // the arena starts at a multiple of this in the value space

struct WordFoldArgs {
    const uint32_t* entries;   // (source in chunk) << 16 | row in block of rows
    const uint32_t* seg;       // first entry of (chunk, block of rows), then the entry count
    int n_seg, n_blk;          // chunks x blocks of 65,536 rows; blocks
    int64_t n_entries;
    const void* T;             // n_terms words
    const void* arena;         // n_ops words
    int64_t n_terms, t_span, n_ops;  // t_span: n_terms rounded up, where the arena starts
    void* Y;
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

template <class S>
__global__ void __launch_bounds__(kWordThreads, 1) k_word_fold(WordFoldArgs a) {
    using T = typename S::T;
    extern __shared__ __align__(16) unsigned char word_smem[];
    T* vals = reinterpret_cast<T*>(word_smem);
    dependents_may_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t per = ((a.n_entries + gridDim.x - 1) / gridDim.x + 31) & ~(int64_t)31;
    int64_t at = (int64_t)blockIdx.x * per;
    const int64_t end = min(at + per, a.n_entries);
    int s = 0;  // the segment that holds entry `at`: the last one that starts at or before it
    for (int lo = 0, hi = a.n_seg; lo < hi;) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(a.seg + mid) <= (uint64_t)at) {
            s = mid;
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    wait_for_previous_kernel();
    int loaded = -1;
    for (; at < end; ++s) {
        const int64_t to = min((int64_t)__ldg(a.seg + s + 1), end);
        if (to <= at) continue;
        const int chunk = s / a.n_blk;
        T* Y = static_cast<T*>(a.Y) + ((int64_t)(s - chunk * a.n_blk) << 16);
        if (chunk != loaded) {
            __syncthreads();  // the chunk before is no longer read
            load_word_chunk<T>(a, chunk, vals);
            __syncthreads();
            loaded = chunk;
        }
        for (int64_t b = at + warp * (32 * kWordBatch); b < to; b += kWordThreads * kWordBatch) {
            uint32_t e[kWordBatch];
#pragma unroll
            for (int u = 0; u < kWordBatch; ++u) {
                const int64_t i = b + u * 32 + lane;
                e[u] = i < to ? __ldg(a.entries + i) : 0xffffffffu;  // no source is 0xffff
            }
#pragma unroll
            for (int u = 0; u < kWordBatch; ++u) {
                const bool valid = e[u] != 0xffffffffu;
                T v = valid ? vals[e[u] >> 16] : S::zero();
                const uint32_t row = e[u] & 0xffffu;
                const uint32_t key = valid ? row : 0x10000u;
                const uint32_t before = __shfl_up_sync(0xffffffffu, key, 1);
                const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != key);
                const unsigned above = heads & (0xfffffffeu << lane);
                const int last = above ? __ffs(above) - 2 : 31;  // last lane of this lane's run
                // step d is needed while some run is longer than d (d lanes in a row that are no head)
                unsigned m = ~heads;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    if (m == 0) break;
                    const T o = __shfl_down_sync(0xffffffffu, v, d);
                    if (lane + d <= last) v = S::oplus(v, o);
                    m &= m >> d;
                }
                if (valid && (heads >> lane & 1u)) S::red(Y + row, v);
            }
        }
    }
}

// Sort keys of the emissions: source in chunk << 48 | chunk << row_bits | row,
// to be sorted by the bits below 48.
static __global__ void __launch_bounds__(256) k_word_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ row,
                                                          int64_t n, int64_t t_span, int row_bits,
                                                          uint64_t* __restrict__ key) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int32_t c = src[i];
        const int64_t v = c >= 0 ? t_span + c : -(int64_t)c - 1;
        const int64_t chunk = v / kWordChunk;
        key[i] = (uint64_t)(v - chunk * kWordChunk) << 48 | (uint64_t)chunk << row_bits | (uint32_t)row[i];
    }
}

static __global__ void __launch_bounds__(256) k_word_entries(const uint64_t* __restrict__ key, int64_t n,
                                                             uint32_t* __restrict__ entries) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
        entries[i] = (uint32_t)(key[i] >> 48) << 16 | (uint32_t)(key[i] & 0xffffu);
}

// seg[s]: the first entry whose (chunk, block of rows) is s or later.
static __global__ void __launch_bounds__(256) k_word_segments(const uint64_t* __restrict__ key, int64_t n, int row_bits,
                                                              int n_blk, int n_seg, uint32_t* __restrict__ seg) {
    const uint64_t low = (1ull << 48) - 1;
    for (int s = blockIdx.x * 256 + threadIdx.x; s <= n_seg; s += gridDim.x * 256) {
        const uint64_t want = (uint64_t)(s / n_blk) << row_bits | (uint64_t)(s % n_blk) << 16;
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((key[mid] & low) < want) lo = mid + 1;
            else hi = mid;
        }
        seg[s] = (uint32_t)lo;
    }
}

}  // namespace gmr
