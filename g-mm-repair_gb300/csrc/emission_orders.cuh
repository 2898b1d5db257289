// The engine's other orders of a plan's emissions, built on the GPU from the
// uploaded (level, row, source) order with stable radix sorts: by source slot
// (push lists) and by source chunk within a level.  On the host these two were
// most of creating an engine (109 M emissions: 880 and 683 ms of 1.75 s; 6.6 M:
// 32 of 45 ms, push lists alone), as single-threaded passes with a random
// access per emission.
#pragma once

#include <cstdint>

#include "device_util.cuh"
#include "sort.cuh"

namespace gmr {
namespace orders {

// Level of emission e: em_off[level] <= e < em_off[level + 1].
__device__ __forceinline__ int level_of(const int64_t* __restrict__ em_off, int n_levels, int64_t e) {
    int lo = 0, hi = n_levels;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (em_off[mid] <= e) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Levels (1..depth) with an emission whose source is no slot of that level.
static __global__ void __launch_bounds__(256) k_mixed_levels(const int32_t* __restrict__ src, int64_t e0, int64_t e1,
                                                             const int64_t* __restrict__ em_off,
                                                             const int64_t* __restrict__ lvl_off, int n_levels,
                                                             uint8_t* __restrict__ mixed) {
    for (int64_t e = e0 + (int64_t)blockIdx.x * 256 + threadIdx.x; e < e1; e += (int64_t)gridDim.x * 256) {
        const int k = level_of(em_off, n_levels, e);
        const int64_t s = src[e];
        if (s < lvl_off[k - 1] || s >= lvl_off[k]) mixed[k] = 1;
    }
}

// Push order: key = source slot (n_ops: a level that cannot push), value = row.
static __global__ void __launch_bounds__(256) k_push_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ row,
                                                          int64_t e0, int64_t n, const int64_t* __restrict__ em_off,
                                                          int n_levels, const uint8_t* __restrict__ mixed, int64_t n_ops,
                                                          uint64_t* __restrict__ key, uint32_t* __restrict__ val) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        key[i] = mixed[level_of(em_off, n_levels, e0 + i)] ? (uint64_t)n_ops : (uint64_t)src[e0 + i];
        val[i] = (uint32_t)row[e0 + i];
    }
}

// Chunk order: key = row << 32 | chunk, chunks numbered level by level
// (chunk_base), value = source reference.
static __global__ void __launch_bounds__(256) k_chunk_keys(const int32_t* __restrict__ src, const int32_t* __restrict__ row,
                                                           int64_t n, const int64_t* __restrict__ em_off,
                                                           const int64_t* __restrict__ lvl_off,
                                                           const int64_t* __restrict__ chunk_base, int n_levels,
                                                           int64_t chunk_slots, uint64_t* __restrict__ key,
                                                           uint32_t* __restrict__ val) {
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256) {
        const int k = level_of(em_off, n_levels, e);
        const int32_t c = src[e];
        const int64_t at = c >= 0 ? (int64_t)c - (k ? lvl_off[k - 1] : 0) : -(int64_t)c - 1;
        key[e] = (uint64_t)(uint32_t)row[e] << 32 | (uint64_t)(chunk_base[k] + at / chunk_slots);
        val[e] = (uint32_t)c;
    }
}

// first[g] for g = 0..groups: the first j whose key's low 32 bits are g or more.
// A search per group: its time does not depend on how the keys lie (one thread
// per key that fills the groups since the key before it walks whole levels that
// emit nothing alone).
template <class T>
__global__ void __launch_bounds__(256) k_group_firsts(const uint64_t* __restrict__ key, int64_t n, int64_t groups,
                                                      T* __restrict__ first) {
    for (int64_t g = (int64_t)blockIdx.x * 256 + threadIdx.x; g <= groups; g += (int64_t)gridDim.x * 256) {
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((int64_t)(uint32_t)key[mid] < g) lo = mid + 1;
            else hi = mid;
        }
        first[g] = (T)lo;
    }
}

static __global__ void __launch_bounds__(256) k_chunk_unpack(const uint64_t* __restrict__ key, int64_t n,
                                                             int32_t* __restrict__ row, uint32_t* __restrict__ head) {
    for (int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x; j < n; j += (int64_t)gridDim.x * 256) {
        row[j] = (int32_t)(key[j] >> 32);
        head[j] = j == 0 || key[j] != key[j - 1];
    }
}

static __global__ void __launch_bounds__(256) k_chunk_segments(const uint64_t* __restrict__ key,
                                                               const uint32_t* __restrict__ head,
                                                               const uint32_t* __restrict__ index, int64_t n,
                                                               int32_t* __restrict__ seg_row, int64_t* __restrict__ seg_start) {
    for (int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x; j <= n; j += (int64_t)gridDim.x * 256) {
        if (j == n) {
            seg_start[index[n]] = n;
        } else if (head[j]) {
            seg_row[index[j]] = (int32_t)(key[j] >> 32);
            seg_start[index[j]] = j;
        }
    }
}

// out[i] = a[at[i]] (at and out may be the same array).
static __global__ void __launch_bounds__(256) k_pick(const uint32_t* __restrict__ a, const int64_t* at, int64_t n,
                                                     int64_t* out) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) out[i] = a[at[i]];
}

}  // namespace orders
}  // namespace gmr
