// The two ends of a sampling call, on the device: the reference's sorted
// uniforms (src/engines/dense/sample.cpp:36-42 over common::Rng,
// src/common/rng.cpp:176-186) before the walk, and the walk's basis states as
// (outcome, count) pairs after it.
//
// On the host these were what bounded a call: for 1e6 shots the generator, a
// bucket sort on eight threads, two 8 MB pageable copies and a pass over
// pairs took 20 ms around 3 ms of kernels.  Here the words come from one CTA
// (uniforms.cuh), are spread over buckets by their top bits and sorted there
// in shared memory, and only the distinct outcomes cross to the host.
#include <cuda_runtime.h>

#include <cstdint>

#include "mb2_internal.h"
#include "uniforms.cuh"

namespace mb2 {
namespace {

constexpr uint32_t kSortThreads = 256;
constexpr uint32_t kSortMean = 512;  // shots per bucket at most, on average
constexpr uint32_t kSortCap = 1024;  // keys a CTA sorts in shared memory
constexpr uint32_t kRleThreads = 256;
constexpr uint32_t kRleItems = 4;
constexpr uint32_t kRleTile = kRleThreads * kRleItems;

// Buckets by a key's top bits: uniform keys, so the sizes are within a few
// standard deviations (23) of their mean, at most half of what the shared
// memory holds; a fuller bucket is sorted where it lies.  Small buckets cost
// little to sort and spread the counters' atomics (1e6 shots: 2048 a bucket
// 138 us to count and 84 to sort, 512 a bucket 43 and 67).
uint32_t bucket_bits(uint64_t shots) {
    uint32_t b = 0;
    while (b < 24 && (shots >> b) > kSortMean) ++b;
    return b;
}

__global__ void __launch_bounds__(kWordThreads) k_words(const __grid_constant__ MtSeed seed, uint64_t shots,
                                                        uint64_t* __restrict__ words) {
    mt_words(seed, shots, words);
}

// Each key's place within its bucket (any order: equal keys are alike and
// the bucket is sorted afterwards).
__global__ void k_bucket_count(const uint64_t* __restrict__ words, uint64_t shots, uint32_t shift,
                               uint32_t* __restrict__ count, uint32_t* __restrict__ place) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < shots;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        place[i] = atomicAdd(count + (mt_key(words[i]) >> shift), 1u);
}

// Exclusive scan of `count` counters by one CTA of 1024 threads; total at [count].
template <typename T>
__device__ __forceinline__ void scan_cta(const uint32_t* __restrict__ in, uint64_t count, T* __restrict__ out) {
    __shared__ T warp_sum[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    T carry = 0;
    for (uint64_t b = 0; b < count; b += 1024) {
        const uint64_t i = b + threadIdx.x;
        const T v = i < count ? in[i] : 0u;
        T s = v;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const T p = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += p;
        }
        if (lane == 31) warp_sum[warp] = s;
        __syncthreads();
        T before = 0, total = 0;
        for (uint32_t w = 0; w < 32; ++w) {
            const T x = warp_sum[w];
            before += w < warp ? x : 0;
            total += x;
        }
        if (i < count) out[i] = carry + before + s - v;
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[count] = carry;
}

__global__ void __launch_bounds__(1024) k_scan(const uint32_t* __restrict__ in, uint64_t count,
                                               uint64_t* __restrict__ out) {
    scan_cta<unsigned long long>(in, count, reinterpret_cast<unsigned long long*>(out));
}

__global__ void k_bucket_scatter(const uint64_t* __restrict__ words, uint64_t shots, uint32_t shift,
                                 const uint64_t* __restrict__ start, const uint32_t* __restrict__ place,
                                 uint64_t* __restrict__ out) {
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < shots;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t k = mt_key(words[i]);
        out[start[k >> shift] + place[i]] = k;
    }
}

// Sorts v[0..n) ascending: the bitonic network whose comparators all point
// the same way (the first step of each merge compares mirrored positions),
// so places past n stand for keys above every other and are skipped.
__device__ __forceinline__ void sort_cta(uint64_t* v, uint64_t n) {
    uint64_t pow2 = 1;
    while (pow2 < n) pow2 <<= 1;
    for (uint64_t size = 2; size <= pow2; size <<= 1) {
        for (uint64_t gap = size >> 1; gap > 0; gap >>= 1) {
            for (uint64_t t = threadIdx.x; t < (pow2 >> 1); t += kSortThreads) {
                const uint64_t low = t & (gap - 1), a = ((t ^ low) << 1) | low;
                const uint64_t b = gap == (size >> 1) ? a ^ (size - 1) : a | gap;
                if (b < n) {
                    const uint64_t x = v[a], y = v[b];
                    if (x > y) {
                        v[a] = y;
                        v[b] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// One CTA per bucket: its keys sorted, as uniforms k * 2^-53 (exact) at the
// bucket's place in u.
__global__ void __launch_bounds__(kSortThreads) k_bucket_sort(uint64_t* __restrict__ keys,
                                                              const uint64_t* __restrict__ start,
                                                              double* __restrict__ u) {
    __shared__ uint64_t sh[kSortCap];
    const uint64_t begin = start[blockIdx.x], n = start[blockIdx.x + 1] - begin;
    uint64_t* v = keys + begin;
    if (n <= kSortCap) {
        for (uint64_t i = threadIdx.x; i < n; i += kSortThreads) sh[i] = v[i];
        v = sh;
    }
    __syncthreads();
    sort_cta(v, n);
    for (uint64_t i = threadIdx.x; i < n; i += kSortThreads)
        u[begin + i] = static_cast<double>(v[i]) * (1.0 / 9007199254740992.0);
}

// Runs of equal basis states (non-decreasing): the runs that begin in each
// tile of kRleTile shots, then each run's state and first shot at its rank.
__global__ void __launch_bounds__(kRleThreads) k_run_count(const uint64_t* __restrict__ basis, uint64_t shots,
                                                           uint32_t* __restrict__ heads) {
    const uint64_t b = static_cast<uint64_t>(blockIdx.x) * kRleTile;
    uint32_t n = 0;
#pragma unroll
    for (uint32_t k = 0; k < kRleItems; ++k) {
        const uint64_t i = b + k * kRleThreads + threadIdx.x;
        n += __syncthreads_count(i < shots && (i == 0 || basis[i] != basis[i - 1]));
    }
    if (threadIdx.x == 0) heads[blockIdx.x] = n;
}

__global__ void __launch_bounds__(kRleThreads)
    k_run_heads(const uint64_t* __restrict__ basis, uint64_t shots, const uint64_t* __restrict__ before,
                uint64_t* __restrict__ outcomes, uint64_t* __restrict__ first) {
    __shared__ uint32_t warp_heads[kRleThreads / 32];
    const uint64_t b = static_cast<uint64_t>(blockIdx.x) * kRleTile;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t rank = before[blockIdx.x];
    for (uint32_t k = 0; k < kRleItems; ++k) {
        const uint64_t i = b + k * kRleThreads + threadIdx.x;
        const uint64_t v = i < shots ? basis[i] : 0;
        const bool head = i < shots && (i == 0 || v != basis[i - 1]);
        const uint32_t votes = __ballot_sync(0xffffffffu, head);
        if (lane == 0) warp_heads[warp] = __popc(votes);
        __syncthreads();
        uint64_t r = rank + __popc(votes & ((1u << lane) - 1u));
        for (uint32_t w = 0; w < kRleThreads / 32; ++w) {
            r += w < warp ? warp_heads[w] : 0u;
            rank += warp_heads[w];
        }
        if (head) {
            outcomes[r] = v;
            first[r] = i;
        }
        __syncthreads();
    }
}

__global__ void k_run_lengths(const uint64_t* __restrict__ first, const uint64_t* __restrict__ runs, uint64_t shots,
                              uint64_t* __restrict__ counts) {
    const uint64_t n = *runs;
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        counts[r] = (r + 1 < n ? first[r + 1] : shots) - first[r];
}

size_t al(size_t b) { return (b + 255) & ~size_t{255}; }
unsigned blocks_for(uint64_t items, uint64_t per) {
    const uint64_t b = (items + per - 1) / per;
    return static_cast<unsigned>(b < 1184 ? b : 1184);  // 148 SMs, eight CTAs of 256 threads each
}

}  // namespace

size_t uniforms_scratch_bytes(uint64_t shots) {
    const uint64_t nb = uint64_t{1} << bucket_bits(shots);
    return al(mt_room(shots) * 8) + al(shots * 8) + al(shots * 4) + al(nb * 4) + al((nb + 1) * 8);
}

int launch_sort_words(const uint64_t* words, uint64_t shots, void* scratch, double* dev_u, void* stream) {
    const auto s = static_cast<cudaStream_t>(stream);
    const uint32_t bits = bucket_bits(shots);
    const uint64_t nb = uint64_t{1} << bits;
    auto* p = static_cast<unsigned char*>(scratch) + al(mt_room(shots) * 8);
    auto* keys = reinterpret_cast<uint64_t*>(p);
    p += al(shots * 8);
    auto* place = reinterpret_cast<uint32_t*>(p);
    p += al(shots * 4);
    auto* count = reinterpret_cast<uint32_t*>(p);
    p += al(nb * 4);
    auto* start = reinterpret_cast<uint64_t*>(p);
    if (cudaError_t e = cudaMemsetAsync(count, 0, nb * 4, s); e != cudaSuccess) return record_cuda_error(e);
    k_bucket_count<<<blocks_for(shots, 256), 256, 0, s>>>(words, shots, 53 - bits, count, place);
    k_scan<<<1, 1024, 0, s>>>(count, nb, start);
    k_bucket_scatter<<<blocks_for(shots, 256), 256, 0, s>>>(words, shots, 53 - bits, start, place, keys);
    k_bucket_sort<<<static_cast<unsigned>(nb), kSortThreads, 0, s>>>(keys, start, dev_u);
    note_launches(4);
    return launch_status();
}

int launch_sorted_uniforms(uint64_t shots, uint64_t seed, void* scratch, double* dev_u, void* stream) {
    auto* words = static_cast<uint64_t*>(scratch);
    k_words<<<1, kWordThreads, 0, static_cast<cudaStream_t>(stream)>>>(MtSeed(seed), shots, words);
    note_launches(1);
    if (int rc = launch_status(); rc != MB2_OK) return rc;
    return launch_sort_words(words, shots, scratch, dev_u, stream);
}

size_t runs_scratch_bytes(uint64_t shots) {
    const uint64_t tiles = (shots + kRleTile - 1) / kRleTile;
    return al(tiles * 4) + al((tiles + 1) * 8) + al(shots * 8);
}

int launch_runs(const uint64_t* dev_basis, uint64_t shots, void* scratch, uint64_t* dev_outcomes,
                uint64_t* dev_counts, const uint64_t** dev_runs, void* stream) {
    const auto s = static_cast<cudaStream_t>(stream);
    const uint64_t tiles = (shots + kRleTile - 1) / kRleTile;
    auto* p = static_cast<unsigned char*>(scratch);
    auto* heads = reinterpret_cast<uint32_t*>(p);
    p += al(tiles * 4);
    auto* before = reinterpret_cast<uint64_t*>(p);
    p += al((tiles + 1) * 8);
    auto* first = reinterpret_cast<uint64_t*>(p);
    k_run_count<<<static_cast<unsigned>(tiles), kRleThreads, 0, s>>>(dev_basis, shots, heads);
    k_scan<<<1, 1024, 0, s>>>(heads, tiles, before);
    k_run_heads<<<static_cast<unsigned>(tiles), kRleThreads, 0, s>>>(dev_basis, shots, before, dev_outcomes, first);
    k_run_lengths<<<blocks_for(shots, 256), 256, 0, s>>>(first, before + tiles, shots, dev_counts);
    *dev_runs = before + tiles;
    note_launches(4);
    return launch_status();
}

}  // namespace mb2
