// The reference's sort-then-walk (src/engines/dense/sample.cpp:55-69) by one
// CTA over a short list of probabilities: shot s, in ascending order of the
// uniforms u, goes to the first index whose running sum (in index order, each
// add rounded) exceeds u[s], and to the last index when none does.
//
// Only the sums are a serial chain.  The CTA fetches kWalkStage probabilities
// at once, one thread adds them in order (at the latency of an FP64 add, not
// of a load from memory per probability and per shot), and every shot below
// the stage's largest sum is placed by a binary search.  A density matrix's
// diagonal can hold roundings below zero, so sums can fall; the largest sum so
// far never does, and first exceeds u[s] at the same index as the sum itself.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mb2 {

constexpr uint32_t kWalkThreads = 512;
constexpr uint32_t kWalkStage = 2048;

// prob(i): the probability of index i < count.  blockDim.x == kWalkThreads.
template <typename PROB>
__device__ __forceinline__ void walk_cta(uint32_t count, PROB prob, const double* __restrict__ u, uint64_t shots,
                                         uint64_t* __restrict__ basis) {
    constexpr uint32_t kPer = kWalkStage / kWalkThreads;
    __shared__ double sums[kWalkStage], warp_top[kWalkThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    double cumulative = 0.0;  // thread 0
    double largest = -1.0;    // before this stage, in every thread (every u is at least 0)
    uint64_t s0 = 0;          // shots placed so far, in every thread
    for (uint32_t b0 = 0; b0 < count && s0 < shots; b0 += kWalkStage) {
        const uint32_t len = count - b0 < kWalkStage ? count - b0 : kWalkStage;
        for (uint32_t b = tid; b < len; b += kWalkThreads) sums[b] = prob(b0 + b);
        __syncthreads();
        if (tid == 0) {
#pragma unroll 16
            for (uint32_t b = 0; b < len; ++b) {
                cumulative = __dadd_rn(cumulative, sums[b]);
                sums[b] = cumulative;
            }
        }
        __syncthreads();
        // The largest sum up to each index (fmax passes over a NaN sum, which
        // exceeds nothing), kPer indexes a thread.
        double top[kPer];
        double run = -1.0;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t b = tid * kPer + k;
            run = fmax(run, b < len ? sums[b] : -1.0);
            top[k] = run;
        }
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run = fmax(run, v);
        }
        if (lane == 31) warp_top[warp] = run;
        double before = __shfl_up_sync(0xffffffffu, run, 1);
        if (lane == 0) before = -1.0;
        __syncthreads();
        double all = largest;
        for (uint32_t w = 0; w < kWalkThreads / 32; ++w) {
            if (w == warp) before = fmax(before, all);
            all = fmax(all, warp_top[w]);
        }
        largest = all;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) sums[tid * kPer + k] = fmax(before, top[k]);
        __syncthreads();
        uint64_t lo = s0, hi = shots;  // the shots below the stage's largest sum end here
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if (u[mid] < largest) lo = mid + 1;
            else hi = mid;
        }
        for (uint64_t s = s0 + tid; s < lo; s += kWalkThreads) {
            const double x = u[s];
            uint32_t a = 0, b = len - 1;  // x < sums[len - 1]
            while (a < b) {
                const uint32_t mid = (a + b) >> 1;
                if (x < sums[mid]) b = mid;
                else a = mid + 1;
            }
            basis[s] = b0 + a;
        }
        s0 = lo;
        __syncthreads();  // sums and warp_top are written again
    }
    for (uint64_t s = s0 + tid; s < shots; s += kWalkThreads) basis[s] = count - 1;
}

}  // namespace mb2
