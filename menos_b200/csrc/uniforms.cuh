// std::mt19937_64 (Matsumoto and Nishimura's 64-bit Mersenne Twister) by one
// CTA: the words of the reference's common::Rng, (w >> 11) being a uniform's
// numerator over 2^53 (src/common/rng.cpp:176-186).
//
// A word depends on the words 312, 311 and 156 places before it, so 156 words
// can be made at once: thread t holds x[t] and x[t + 156] and makes the next
// 312 words in two steps, of which only the neighbours' words (t + 1) cross
// threads -- through shared memory, double-buffered, one barrier per 312
// words.  The latency of a step bounds it (3205 of them for 1e6 words, 0.57 ms
// against 3 ms on a host core), so the tempering is left to the readers
// (mt_key): with it in the step the same words took 0.73 ms.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mb2 {

constexpr uint32_t kMtHalf = 156;
constexpr uint32_t kWordThreads = 160;  // five warps; four threads idle

// The generator's state after seeding.
struct MtSeed {
    uint64_t x[2 * kMtHalf];
    explicit MtSeed(uint64_t seed) {
        x[0] = seed;
        for (uint32_t i = 1; i < 2 * kMtHalf; ++i)
            x[i] = 6364136223846793005ull * (x[i - 1] ^ (x[i - 1] >> 62)) + i;
    }
};

__device__ __forceinline__ uint64_t mt_twist(uint64_t a, uint64_t next) {
    const uint64_t y = (a & 0xFFFFFFFF80000000ull) | (next & 0x7FFFFFFFull);
    return (y >> 1) ^ ((y & 1) ? 0xB5026F5AA96619E9ull : 0ull);
}

// A uniform's numerator from a state word.
__device__ __forceinline__ uint64_t mt_key(uint64_t x) {
    x ^= (x >> 29) & 0x5555555555555555ull;
    x ^= (x << 17) & 0x71D67FFFEDA60000ull;
    x ^= (x << 37) & 0xFFF7EEE000000000ull;
    return (x ^ (x >> 43)) >> 11;
}

// words[i] = state word i (mt_key of it is the key), i < count.  Called by
// the first kWordThreads threads of a CTA; `words` has room for whole steps
// of 312 (mt_room).
__host__ __device__ constexpr uint64_t mt_room(uint64_t count) {
    return (count + 2 * kMtHalf - 1) / (2 * kMtHalf) * (2 * kMtHalf);
}
__device__ __forceinline__ void mt_words(const MtSeed& seed, uint64_t count, uint64_t* __restrict__ words) {
    __shared__ uint64_t sh[2][2 * kMtHalf];
    const uint32_t t = threadIdx.x;
    const bool on = t < kMtHalf;
    uint64_t a = on ? seed.x[t] : 0, b = on ? seed.x[t + kMtHalf] : 0;
    uint32_t cur = 0;
    for (uint64_t base = 0; base < count; base += 2 * kMtHalf, cur ^= 1u) {
        uint64_t* x = sh[cur];
        if (on) {
            x[t] = a;
            x[t + kMtHalf] = b;
        }
        // (The other buffer's readers of the step before have all arrived
        // here, so the next step may write it.)
        asm volatile("bar.sync 1, %0;\n" ::"n"(kWordThreads) : "memory");
        if (on) {
            const uint64_t a_next = x[t + 1];
            // The word after the last one is the first of the new words.
            const uint64_t b_next = t + 1 < kMtHalf ? x[t + 1 + kMtHalf] : x[kMtHalf] ^ mt_twist(x[0], x[1]);
            a = b ^ mt_twist(a, a_next);
            b = a ^ mt_twist(b, b_next);
            words[base + t] = a;
            words[base + t + kMtHalf] = b;
        }
    }
}

}  // namespace mb2
