// Device counts sampler with the reference's exact results.
//
// The reference (src/engines/dense/sample.cpp:24-75) sorts `shots` uniforms
// and walks the basis states once, cumulative = fl(cumulative + |a_i|^2)
// strictly in index order; shot s lands on the first basis state i whose
// running sum c_i exceeds u_s, and shots past the end go to the last state.
// The running sum drifts from the exact prefix sum by up to ~N ulps, so a
// plain parallel scan would move shots.  This sampler reproduces the chain
// c_i bit for bit in parallel:
//
// Within one binade [2^e, 2^(e+1)) every c is M*u with u = 2^(e-52) and
// M in [2^52, 2^53).  Adding p = (k + f) u (k integer, 0 <= f < 1, exact
// since p/u is a power-of-two scaling) rounds to (M + k) u for f < 1/2,
// (M + k + 1) u for f > 1/2 and, on a tie, to whichever of the two has an
// even M.  So each element is a map from the parity of M to an increment;
// those maps compose associatively, and a chunk of 4096 elements reduces to
// one such map.  Chunks whose run stays inside one binade are advanced in
// O(1) from their exact start value; chunks that cross a binade boundary
// (the first few, while the sum is small, and one per boundary) are advanced
// by runs of 16 elements, the crossing run with the reference's own FP64
// adds.  The chunk's binade is guessed from an approximate prefix sum; a
// wrong guess only costs that longer way, never the result.
//
// At 27 qubits and 1e6 shots (a 2 GiB state, three reads of it): 2.96 ms with
// one-CTA scans, element-by-element crossings, ldexp and floor per element
// and threads loading their own runs; 1.8 ms now, draws and their sort included.
//
// |a|^2 is re*re + im*im with each product and the sum rounded (std::norm,
// no FMA).
#include <cuda_runtime.h>

#include <cstdint>

#include "mb2_internal.h"
#include "uniforms.cuh"

namespace mb2 {
namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = kSampleChunk / kThreads;  // 16

__device__ __forceinline__ double prob(double2 a) { return __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y)); }
// A complex64 amplitude's probability in FP64 (the squares of FP32 values are exact).
__device__ __forceinline__ double prob(float2 a) {
    return __dadd_rn(__dmul_rn(static_cast<double>(a.x), static_cast<double>(a.x)),
                     __dmul_rn(static_cast<double>(a.y), static_cast<double>(a.y)));
}

// Step A: approximate chunk sums (any order; only used to guess binades).
template <typename A>
__device__ __forceinline__ void chunk_sum(const A* __restrict__ st, uint64_t n_amps, uint32_t chunk, uint64_t j,
                                          double* __restrict__ sums) {
    const uint64_t base = j * chunk;
    double s = 0.0;
    for (uint32_t i = threadIdx.x; i < chunk; i += kThreads)
        if (base + i < n_amps) s += prob(st[base + i]);
    __shared__ double sh[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) t += sh[w];
        sums[j] = t;
    }
}

template <typename A>
__global__ void __launch_bounds__(kThreads) k_chunk_sums(const A* __restrict__ st, uint64_t n_amps,
                                                         uint32_t chunk, double* __restrict__ sums) {
    const uint64_t t = blockIdx.y;
    chunk_sum(st + t * n_amps, n_amps, chunk, blockIdx.x, sums + t * gridDim.x);
}

// The same beside the draws' generator, whose chain of steps runs on one CTA
// (the first) while the others read the state.
template <typename A>
__global__ void __launch_bounds__(kThreads)
    k_chunk_sums_words(const A* __restrict__ st, uint64_t n_amps, uint32_t chunk, double* __restrict__ sums,
                       const __grid_constant__ MtSeed seed, uint64_t shots, uint64_t* __restrict__ words) {
    if (blockIdx.x == 0) {
        if (threadIdx.x < kWordThreads) mt_words(seed, shots, words);
        return;
    }
    chunk_sum(st, n_amps, chunk, blockIdx.x - 1, sums);
}

// Step B: exclusive scan of the chunk sums within each block of kScanBlock
// chunks (approximate), and each block's total; step C adds the totals of
// the blocks before its own.
constexpr uint32_t kScanBlock = 1024;
__global__ void __launch_bounds__(kScanBlock) k_scan_sums(const double* __restrict__ sums, uint64_t nchunks,
                                                          double* __restrict__ starts, double* __restrict__ totals) {
    __shared__ double warp_sum[32];
    sums += blockIdx.y * nchunks;
    starts += blockIdx.y * nchunks;
    totals += static_cast<uint64_t>(blockIdx.y) * gridDim.x;
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * kScanBlock + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const double v = i < nchunks ? sums[i] : 0.0;
    double s = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const double q = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += q;
    }
    if (lane == 31) warp_sum[warp] = s;
    __syncthreads();
    double before = 0.0, total = 0.0;
    for (uint32_t w = 0; w < 32; ++w) {
        before += w < warp ? warp_sum[w] : 0.0;
        total += warp_sum[w];
    }
    if (i < nchunks) starts[i] = before + (s - v);
    if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// A parity map: what a run of elements adds to M when M is even (inc0) or odd
// (inc1).  The parity afterwards follows from the sum.
struct PMap {
    long long inc0, inc1;
};

__device__ __forceinline__ PMap compose(const PMap& a, const PMap& b) {
    // a then b
    return PMap{a.inc0 + ((a.inc0 & 1) ? b.inc1 : b.inc0), a.inc1 + ((a.inc1 & 1) ? b.inc0 : b.inc1)};
}

__device__ __forceinline__ PMap shfl_up(const PMap& m, uint32_t o) {
    return PMap{__shfl_up_sync(0xffffffffu, m.inc0, o), __shfl_up_sync(0xffffffffu, m.inc1, o)};
}

// One element's map, scale = 1 / u.  q = p / u (an exact scaling), at most
// 2^52: from 2^52 on, the element takes M out of its binade whatever it was.
// Adding 2^52 rounds q to an integer, to the even one on a tie, which is what
// the sum M + q does for an even M; an odd M takes the tie's other side.
// (Two FP64 adds and integer work: ldexp, floor and a conversion for each
// element were what bounded steps C and E.)
constexpr double kTwo52 = 4503599627370496.0;
__device__ __forceinline__ PMap element_map(double p, double scale) {
    double q = __dmul_rn(p, scale);
    q = q < kTwo52 ? q : kTwo52;
    const double t = __dadd_rn(q, kTwo52);
    const double d = __dsub_rn(q, __dsub_rn(t, kTwo52));
    const long long r = __double_as_longlong(t) - __double_as_longlong(kTwo52);
    return PMap{r, fabs(d) == 0.5 ? (d > 0.0 ? r + 1 : r - 1) : r};
}

__device__ __forceinline__ int binade_of(double c) {
    int e;
    frexp(c, &e);  // c = f * 2^e, f in [0.5, 1): binade 2^(e-1)
    return e - 1;
}

// Binades the maps are used in: u and 1 / u are normal numbers there.
constexpr int kMinBinade = -900, kMaxBinade = 900;

// A chunk's probabilities in shared memory, read from the state in
// contiguous order: element i at pad(i), so that threads reading their runs
// of 16 elements hit distinct banks (a thread loading its own run straight
// from memory touches a line of its own per load).
__device__ __forceinline__ uint32_t pad(uint32_t i) { return i + (i >> 4); }
constexpr uint32_t kPadded = kSampleChunk + kSampleChunk / 16;
static_assert(kPerThread == 16, "pad() spaces runs of 16");

template <typename A>
__device__ __forceinline__ void stage_chunk(const A* __restrict__ st, uint64_t base, uint32_t chunk, double* sh) {
    if (chunk == kSampleChunk) {
        A v[kPerThread];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) v[k] = st[base + k * kThreads + threadIdx.x];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) sh[pad(k * kThreads + threadIdx.x)] = prob(v[k]);
    } else {
        for (uint32_t i = threadIdx.x; i < kSampleChunk; i += kThreads) sh[pad(i)] = i < chunk ? prob(st[base + i]) : 0.0;
    }
    __syncthreads();
}

// Step C: each chunk's composed map for the binade its approximate start
// lies in.  A chunk whose approximate range is not safely inside one binade
// is marked for the exact chain (step D).
struct ChunkMap {
    long long inc0, inc1;
    int e;      // binade the map is for
    int valid;  // 0: crossed by the exact chain
};

template <typename A>
__global__ void __launch_bounds__(kThreads) k_chunk_maps(const A* __restrict__ st, uint64_t n_amps,
                                                         uint32_t chunk, const double* __restrict__ starts,
                                                         const double* __restrict__ totals,
                                                         const double* __restrict__ sums,
                                                         ChunkMap* __restrict__ maps) {
    __shared__ double sh[kPadded];
    __shared__ double s_start;
    const uint64_t j = blockIdx.x, nchunks = gridDim.x;
    const uint64_t base = j * chunk;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    st += blockIdx.y * n_amps;
    starts += blockIdx.y * nchunks;
    totals += blockIdx.y * ((nchunks + kScanBlock - 1) / kScanBlock);
    sums += blockIdx.y * nchunks;
    maps += blockIdx.y * nchunks;
    if (warp == 0) {
        double t = 0.0;
        for (uint64_t b = lane; b < j / kScanBlock; b += 32) t += totals[b];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) s_start = t + starts[j];
    }
    __syncthreads();
    const double a = s_start;
    const double hi = a + sums[j];
    // Generous drift allowance (relative): the chain's rounding drift plus
    // the approximate scan's error.
    const double slack = (static_cast<double>(base + chunk) + 1.0e6) * 2.3e-16;
    const int e = a > 0.0 ? binade_of(a) : -2000;
    const double lo_edge = ldexp(1.0, e), hi_edge = ldexp(1.0, e + 1);
    const bool ok = a > 0.0 && e > kMinBinade && e < kMaxBinade && a * (1.0 - slack) > lo_edge &&
                    hi * (1.0 + slack) < hi_edge;
    if (!ok) {  // (uniform over the CTA)
        if (threadIdx.x == 0) maps[j] = ChunkMap{0, 0, e, 0};
        return;
    }
    stage_chunk(st, base, chunk, sh);
    // Each thread composes its contiguous run of 16 elements in order.
    const double scale = ldexp(1.0, 52 - e);
    PMap acc{0, 0};
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) acc = compose(acc, element_map(sh[pad(threadIdx.x * kPerThread + i)], scale));
    // Ordered reduction across the block: warp shuffles (lane order), then warps.
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const PMap other{__shfl_down_sync(0xffffffffu, acc.inc0, o), __shfl_down_sync(0xffffffffu, acc.inc1, o)};
        if ((lane & (2 * o - 1)) == 0) acc = compose(acc, other);
    }
    __shared__ PMap wm[kThreads / 32];
    if (lane == 0) wm[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        PMap t = wm[0];
        for (int w = 1; w < kThreads / 32; ++w) t = compose(t, wm[w]);
        maps[j] = ChunkMap{t.inc0, t.inc1, e, 1};
    }
}

// The exact chain across one chunk by the whole CTA: sh holds the chunk's
// probabilities (stage_chunk); returns the sum after it from the sum c before
// it (the same in every thread).  STORE: sh's elements become the running
// sums.  Runs of 16 elements are advanced by maps of c's binade up to the
// first run whose end leaves it; that run is added element by element, and
// the rest continues in the new binade.  A chunk crosses a binade rarely (the
// first chunk about a dozen times), and adding its 4096 elements one after
// another took 36 us where this takes a few per crossing.
constexpr long long kSaturated = 1LL << 59;  // past every binade's end; a sum of 15 of them fits

template <bool STORE>
__device__ __forceinline__ double walk_run(double* sh, uint32_t run, double c) {
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
        double& x = sh[pad(run * kPerThread + i)];
        c = __dadd_rn(c, x);
        if (STORE) x = c;
    }
    return c;
}

template <bool STORE>
__device__ double chain_chunk(double* sh, double c) {
    __shared__ PMap warp_map[kThreads / 32];
    __shared__ uint32_t warp_first[kThreads / 32];
    __shared__ double s_c;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    bool finite = true, some = false;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
        const double x = sh[pad(tid * kPerThread + i)];
        finite = finite && x >= 0.0 && x <= 1.7976931348623157e308;
        some = some || x != 0.0;
    }
    if (!__syncthreads_and(finite)) {
        // Not probabilities (a NaN or infinite amplitude): one thread, in
        // order.  No uniform is below a NaN sum, so the stored sums stay at
        // the largest one before it.
        if (tid == 0) {
            double cc = c, top = c;
            for (uint32_t i = 0; i < kSampleChunk; ++i) {
                double& x = sh[pad(i)];
                cc = __dadd_rn(cc, x);
                top = cc > top ? cc : top;
                if (STORE) x = top;
            }
            s_c = cc;
        }
        __syncthreads();
        return s_c;
    }
    uint32_t pos = 0;  // the first run not yet passed
    while (pos < kThreads) {
        uint32_t walked;  // the run added element by element (kThreads: none)
        double c_run = c;
        if (!(c >= 0x1p-880 && c < 0x1p880)) {
            // Nothing summed yet (or out of the maps' range): on to the next
            // run that holds something.
            const uint32_t votes = __ballot_sync(0xffffffffu, tid >= pos && some);
            if (lane == 0) warp_first[warp] = votes ? warp * 32 + __ffs(votes) - 1 : kThreads;
            __syncthreads();
            walked = kThreads;
            for (uint32_t w = 0; w < kThreads / 32; ++w) walked = min(walked, warp_first[w]);
            if (STORE && tid >= pos && tid < walked) {
#pragma unroll
                for (int i = 0; i < kPerThread; ++i) sh[pad(tid * kPerThread + i)] = c;
            }
            if (walked == kThreads) return c;
        } else {
            const int e = binade_of(c);
            const double u = ldexp(1.0, e - 52), scale = ldexp(1.0, 52 - e);
            const long long m0 = static_cast<long long>(__dmul_rn(c, scale));  // exact: c is on the grid
            PMap inc{0, 0};
            if (tid >= pos) {
#pragma unroll
                for (int i = 0; i < kPerThread; ++i)
                    inc = compose(inc, element_map(sh[pad(tid * kPerThread + i)], scale));
            }
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const PMap prev = shfl_up(inc, o);
                if (lane >= o) inc = compose(prev, inc);
            }
            inc.inc0 = min(inc.inc0, kSaturated);
            inc.inc1 = min(inc.inc1, kSaturated);
            if (lane == 31) warp_map[warp] = inc;
            __syncthreads();
            PMap before{0, 0};
            for (uint32_t w = 0; w < warp; ++w) before = compose(before, warp_map[w]);
            PMap ex = shfl_up(inc, 1);
            if (lane == 0) ex = PMap{0, 0};
            ex = compose(before, ex);
            inc = compose(before, inc);
            const bool odd = m0 & 1;
            const long long m_end = m0 + (odd ? inc.inc1 : inc.inc0);
            // The sums never fall, so the runs past the binade's end are the last ones.
            walked = kThreads - __syncthreads_count(tid >= pos && m_end >= (1LL << 53));
            long long m = m0 + (odd ? ex.inc1 : ex.inc0);
            if (tid == walked) c_run = static_cast<double>(m) * u;  // exact: m < 2^53
            if (STORE && tid >= pos && tid < walked) {
#pragma unroll
                for (int i = 0; i < kPerThread; ++i) {
                    double& x = sh[pad(tid * kPerThread + i)];
                    const PMap em = element_map(x, scale);
                    m += (m & 1) ? em.inc1 : em.inc0;
                    x = static_cast<double>(m) * u;
                }
            }
            if (walked == kThreads) {
                if (tid == kThreads - 1) s_c = static_cast<double>(m_end) * u;
                __syncthreads();
                return s_c;
            }
        }
        if (tid == walked) s_c = walk_run<STORE>(sh, tid, c_run);
        __syncthreads();
        c = s_c;
        pos = walked + 1;
        __syncthreads();  // s_c and the warps' words are written again
    }
    return c;
}

// Step D: the exact chain at every chunk start.
//
// D1: chunks whose maps are valid for the same binade form segments (cut at
// every kSegBlock chunks); a segmented scan gives each chunk the composition
// of the segment's chunks before it (`excl`) and each segment head the whole
// segment's map and length.
// D2 (one CTA): walks the segments in order with the exact running value c.
// A segment is crossed in O(1) when c lies in its binade and the segment does
// not leave it; otherwise its chunks are taken one at a time (O(1) per chunk
// under the same checks, or chain_chunk).
// D3 (step E's bounds): the start of every chunk inside a crossed segment,
// exactly, from the segment's start value and `excl`.
// cstart[j] = the chain before chunk j; cstart[nchunks] = the final sum.
struct SMap {
    PMap map;
    unsigned count;
    unsigned pad;
};

constexpr uint32_t kSegThreads = 512;
constexpr uint32_t kSegPer = 4;
constexpr uint32_t kSegBlock = kSegThreads * kSegPer;

__device__ __forceinline__ bool seg_head(const ChunkMap* maps, uint64_t j) {
    if (j % kSegBlock == 0 || !maps[j].valid || !maps[j - 1].valid) return true;
    return maps[j].e != maps[j - 1].e;
}

// a then b, unless b begins a segment of its own (head).
__device__ __forceinline__ SMap seg_compose(const SMap& a, const SMap& b, bool b_head) {
    if (b_head) return b;
    return SMap{compose(a.map, b.map), a.count + b.count, 0};
}

// One CTA per kSegBlock chunks, kSegPer contiguous chunks a thread.
__global__ void __launch_bounds__(kSegThreads) k_seg_scan(const ChunkMap* __restrict__ maps, uint64_t nchunks,
                                                          SMap* __restrict__ excl, SMap* __restrict__ seg_total,
                                                          unsigned char* __restrict__ direct) {
    __shared__ SMap warp_agg[kSegThreads / 32];
    __shared__ bool warp_head[kSegThreads / 32];
    maps += blockIdx.y * nchunks;
    excl += blockIdx.y * nchunks;
    seg_total += blockIdx.y * nchunks;
    direct += blockIdx.y * nchunks;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t b = static_cast<uint64_t>(blockIdx.x) * kSegBlock + threadIdx.x * kSegPer;
    SMap one[kSegPer];
    bool head[kSegPer + 1];
    SMap agg{{0, 0}, 0, 0};
    bool any = false;
#pragma unroll
    for (uint32_t i = 0; i < kSegPer; ++i) {
        const uint64_t j = b + i;
        one[i] = SMap{{0, 0}, 0, 0};
        head[i] = false;
        if (j < nchunks) {
            one[i] = SMap{{maps[j].inc0, maps[j].inc1}, 1, 0};
            head[i] = seg_head(maps, j);
            direct[j] = 0;
        }
        agg = seg_compose(agg, one[i], head[i]);
        any = any || head[i];
    }
    head[kSegPer] = b + kSegPer >= nchunks || seg_head(maps, b + kSegPer);
    // Inclusive segmented scan over the warp, then the warps before.
    SMap inc = agg;
    bool inc_head = any;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        SMap prev;
        prev.map = shfl_up(inc.map, o);
        prev.count = __shfl_up_sync(0xffffffffu, inc.count, o);
        prev.pad = 0;
        const bool prev_head = __shfl_up_sync(0xffffffffu, inc_head, o);
        if (lane >= o) {
            inc = seg_compose(prev, inc, inc_head);
            inc_head = inc_head || prev_head;
        }
    }
    if (lane == 31) {
        warp_agg[warp] = inc;
        warp_head[warp] = inc_head;
    }
    __syncthreads();
    SMap before{{0, 0}, 0, 0};
    for (uint32_t w = 0; w < warp; ++w) before = seg_compose(before, warp_agg[w], warp_head[w]);
    SMap run;  // the open segment before this thread's chunks
    run.map = shfl_up(inc.map, 1);
    run.count = __shfl_up_sync(0xffffffffu, inc.count, 1);
    run.pad = 0;
    const bool run_head = __shfl_up_sync(0xffffffffu, inc_head, 1);
    run = lane == 0 ? before : seg_compose(before, run, run_head);
#pragma unroll
    for (uint32_t i = 0; i < kSegPer; ++i) {
        const uint64_t j = b + i;
        if (j >= nchunks) break;
        if (head[i]) run = SMap{{0, 0}, 0, 0};
        excl[j] = run;
        run = seg_compose(run, one[i], false);
        const bool last = j + 1 == nchunks || (i + 1 < kSegPer ? head[i + 1] : head[kSegPer]);
        if (last) seg_total[j + 1 - run.count] = run;
    }
}

__device__ __forceinline__ bool advance_exact(double& c, int e, const PMap& m) {
    if (!(c > 0.0) || binade_of(c) != e) return false;
    const double u = ldexp(1.0, e - 52);
    const long long M = static_cast<long long>(c / u);  // exact: c is on the grid
    const long long M2 = M + ((M & 1) ? m.inc1 : m.inc0);
    if (M2 >= (1LL << 53)) return false;
    c = static_cast<double>(M2) * u;  // exact: M2 < 2^53
    return true;
}

template <typename A>
__global__ void __launch_bounds__(kThreads) k_seg_chain(const A* __restrict__ st, uint64_t n_amps, uint32_t chunk,
                                                        uint64_t nchunks, const ChunkMap* __restrict__ maps,
                                                        const SMap* __restrict__ seg_total,
                                                        double* __restrict__ cstart,
                                                        unsigned char* __restrict__ direct,
                                                        double* __restrict__ seg_c) {
    __shared__ double sh[kPadded];
    st += blockIdx.y * n_amps;
    maps += blockIdx.y * nchunks;
    seg_total += blockIdx.y * nchunks;
    cstart += blockIdx.y * (nchunks + 1);
    direct += blockIdx.y * nchunks;
    seg_c += blockIdx.y * nchunks;
    double c = 0.0;  // (the same in every thread, as is everything that steers the loop)
    uint64_t j = 0;
    while (j < nchunks) {
        const ChunkMap m = maps[j];
        const SMap t = seg_total[j];  // read with the map, used at a segment's head only
        if (seg_head(maps, j) && m.valid) {
            double c2 = c;
            if (advance_exact(c2, m.e, t.map)) {
                if (threadIdx.x == 0) seg_c[j] = c;
                c = c2;
                j += t.count;
                continue;
            }
        }
        // This chunk on its own.
        if (threadIdx.x == 0) {
            cstart[j] = c;
            direct[j] = 1;
        }
        if (!(m.valid && advance_exact(c, m.e, PMap{m.inc0, m.inc1}))) {
            __syncthreads();
            stage_chunk(st, j * chunk, chunk, sh);
            c = chain_chunk<false>(sh, c);
        }
        ++j;
    }
    if (threadIdx.x == 0) cstart[nchunks] = c;
}

// Number of sorted uniforms strictly below x.
__device__ __forceinline__ uint64_t count_below(const double* __restrict__ u, uint64_t shots, double x) {
    uint64_t lo = 0, hi = shots;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (u[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The chain of a state of one chunk.
template <typename A>
__global__ void __launch_bounds__(kThreads) k_chain_one(const A* __restrict__ st, uint32_t n_amps,
                                                        double* __restrict__ cstart) {
    __shared__ double sh[kPadded];
    stage_chunk(st + static_cast<uint64_t>(blockIdx.y) * n_amps, 0, n_amps, sh);
    const double c = chain_chunk<false>(sh, 0.0);
    if (threadIdx.x == 0) cstart[2 * blockIdx.y + 1] = c;
}

// Every chunk's exact start, and its shot index: bounds[j] = the uniforms
// below cstart[j] (j = 0..nchunks), one thread per boundary, so the searches'
// dependent loads overlap across the grid.
__global__ void __launch_bounds__(kThreads) k_shot_bounds(uint64_t nchunks, const ChunkMap* __restrict__ maps,
                                                          const SMap* __restrict__ excl,
                                                          const unsigned char* __restrict__ direct,
                                                          const double* __restrict__ seg_c,
                                                          double* __restrict__ cstart, const double* __restrict__ u,
                                                          uint64_t shots, uint64_t* __restrict__ bounds) {
    const uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j > nchunks) return;
    double c;
    if (j == nchunks || direct[j]) {
        c = cstart[j];
    } else {
        const SMap x = excl[j];
        const double c0 = seg_c[j - x.count];
        const double g = ldexp(1.0, maps[j].e - 52);
        const long long M = static_cast<long long>(c0 / g);
        c = static_cast<double>(M + ((M & 1) ? x.map.inc1 : x.map.inc0)) * g;
        cstart[j] = c;
    }
    // After a NaN sum nothing is placed any more: the shots that are left
    // belong to the chunk that holds it.
    bounds[j] = c != c ? shots : count_below(u, shots, c);
}

// Step E: per chunk, the exact running sums of its elements, then each of
// its shots placed on the first element whose sum exceeds the uniform.
// Shots at or past the final sum go to the last basis state.  A state of one
// chunk needs no other step: its chain starts at zero and every shot is its
// own (bounds == nullptr).
template <typename A>
__global__ void __launch_bounds__(kThreads) k_assign(const A* __restrict__ st, uint64_t n_amps,
                                                     uint32_t chunk, uint64_t nchunks,
                                                     const double* __restrict__ cstart,
                                                     const double* __restrict__ u, uint64_t shots,
                                                     const uint64_t* __restrict__ bounds,
                                                     uint64_t* __restrict__ basis) {
    __shared__ double cs[kPadded];
    const uint64_t j = blockIdx.x;
    const uint64_t base = j * chunk;
    const uint64_t lo = bounds == nullptr ? 0 : bounds[j], hi = bounds == nullptr ? shots : bounds[j + 1];
    if (bounds != nullptr && j + 1 == nchunks)
        for (uint64_t s = bounds[nchunks] + threadIdx.x; s < shots; s += kThreads) basis[s] = n_amps - 1;
    if (lo >= hi) return;  // (uniform over the CTA)
    stage_chunk(st, base, chunk, cs);
    chain_chunk<true>(cs, bounds == nullptr ? 0.0 : cstart[j]);
    __syncthreads();
    for (uint64_t s = lo + threadIdx.x; s < hi; s += kThreads) {
        const double x = u[s];
        uint32_t a = 0, b = chunk;  // first i with x < cs[i]
        while (a < b) {
            const uint32_t mid = (a + b) >> 1;
            if (x < cs[pad(mid)]) b = mid;
            else a = mid + 1;
        }
        basis[s] = a < chunk ? base + a : n_amps - 1;  // (past the final sum, or a NaN one)
    }
}

}  // namespace

namespace {

// The chain's arrays in a caller's scratch.
struct Scratch {
    uint64_t nchunks;
    uint32_t chunk;
    double *sums, *starts, *totals, *cstart, *seg_c;
    ChunkMap* maps;
    SMap *excl, *seg_total;
    unsigned char* direct;
    uint64_t* bounds;
    size_t bytes;
    // Steps A to D run for `batch` states at once (one after another in memory,
    // the grid's y), each with its own part of every array.
    Scratch(uint32_t n, void* scratch, uint64_t batch = 1) {
        const uint64_t na = uint64_t{1} << n;
        chunk = static_cast<uint32_t>(na < kSampleChunk ? na : kSampleChunk);
        nchunks = na / chunk;
        bytes = 0;
        auto take = [&](size_t b) {
            void* p = static_cast<unsigned char*>(scratch) + bytes;
            bytes += (b + 255) & ~size_t{255};
            return p;
        };
        sums = static_cast<double*>(take(batch * nchunks * 8));
        starts = static_cast<double*>(take(batch * nchunks * 8));
        totals = static_cast<double*>(take(batch * ((nchunks + kScanBlock - 1) / kScanBlock) * 8));
        cstart = static_cast<double*>(take(batch * (nchunks + 1) * 8));
        seg_c = static_cast<double*>(take(batch * nchunks * 8));
        maps = static_cast<ChunkMap*>(take(batch * nchunks * sizeof(ChunkMap)));
        excl = static_cast<SMap*>(take(batch * nchunks * sizeof(SMap)));
        seg_total = static_cast<SMap*>(take(batch * nchunks * sizeof(SMap)));
        direct = static_cast<unsigned char*>(take(batch * nchunks));
        bounds = static_cast<uint64_t*>(take(batch * (nchunks + 1) * 8));
    }
};

// Steps B to D (after the chunk sums).
template <typename A>
void launch_chain(const A* st, uint32_t n, const Scratch& w, cudaStream_t s, uint32_t batch = 1) {
    const uint64_t na = uint64_t{1} << n;
    const auto blocks = [&](uint64_t per) { return dim3(static_cast<unsigned>((w.nchunks + per - 1) / per), batch); };
    k_scan_sums<<<blocks(kScanBlock), kScanBlock, 0, s>>>(w.sums, w.nchunks, w.starts, w.totals);
    k_chunk_maps<<<blocks(1), kThreads, 0, s>>>(st, na, w.chunk, w.starts, w.totals, w.sums, w.maps);
    k_seg_scan<<<blocks(kSegBlock), kSegThreads, 0, s>>>(w.maps, w.nchunks, w.excl, w.seg_total, w.direct);
    k_seg_chain<<<dim3(1, batch), kThreads, 0, s>>>(st, na, w.chunk, w.nchunks, w.maps, w.seg_total, w.cstart,
                                                    w.direct, w.seg_c);
}

// The exact chain alone: the reference's sequential sum of |a_i|^2 over each
// whole state is its final value, cstart[nchunks].
template <typename A>
void launch_norms_t(const A* st, uint32_t n, uint32_t batch, const Scratch& w, cudaStream_t s) {
    if (w.nchunks == 1) {
        k_chain_one<<<dim3(1, batch), kThreads, 0, s>>>(st, w.chunk, w.cstart);
        note_launches(1);
        return;
    }
    k_chunk_sums<<<dim3(static_cast<unsigned>(w.nchunks), batch), kThreads, 0, s>>>(st, uint64_t{1} << n, w.chunk,
                                                                                    w.sums);
    launch_chain(st, n, w, s, batch);
    note_launches(5);
}

// dev_u: the sorted uniforms, or with draw != nullptr where they go, the
// draws being made on the way (sort_scratch: uniforms_scratch_bytes).
template <typename A>
int launch_sample_t(const void* amps, uint32_t n, double* dev_u, uint64_t shots, const uint64_t* draw,
                    void* sort_scratch, void* scratch, uint64_t* dev_basis, cudaStream_t s) {
    const auto* st = static_cast<const A*>(amps);
    const uint64_t na = uint64_t{1} << n;
    const Scratch w(n, scratch);
    const bool one = w.nchunks == 1;
    if (draw != nullptr && !one) {
        auto* words = static_cast<uint64_t*>(sort_scratch);
        k_chunk_sums_words<<<static_cast<unsigned>(w.nchunks + 1), kThreads, 0, s>>>(st, na, w.chunk, w.sums,
                                                                                     MtSeed(*draw), shots, words);
        if (int rc = launch_sort_words(words, shots, sort_scratch, dev_u, s); rc != MB2_OK) return rc;
    } else if (draw != nullptr) {
        if (int rc = launch_sorted_uniforms(shots, *draw, sort_scratch, dev_u, s); rc != MB2_OK) return rc;
    } else if (!one) {
        k_chunk_sums<<<static_cast<unsigned>(w.nchunks), kThreads, 0, s>>>(st, na, w.chunk, w.sums);
    }
    if (!one) {
        launch_chain(st, n, w, s);
        k_shot_bounds<<<static_cast<unsigned>((w.nchunks + 1 + kThreads - 1) / kThreads), kThreads, 0, s>>>(
            w.nchunks, w.maps, w.excl, w.direct, w.seg_c, w.cstart, dev_u, shots, w.bounds);
    }
    k_assign<<<static_cast<unsigned>(w.nchunks), kThreads, 0, s>>>(st, na, w.chunk, w.nchunks, w.cstart, dev_u, shots,
                                                                   one ? nullptr : w.bounds, dev_basis);
    note_launches(one ? 1 : 7);
    return launch_status();
}

}  // namespace

size_t sample_scratch_bytes(uint32_t n, uint64_t shots) {
    (void)shots;
    return Scratch(n, nullptr).bytes;
}

size_t norms_scratch_bytes(uint32_t n, uint32_t batch) { return Scratch(n, nullptr, batch).bytes; }

int launch_norms(const void* amps, uint32_t n, uint32_t batch, void* scratch, const double** norms, uint64_t* pitch,
                 void* stream, int precision) {
    if (batch < 1 || batch > 65535) return MB2_ERR_INVALID;
    const auto s = static_cast<cudaStream_t>(stream);
    const Scratch w(n, scratch, batch);
    if (precision == MB2_C64) launch_norms_t(static_cast<const float2*>(amps), n, batch, w, s);
    else launch_norms_t(static_cast<const double2*>(amps), n, batch, w, s);
    *norms = w.cstart + w.nchunks;
    *pitch = w.nchunks + 1;
    return launch_status();
}

int launch_exact_norm(const void* amps, uint32_t n, void* scratch, double* host_total, void* stream, int precision) {
    const auto s = static_cast<cudaStream_t>(stream);
    const double* norm = nullptr;
    uint64_t pitch = 0;
    if (int rc = launch_norms(amps, n, 1, scratch, &norm, &pitch, stream, precision); rc != MB2_OK) return rc;
    if (cudaMemcpyAsync(host_total, norm, sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return record_cuda_error(static_cast<int>(cudaGetLastError()));
    return MB2_OK;
}

int launch_sample(const void* amps, uint32_t n, double* dev_u, uint64_t shots, const uint64_t* draw,
                  void* sort_scratch, void* scratch, uint64_t* dev_basis, void* stream, int precision) {
    const auto s = static_cast<cudaStream_t>(stream);
    return precision == MB2_C64
               ? launch_sample_t<float2>(amps, n, dev_u, shots, draw, sort_scratch, scratch, dev_basis, s)
               : launch_sample_t<double2>(amps, n, dev_u, shots, draw, sort_scratch, scratch, dev_basis, s);
}

}  // namespace mb2
