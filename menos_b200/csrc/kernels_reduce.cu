// Pauli-string expectation and norm reductions (FP64), fixed-order.
//
// <psi|P|psi> = i^popcount(x&z) * sum_m conj(psi[m]) psi[m^x] (-1)^popcount(z & (m^x))
// (src/kernels/cpu/dense_kernels.cpp:544-569).  The pair (m, m^x) is visited
// once, from the member whose bit h (the highest bit of x) is clear:
//     t = conj(a_m) a_m'                 (m' = m ^ x)
//     contribution = t s(m') + conj(t) s(m)
// so each amplitude is read once per term.  Partial sums land in a fixed
// number of blocks and are added in block order by one thread per term, so
// the value does not depend on the GPU's SM count or on what else runs.
// Like the reference's CUDA reduction (dense_kernels.h:237-246) it is not
// bitwise the CPU's sequential sum; the parity tests bound the difference.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "mb2_internal.h"
#include "walk.cuh"

namespace mb2 {
namespace {

__device__ __forceinline__ uint64_t insert_zero(uint64_t i, uint32_t pos) {
    const uint64_t low = (uint64_t{1} << pos) - 1;
    return ((i & ~low) << 1) | (i & low);
}

constexpr int kThreads = 256;

__device__ __forceinline__ void block_reduce2(double& re, double& im) {
    __shared__ double sre[kThreads / 32], sim[kThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        sre[w] = re;
        sim[w] = im;
    }
    __syncthreads();
    if (w == 0) {
        re = l < kThreads / 32 ? sre[l] : 0.0;
        im = l < kThreads / 32 ? sim[l] : 0.0;
        for (int o = 4; o > 0; o >>= 1) {
            re += __shfl_down_sync(0xffffffffu, re, o);
            im += __shfl_down_sync(0xffffffffu, im, o);
        }
    }
}

__device__ __forceinline__ double2 as_d2(double2 a) { return a; }
__device__ __forceinline__ double2 as_d2(float2 a) { return make_double2(a.x, a.y); }

// A: double2 (complex128 state) or float2 (complex64 state, promoted to FP64).
template <typename A>
__global__ void __launch_bounds__(kThreads)
    k_expectation(const A* __restrict__ st, uint32_t n, const uint64_t* __restrict__ xs,
                  const uint64_t* __restrict__ zs, double* __restrict__ partials) {
    const uint32_t term = blockIdx.y;
    const uint64_t x = xs[term], z = zs[term];
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    double re = 0.0, im = 0.0;
    if (x == 0) {
        const uint64_t na = uint64_t{1} << n;
        for (uint64_t m = first; m < na; m += stride) {
            const double2 a = as_d2(st[m]);
            const double p = __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
            re = (__popcll(z & m) & 1) ? __dsub_rn(re, p) : __dadd_rn(re, p);
        }
    } else {
        const uint32_t h = 63 - __clzll(static_cast<long long>(x));
        const uint64_t np = (uint64_t{1} << n) >> 1;
        for (uint64_t c = first; c < np; c += stride) {
            const uint64_t m = insert_zero(c, h);
            const uint64_t m2 = m ^ x;
            const double2 a = as_d2(st[m]), b = as_d2(st[m2]);
            // t = conj(a) * b
            const double tr = __dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y));
            const double ti = __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x));
            const bool neg2 = __popcll(z & m2) & 1;  // sign of the (m, m') term
            const bool neg1 = __popcll(z & m) & 1;   // sign of the (m', m) term, conj(t)
            re = neg2 ? __dsub_rn(re, tr) : __dadd_rn(re, tr);
            im = neg2 ? __dsub_rn(im, ti) : __dadd_rn(im, ti);
            re = neg1 ? __dsub_rn(re, tr) : __dadd_rn(re, tr);
            im = neg1 ? __dadd_rn(im, ti) : __dsub_rn(im, ti);
        }
    }
    block_reduce2(re, im);
    if (threadIdx.x == 0) {
        double* p = partials + 2 * (static_cast<uint64_t>(term) * gridDim.x + blockIdx.x);
        p[0] = re;
        p[1] = im;
    }
}

// One CTA per term: the partials in block order, then i^popcount(x&z).  The
// order is part of the result, so one thread adds each part; what bounded a
// thread per term was a load from global memory before every add (512 blocks:
// 56-70 us whatever the state's size).  Here the CTA stages kFinishStage
// blocks' partials in shared memory in parallel, and threads 0 (real) and 1
// (imaginary) add from there at the latency of an FP64 add: 64 terms 70 -> 6 us.
constexpr uint32_t kFinishThreads = 256;
constexpr uint32_t kFinishStage = 512;
__global__ void __launch_bounds__(kFinishThreads)
    k_expectation_finish(const double* __restrict__ partials, uint32_t blocks, const uint64_t* __restrict__ xs,
                         const uint64_t* __restrict__ zs, double* __restrict__ out) {
    __shared__ double part[2][kFinishStage];
    const uint32_t t = blockIdx.x;
    const double2* p = reinterpret_cast<const double2*>(partials) + static_cast<uint64_t>(t) * blocks;
    double sum = 0.0;  // threads 0 and 1: the real and the imaginary part
    for (uint32_t b0 = 0; b0 < blocks; b0 += kFinishStage) {
        const uint32_t len = blocks - b0 < kFinishStage ? blocks - b0 : kFinishStage;
        for (uint32_t b = threadIdx.x; b < len; b += kFinishThreads) {
            const double2 v = p[b0 + b];
            part[0][b] = v.x;
            part[1][b] = v.y;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            const double* q = part[threadIdx.x];
#pragma unroll 16
            for (uint32_t b = 0; b < len; ++b) sum = __dadd_rn(sum, q[b]);
        }
        __syncthreads();
    }
    const double im = __shfl_sync(0xffffffffu, sum, 1);
    if (threadIdx.x != 0) return;
    const double re = sum;
    const int ph = __popcll(xs[t] & zs[t]) & 3;
    double orr = re, oi = im;
    if (ph == 1) {
        orr = -im;
        oi = re;
    } else if (ph == 2) {
        orr = -re;
        oi = -im;
    } else if (ph == 3) {
        orr = im;
        oi = -re;
    }
    out[2 * t] = orr;
    out[2 * t + 1] = oi;
}

// ---- grouped terms: one state read per group --------------------------------
// A group's terms have X masks whose bits above c lie in a subspace V of
// dimension d.  A tile is a coset of V: 2^d chunks of 2^c contiguous
// amplitudes (chunk k's high bits are rep ^ span[k]), so for every term the
// partner m ^ x of each amplitude m is in the same tile, at tile index
// L ^ dl with dl = (kx << c) | xl.
//
// With s(m) = (-1)^popcount(z & m) and s(m ^ x) = s(m) (-1)^popcount(z & x),
// the pair's share t s(m') + conj(t) s(m), t = conj(a_m) a_m', is
// 2 s(m) Re t when popcount(z & x) is even and -2i s(m) Im t when it is odd,
// so one real accumulator per term suffices; seen from the other member the
// same pair gives the same s(m) Re t (or s(m) Im t), so a pair may equally be
// visited once with weight 2 or from both members with weight 1.
//
// Thread r of the CTA owns tile amplitudes L = r | i << 9 (i < 2^(c+d-9),
// two or four), read into registers once per tile; per term it visits its
// own amplitudes and reads only the partners from shared memory.  When dl
// has a bit b >= 9 (the plan's coordinates give most terms the highest bit of
// the tile index) the visiting member is the one with bit b clear (half of
// every thread's amplitudes, weight 2); otherwise every member visits
// (weight 1).  s(m) is linear over XOR in the tile index apart from the
// coset representative: s = parity(z_hi & rep) ^ sigma(r) ^ sigma(i << 9),
// with sigma(L) = parity(z_lo & L) ^ parity(z_hi & span[L >> c]); the
// thread's sigma(r) of every term is a register bit mask, sigma(i << 9) a
// per-term byte.  Each term runs a body compiled for its (own count,
// visiting bit, mode): its products are independent and summed as a
// balanced tree before one add into the thread's sum of the term.
// Partial sums go to fixed slots (term, CTA) and are added in CTA order by
// the finish kernel.
using GroupTerm = PauliGroupTerm;
constexpr uint32_t kChunkWords = (1u << kPauliMaxSpan) / 32;
constexpr uint32_t kOwnShift = 9;  // log2(kGroupThreads): tile bits of the thread index
constexpr int kGroupThreads = 1 << kOwnShift;
constexpr uint32_t kMaxOwn = 1u << (kPauliTileQubits - kOwnShift);
static_assert(kPauliMinTileQubits >= kOwnShift + 1, "every thread owns at least two amplitudes");

// cp.async of one amplitude (16 or 8 bytes), global -> shared.
__device__ __forceinline__ void cp_async_amp(double2* smem, const double2* gmem) {
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_amp(float2* smem, const float2* gmem) {
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// Per-group tables in shared memory: the span, the parity of z_hi & span[k]
// per chunk k, per term its partner offset, body, sigma(i << 9) bits and
// high z bits.
struct GroupShared {
    uint64_t sspan[1u << kPauliMaxSpan];
    uint64_t off[kMaxOwn];  // state index of own amplitude i, XOR that of own amplitude 0
    uint32_t cpar[kMaxGroupTerms][kChunkWords];  // parity of z_hi & span[k], bit k
    uint32_t tdl[kMaxGroupTerms], tzl[kMaxGroupTerms], tmode[kMaxGroupTerms];
    uint32_t tcode[kMaxGroupTerms];  // the term's body (term_body)
    // The terms in the order they are reduced (the places): regular pairs, Z
    // strings with a sum in a register, other Z strings, other pairs (below).
    // Per place the term, what its body needs in one word -- dl, its code from
    // bit 16 (a regular pair: its mode), and from bit 24 sigma(i << kOwnShift)
    // per own amplitude i; one more to read ahead -- and its high z bits.
    uint32_t place[kMaxGroupTerms], regular, held, zs;  // the first three kinds end there
    uint32_t tword[kMaxGroupTerms + 1];
    uint64_t pzh[32];  // zero past the terms
    uint32_t tweight[kMaxGroupTerms];  // 2: each pair visited once; 1: from both members
    uint64_t tzh[kMaxGroupTerms];
    double red[kGroupThreads / 32];
};
// Sums in registers while the tiles are read: up to kPauliHeldTerms terms,
// first the regular pairs -- those whose members differ in the tile index's
// highest bit, in tiles of four own amplitudes: nearly all, by the plan's
// choice of coordinates -- then Z strings (pauli_can_hold).  The other terms'
// sums, one per thread or one per pair of neighbouring threads (paired, 0 or
// 1), follow the tile buffers in dynamic shared memory: that of the term at
// place p at acc[((p - held) * kGroupThreads + thread) >> paired].

// sigma(L): the sign parity of tile index L without the coset's part.
__device__ __forceinline__ uint32_t group_sigma(const GroupShared& g, uint32_t t, uint32_t L, uint32_t c) {
    const uint32_t k = L >> c;
    return ((g.cpar[t][k >> 5] >> (k & 31u)) ^ static_cast<uint32_t>(__popc(g.tzl[t] & L))) & 1u;
}

// Term bodies: (own amplitudes, selector bit, mode).  Code = base of the
// own count (0 for two, 4 for four) + 2 * (selector bit + 1) + (mode - 1),
// the selector bit -1 meaning every member visits; Z strings have none.
__host__ __device__ constexpr uint32_t body_code(uint32_t own, int selb, uint32_t mode) {
    return (own == 4 ? 4u : 0u) + 2u * static_cast<uint32_t>(selb + 1) + (mode - 1);
}

// Fills the tables and clears the accumulators; returns this thread's
// sigma(r) of every term (bit p: the term at place p).
__device__ __forceinline__ uint32_t group_setup(GroupShared& g, double* acc, uint32_t held, uint32_t paired, uint32_t c, uint32_t d,
                                                const uint64_t* __restrict__ span,
                                                const GroupTerm* __restrict__ terms, uint32_t nterms) {
    const uint32_t nchunks = 1u << d;
    const uint32_t own = 1u << (c + d - kOwnShift);
    for (uint32_t i = threadIdx.x; i < nchunks; i += kGroupThreads) g.sspan[i] = span[i];
    if (threadIdx.x < 32) g.pzh[threadIdx.x] = 0;
    __syncthreads();
    if (threadIdx.x < own) {
        const uint32_t L = threadIdx.x << kOwnShift;
        g.off[threadIdx.x] = (g.sspan[L >> c] << c) | (L & ((1u << c) - 1));
    }
    for (uint32_t t = threadIdx.x; t < nterms; t += kGroupThreads) {
        const GroupTerm T = terms[t];
        const uint32_t dl = (T.kx << c) | T.xl;
        g.tdl[t] = dl;
        g.tzl[t] = static_cast<uint32_t>(T.z & ((uint64_t{1} << c) - 1));
        g.tzh[t] = T.z >> c;
        // 0: a Z string (x = 0); 1: real pair sum; 2: imaginary pair sum
        const uint32_t mode = T.x == 0 ? 0u : ((__popcll(T.x & T.z) & 1) ? 2u : 1u);
        g.tmode[t] = mode;
        // The visiting member of a pair: the one whose highest bit of dl
        // among the register index bits is clear; none there: both visit.
        const uint32_t hi = dl >> kOwnShift;
        const int selb = hi == 0 ? -1 : 31 - __clz(hi);
        g.tcode[t] = mode == 0 ? 0u : body_code(own, selb, mode);
        g.tweight[t] = (mode != 0 && selb >= 0) ? 2u : 1u;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kMaxGroupTerms * kChunkWords; i += kGroupThreads) {
        const uint32_t t = i / kChunkWords, w = i % kChunkWords;
        uint32_t bits = 0;
        if (t < nterms)
            for (uint32_t b = 0; b < 32 && w * 32 + b < nchunks; ++b)
                bits |= static_cast<uint32_t>(__popcll(g.tzh[t] & g.sspan[w * 32 + b]) & 1) << b;
        g.cpar[t][w] = bits;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        // The places, by one warp: a lane a term (kMaxGroupTerms <= 32).
        const uint32_t t = threadIdx.x, below = (1u << t) - 1u;
        const bool term = t < nterms, z = term && g.tmode[t] == 0;
        const bool pair = term && !z && pauli_can_hold(false, g.tdl[t], c + d);
        const uint32_t pairs = __ballot_sync(0xffffffffu, pair), zs = __ballot_sync(0xffffffffu, z);
        const uint32_t first = __popc(pairs) < static_cast<int>(kPauliHeldTerms) ? __popc(pairs) : kPauliHeldTerms;
        const bool regular = pair && __popc(pairs & below) < static_cast<int>(kPauliHeldTerms);
        // (Regular pairs past the registers' go with the others.)
        const uint32_t others = __ballot_sync(0xffffffffu, term && !z && !regular);
        if (term)
            g.place[regular ? __popc(pairs & below)
                    : z     ? first + __popc(zs & below)
                            : first + __popc(zs) + __popc(others & below)] = t;
        if (t == 0) {
            g.regular = first;
            g.zs = first + __popc(zs);
            g.held = held;
            g.tword[nterms] = 0;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < ((nterms - held) * kGroupThreads) >> paired; i += kGroupThreads) acc[i] = 0.0;
    for (uint32_t p = threadIdx.x; p < nterms; p += kGroupThreads) {
        const uint32_t t = g.place[p];
        uint32_t bits = 0;
        for (uint32_t i = 0; i < own; ++i) bits |= group_sigma(g, t, i << kOwnShift, c) << i;
        g.tword[p] = g.tdl[t] | ((p < g.regular ? g.tmode[t] : g.tcode[t]) << 16) | (bits << 24);
        g.pzh[p] = g.tzh[t];
    }
    uint32_t sig = 0;
    for (uint32_t p = 0; p < nterms; ++p) sig |= group_sigma(g, g.place[p], threadIdx.x, c) << p;
    __syncthreads();
    return sig;
}

// v with its sign flipped when f is 1 (an integer XOR: exact).
__device__ __forceinline__ double flip_if(double v, uint32_t f) {
    return __hiloint2double(__double2hiint(v) ^ static_cast<int>(f << 31), __double2loint(v));
}

// One term's share of this thread's own amplitudes in one tile, as a
// balanced sum in a fixed order, the second product of each pair added
// without a rounding of its own (FMA): OWN own amplitudes, SELB the register bit
// that marks the non-visiting member (-1: all visit), MODE 1 (Re conj(a) b)
// or 2 (Im conj(a) b); sg bit i: the sign of own amplitude i.  Every branch
// is resolved at compile time.
template <int OWN, int SELB, int MODE, typename A>
__device__ __forceinline__ double term_body(const double2 (&a)[kMaxOwn], const A* __restrict__ cur, uint32_t r,
                                            uint32_t dl, uint32_t sg) {
    constexpr int NV = SELB < 0 ? OWN : OWN / 2;
    constexpr int SB = SELB < 0 ? 0 : SELB;
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        // The k-th visiting own amplitude: k with a zero inserted at SELB.
        const int i = SELB < 0 ? k : (((k >> SB) << (SB + 1)) | (k & ((1 << SB) - 1)));
        const double2 b = as_d2(cur[(r | (static_cast<uint32_t>(i) << kOwnShift)) ^ dl]);
        const double x = MODE == 1 ? __fma_rn(a[i].x, b.x, __dmul_rn(a[i].y, b.y))
                                   : __fma_rn(a[i].x, b.y, -__dmul_rn(a[i].y, b.x));
        v[k] = flip_if(x, (sg >> i) & 1u);
    }
#pragma unroll
    for (int w = 1; w < NV; w <<= 1)
#pragma unroll
        for (int j = 0; j + w < NV; j += 2 * w) v[j] = __dadd_rn(v[j], v[j + w]);
    return v[0];
}

// Adds one gathered coset tile (representative rep) to every term's
// accumulator.  sig: this thread's sigma(r) bits (group_setup).
//
// Bound by shared memory and issue slots: a term is its partner loads, a
// handful of FP64 operations, and what steers them.  So the cosets' signs of
// all terms come from one ballot per tile, a term's tables are one word, 512
// threads own four amplitudes each (two CTAs, 32 warps, per SM hide what 16
// did not), and a regular pair is two partner loads and eight FP64 operations
// without a branch: the mode picks the parts that multiply the partner's by
// selects, the signs ride on them, the sum stays in a register.
// A Z string's signs over a thread's four amplitudes are linear in the two
// index bits, so its sum is, up to one sign, one of four that all of them
// share: one add a term.
// Only the sums that no register holds take shared memory (4 KiB each): with
// all of a 16-term group's there, one CTA fitted an SM.
// 27 qubits, with 256 threads, eight own amplitudes, a branch and a
// shared-memory sum per term; with 512 threads, regular pairs in registers and
// every term's sum in shared memory; now: 64 random strings 7.06, 5.50,
// 5.39 ms; 60 Z strings of a chain 4.13, 5.07, 2.46; 16 strings on the low
// eight qubits, all irregular, 2.04, 2.28, 1.93.  2 random strings at 28
// qubits, bound by the read: 0.89, 0.96, 0.90 (a third buffer in flight and
// one barrier a tile; three instructions to an address instead of a dozen).
template <typename A>
__device__ __forceinline__ void group_tile(GroupShared& g, double (&reg)[kPauliHeldTerms], double* __restrict__ acc,
                                           const A* __restrict__ cur, uint64_t rep,
                                           uint32_t tile_amps, uint32_t nterms, uint32_t paired, uint32_t sig) {
    const uint32_t r = threadIdx.x;
    const uint32_t own = tile_amps >> kOwnShift;
    double2 a[kMaxOwn];
#pragma unroll
    for (uint32_t i = 0; i < kMaxOwn; ++i)
        a[i] = i < own ? as_d2(cur[r | (i << kOwnShift)]) : make_double2(0.0, 0.0);
    // Bit p: the sign of the term at place p at this thread's first amplitude.
    const uint32_t signs = sig ^ __ballot_sync(0xffffffffu, __popcll(g.pzh[r & 31u] & rep) & 1);
    const uint32_t regular = g.regular, held = g.held, zs = g.zs;
#pragma unroll
    for (uint32_t p = 0; p < kPauliHeldTerms; ++p) {
        if (p >= regular) break;  // (uniform over the CTA)
        const uint32_t word = g.tword[p], s0 = signs >> p;
        const bool imag = (word >> 17) & 1u;  // mode 2
        const uint32_t at = r ^ (word & 0xffffu);
        double v[2];
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {  // the own amplitudes whose highest bit is clear
            const double2 b = as_d2(cur[at ^ (i << kOwnShift)]);
            const uint32_t flip = s0 ^ (word >> (24 + i));
            // Re: a.x b.x + a.y b.y; Im: -a.y b.x + a.x b.y.
            const double px = flip_if(imag ? a[i].y : a[i].x, (flip ^ (imag ? 1u : 0u)) & 1u);
            const double py = flip_if(imag ? a[i].x : a[i].y, flip & 1u);
            v[i] = __fma_rn(px, b.x, __dmul_rn(py, b.y));
        }
        reg[p] = __dadd_rn(reg[p], __dadd_rn(v[0], v[1]));
    }
    // A term's sum in shared memory; paired: the two threads' shares first.
    auto add = [&](uint32_t p, double v) {
        if (paired) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
        double& sum = acc[((p - held) * kGroupThreads + r) >> paired];
        if ((r & paired) == 0) sum = __dadd_rn(sum, v);
    };
    uint32_t next = g.tword[zs];
    for (uint32_t p = zs; p < nterms; ++p) {
        const uint32_t word = next;
        next = g.tword[p + 1];
        // Bit i: the sign of own amplitude i.
        const uint32_t sg = (word >> 24) ^ (0u - ((signs >> p) & 1u));
        const uint32_t dl = word & 0xffffu;
        double v = 0.0;
        switch ((word >> 16) & 0xffu) {
            case body_code(2, -1, 1): v = term_body<2, -1, 1>(a, cur, r, dl, sg); break;
            case body_code(2, -1, 2): v = term_body<2, -1, 2>(a, cur, r, dl, sg); break;
            case body_code(2, 0, 1): v = term_body<2, 0, 1>(a, cur, r, dl, sg); break;
            case body_code(2, 0, 2): v = term_body<2, 0, 2>(a, cur, r, dl, sg); break;
            case body_code(4, -1, 1): v = term_body<4, -1, 1>(a, cur, r, dl, sg); break;
            case body_code(4, -1, 2): v = term_body<4, -1, 2>(a, cur, r, dl, sg); break;
            case body_code(4, 0, 1): v = term_body<4, 0, 1>(a, cur, r, dl, sg); break;
            case body_code(4, 0, 2): v = term_body<4, 0, 2>(a, cur, r, dl, sg); break;
            case body_code(4, 1, 1): v = term_body<4, 1, 1>(a, cur, r, dl, sg); break;
            case body_code(4, 1, 2): v = term_body<4, 1, 2>(a, cur, r, dl, sg); break;
            default: break;
        }
        add(p, v);
    }
    if (regular == zs) return;
    // |a|^2 of the own amplitudes, and their four sums: bit 0 of the number is
    // the sign of amplitude 1, bit 1 that of amplitude 2, amplitude 3's follows.
    double q[kMaxOwn];
#pragma unroll
    for (uint32_t i = 0; i < kMaxOwn; ++i) q[i] = __fma_rn(a[i].x, a[i].x, __dmul_rn(a[i].y, a[i].y));
    const double e0 = __dadd_rn(q[0], q[1]), e1 = __dadd_rn(q[2], q[3]), o0 = __dsub_rn(q[0], q[1]),
                 o1 = __dsub_rn(q[2], q[3]);
    const double s00 = __dadd_rn(e0, e1), s01 = __dadd_rn(o0, o1), s10 = __dsub_rn(e0, e1), s11 = __dsub_rn(o0, o1);
    auto z_sum = [&](uint32_t p) {
        const uint32_t word = g.tword[p];
        const double even = (word >> 26) & 1u ? s10 : s00, odd = (word >> 26) & 1u ? s11 : s01;
        return flip_if((word >> 25) & 1u ? odd : even, (signs >> p) & 1u);
    };
#pragma unroll
    for (uint32_t p = 0; p < kPauliHeldTerms; ++p) {
        if (p >= held) break;  // (uniform over the CTA, as the next)
        if (p >= regular) reg[p] = __dadd_rn(reg[p], z_sum(p));
    }
    for (uint32_t p = held; p < zs; ++p) add(p, z_sum(p));
}

// Per term: this CTA's sum in a fixed order (lanes, then warps), written to
// slot_of(t) as (re, im) of the pair sum before the i^popcount(x & z)
// factor, with the term's visit weight; the accumulators are cleared.
template <typename SLOT>
__device__ __forceinline__ void group_write(GroupShared& g, double (&reg)[kPauliHeldTerms], double* __restrict__ acc,
                                            const GroupTerm* __restrict__ terms, uint32_t nterms, uint32_t paired,
                                            SLOT slot_of) {
    const uint32_t held = g.held;
    for (uint32_t p = 0; p < nterms; ++p) {
        const uint32_t t = g.place[p];
        double r = 0.0;
        if (p < held) {
#pragma unroll
            for (uint32_t i = 0; i < kPauliHeldTerms; ++i) r = i == p ? reg[i] : r;
        } else if ((threadIdx.x & paired) == 0) {
            double& sum = acc[((p - held) * kGroupThreads + threadIdx.x) >> paired];
            r = sum;
            sum = 0.0;
        }
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) g.red[threadIdx.x >> 5] = r;
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = 0.0;
            for (int w = 0; w < kGroupThreads / 32; ++w) sum += g.red[w];
            double* out = slot_of(terms[t].out);
            const uint32_t mode = g.tmode[t];
            const double w = static_cast<double>(g.tweight[t]);
            out[0] = mode == 0 ? sum : mode == 1 ? w * sum : 0.0;
            out[1] = mode == 2 ? -w * sum : 0.0;
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < kPauliHeldTerms; ++i) reg[i] = 0.0;
}

// Coset representative: the coset number deposited on the free (non-pivot)
// high bits.
__device__ __forceinline__ uint64_t deposit_bits(uint64_t v, uint64_t mask) {
    uint64_t r = 0;
    while (mask != 0) {
        const uint64_t low = mask & (~mask + 1);
        if (v & 1) r |= low;
        v >>= 1;
        mask ^= low;
    }
    return r;
}

// This thread's first amplitude in the coset of representative 0.  The span
// is linear over XOR in the chunk's number, so its others, and those of other
// cosets, are an XOR away.
__device__ __forceinline__ uint64_t group_base(const GroupShared& g, uint32_t c) {
    return (g.sspan[threadIdx.x >> c] << c) | (threadIdx.x & ((1u << c) - 1));
}

template <typename A>
__device__ __forceinline__ void group_gather(const A* __restrict__ st, uint64_t rep, A* buf, const GroupShared& g,
                                             uint64_t base, uint32_t c, uint32_t tile_amps) {
    const uint64_t first = base ^ (rep << c);
#pragma unroll
    for (uint32_t i = 0; i < kMaxOwn; ++i)
        if ((i << kOwnShift) < tile_amps) cp_async_amp(buf + (threadIdx.x | (i << kOwnShift)), st + (first ^ g.off[i]));
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Cosets are processed with `stages` (two or three) shared-memory buffers: the
// amplitudes of the stages - 1 cosets ahead are gathered with cp.async while
// this one is reduced.
template <typename A>
__global__ void __launch_bounds__(kGroupThreads, 2)
    k_pauli_group(const A* __restrict__ st, uint32_t c, uint32_t d, const uint64_t* __restrict__ span,
                  uint64_t free_mask, const GroupTerm* __restrict__ terms, uint32_t nterms, uint32_t held, uint32_t paired, uint32_t stages, uint64_t ncosets,
                  uint32_t pitch, double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ GroupShared g;
    const uint32_t tile_amps = 1u << (c + d);
    A* const tiles = reinterpret_cast<A*>(gsm);
    double* acc = reinterpret_cast<double*>(tiles + stages * tile_amps);
    const uint32_t sig = group_setup(g, acc, held, paired, c, d, span, terms, nterms);
    const uint64_t base = group_base(g, c);
    double reg[kPauliHeldTerms] = {};
    // Moving gridDim.x cosets on is a masked add on the free bits.
    const uint64_t rstep = deposit_bits(gridDim.x, free_mask);
    auto advance = [&](uint64_t r) { return ((r | ~free_mask) + rstep) & free_mask; };
    uint64_t rep = deposit_bits(blockIdx.x, free_mask), ahead = rep;  // of the tile reduced, of the one gathered
    uint64_t at = blockIdx.x;                                         // the latter's number
    uint32_t fill = 0, cur = 0;                                       // their buffers
    auto gather = [&]() {  // (an empty group past the end keeps the count)
        if (at < ncosets) group_gather(st, ahead, tiles + fill * tile_amps, g, base, c, tile_amps);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        ahead = advance(ahead);
        at += gridDim.x;
        fill = fill + 1 == stages ? 0 : fill + 1;
    };
    for (uint32_t i = 0; i + 1 < stages; ++i) gather();
    for (uint64_t cs = blockIdx.x; cs < ncosets; cs += gridDim.x) {
        // The buffer that is filled now was reduced from in the round before: with
        // three, every thread is past that at this round's barrier.
        if (stages == 2) gather();
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        if (stages == 3) gather();
        group_tile(g, reg, acc, tiles + cur * tile_amps, rep, tile_amps, nterms, paired, sig);
        if (stages == 2) __syncthreads();
        rep = advance(rep);
        cur = cur + 1 == stages ? 0 : cur + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    group_write(g, reg, acc, terms, nterms, paired, [&](uint32_t out) {
        return partials + 2 * (static_cast<uint64_t>(out) * pitch + blockIdx.x);
    });
}

// The same grouped reduction over a batch of states (binding b's 2^n
// amplitudes at b * 2^n).  `per` CTAs share a binding: CTA slot s takes the
// binding's cosets s, s + per, ...; bindings are taken gridDim.x / per
// apart.  Partial (term, binding, slot) lands at
// partials[2 * ((term * bindings + b) * per + s)], so a binding's value
// depends only on its own state and on `per`.
template <typename A>
__global__ void __launch_bounds__(kGroupThreads, 2)
    k_pauli_group_batch(const A* __restrict__ st, uint32_t n, uint32_t c, uint32_t d,
                        const uint64_t* __restrict__ span, uint64_t free_mask, const GroupTerm* __restrict__ terms,
                        uint32_t nterms, uint32_t held, uint32_t paired, uint64_t bindings, uint32_t per,
                        double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ GroupShared g;
    const uint32_t tile_amps = 1u << (c + d);
    A* buf0 = reinterpret_cast<A*>(gsm);
    A* buf1 = buf0 + tile_amps;
    double* acc = reinterpret_cast<double*>(buf1 + tile_amps);
    const uint32_t sig = group_setup(g, acc, held, paired, c, d, span, terms, nterms);
    double reg[kPauliHeldTerms] = {};
    const uint64_t ncosets = uint64_t{1} << (n - c - d);
    const uint32_t slot = blockIdx.x % per;
    const uint64_t b0 = blockIdx.x / per, bstep = gridDim.x / per;
    if (b0 >= bindings) return;  // (uniform over the CTA)
    // This CTA's cosets in each binding, and its work items in order:
    // item f = (binding b0 + (f / mine) * bstep, coset slot + (f % mine) * per).
    const uint64_t mine = ncosets > slot ? (ncosets - slot + per - 1) / per : 0;
    const uint64_t nb = (bindings - b0 + bstep - 1) / bstep;
    auto write = [&](uint64_t b) {
        group_write(g, reg, acc, terms, nterms, paired, [&](uint32_t out) {
            return partials + 2 * ((static_cast<uint64_t>(out) * bindings + b) * per + slot);
        });
    };
    if (mine == 0) {  // more slots than cosets: this slot's partials are zero
        for (uint64_t i = 0; i < nb; ++i) write(b0 + i * bstep);
        return;
    }
    const uint64_t items = nb * mine;
    auto item = [&](uint64_t f, uint64_t& b, uint64_t& rep) {
        b = b0 + (f / mine) * bstep;
        rep = deposit_bits(slot + (f % mine) * per, free_mask);
    };
    uint64_t b = 0, rep = 0;
    item(0, b, rep);
    const uint64_t base = group_base(g, c);
    group_gather(st + (b << n), rep, buf0, g, base, c, tile_amps);
    A* cur = buf0;
    A* nxt = buf1;
    for (uint64_t f = 0; f < items; ++f) {
        uint64_t bn = 0, repn = 0;
        if (f + 1 < items) {
            item(f + 1, bn, repn);
            group_gather(st + (bn << n), repn, nxt, g, base, c, tile_amps);
        } else {
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        group_tile(g, reg, acc, cur, rep, tile_amps, nterms, paired, sig);
        __syncthreads();  // this buffer is the target of the gather after next
        if ((f + 1) % mine == 0) write(b);
        b = bn;
        rep = repn;
        A* tmp = cur;
        cur = nxt;
        nxt = tmp;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// <H> per binding: sum over terms in term order of coef * Re(i^popcount(x&z)
// * (sum over the binding's slots, in slot order, of the partials)).
__global__ void k_batch_group_finish(const double* __restrict__ partials, uint64_t bindings, uint32_t per,
                                     const uint64_t* __restrict__ xs, const uint64_t* __restrict__ zs,
                                     const double* __restrict__ coefs, uint32_t num_terms, double* __restrict__ out) {
    for (uint64_t b = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; b < bindings;
         b += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        double total = 0.0;
        for (uint32_t t = 0; t < num_terms; ++t) {
            const double* p = partials + 2 * ((static_cast<uint64_t>(t) * bindings + b) * per);
            double re = 0.0, im = 0.0;
            for (uint32_t s = 0; s < per; ++s) {
                re += p[2 * s];
                im += p[2 * s + 1];
            }
            const int ph = __popcll(xs[t] & zs[t]) & 3;
            total += coefs[t] * (ph == 0 ? re : ph == 1 ? -im : ph == 2 ? -re : im);
        }
        out[b] = total;
    }
}

}  // namespace

// The shared memory of a group that lets two CTAs share an SM: of its tile
// buffers, and of the sums that no register holds.  Three buffers where they
// leave room for that (at most `most`); where one sum for each thread does
// not, one for each pair of threads (paired).
struct GroupMemory {
    uint32_t stages, paired;
    size_t bytes;
    GroupMemory(uint32_t most, uint32_t tile_qubits, uint32_t nterms, uint32_t held, int precision) {
        const size_t tile = (size_t{1} << tile_qubits) * (precision == MB2_C64 ? sizeof(float2) : sizeof(double2));
        const size_t sums = size_t{nterms - held} * kGroupThreads * sizeof(double);
        auto two_fit = [](size_t dynamic) { return 2 * (dynamic + sizeof(GroupShared) + 1024) <= kSmemPerSm; };
        stages = most == 3 && two_fit(3 * tile + sums) ? 3 : 2;
        paired = two_fit(stages * tile + sums) ? 0 : 1;
        bytes = stages * tile + (sums >> paired);
    }
};

int launch_pauli_group(const void* amps, uint32_t n, uint32_t c, uint32_t d, const uint64_t* dev_span,
                       uint64_t free_mask, const void* dev_terms, uint32_t nterms, uint32_t held, double* dev_partials,
                       uint32_t grid, uint32_t pitch, void* stream, int precision) {
    if (nterms == 0) return MB2_OK;
    if (nterms > kMaxGroupTerms || held > nterms || c + d > kPauliTileQubits || d > kPauliMaxSpan) return MB2_ERR_INVALID;
    const auto s = static_cast<cudaStream_t>(stream);
    const uint64_t ncosets = uint64_t{1} << (n - c - d);
    // Two buffers of 2^(c+d) amplitudes, of which each thread owns two or four.
    if (c + d < kPauliMinTileQubits || grid > pitch) return MB2_ERR_INVALID;
    const GroupMemory mem(3, c + d, nterms, held, precision);
    static const bool attr = [] {  // once, thread-safe (concurrent callers wait for it)
        return cudaFuncSetAttribute(k_pauli_group<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    128 * 1024) == cudaSuccess &&
               cudaFuncSetAttribute(k_pauli_group<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    128 * 1024) == cudaSuccess;
    }();
    if (!attr) return launch_status();
    const auto* terms = static_cast<const GroupTerm*>(dev_terms);
    if (precision == MB2_C64)
        k_pauli_group<float2><<<grid, kGroupThreads, mem.bytes, s>>>(static_cast<const float2*>(amps), c, d, dev_span,
                                                           free_mask, terms, nterms, held, mem.paired, mem.stages, ncosets, pitch, dev_partials);
    else
        k_pauli_group<double2><<<grid, kGroupThreads, mem.bytes, s>>>(static_cast<const double2*>(amps), c, d, dev_span,
                                                            free_mask, terms, nterms, held, mem.paired, mem.stages, ncosets, pitch, dev_partials);
    note_launches(1);
    return launch_status();
}

int launch_pauli_group_batch(const void* amps, uint32_t n, uint32_t c, uint32_t d, const uint64_t* dev_span,
                             uint64_t free_mask, const void* dev_terms, uint32_t nterms, uint32_t held, uint64_t bindings,
                             uint32_t per, double* dev_partials, int sm_count, void* stream, int precision) {
    if (nterms == 0) return MB2_OK;
    if (nterms > kMaxGroupTerms || held > nterms || c + d > kPauliTileQubits || d > kPauliMaxSpan || c + d > n || per == 0 ||
        c + d < kPauliMinTileQubits)
        return MB2_ERR_INVALID;
    const GroupMemory mem(2, c + d, nterms, held, precision);
    static const bool attr = [] {  // once, thread-safe
        return cudaFuncSetAttribute(k_pauli_group_batch<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    128 * 1024) == cudaSuccess &&
               cudaFuncSetAttribute(k_pauli_group_batch<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    128 * 1024) == cudaSuccess;
    }();
    if (!attr) return launch_status();
    // Two CTAs per SM, a multiple of `per`, no more binding lanes than bindings.
    uint64_t lanes = std::max<uint64_t>(1, (2ull * static_cast<uint64_t>(sm_count)) / per);
    lanes = std::min<uint64_t>(lanes, bindings);
    const unsigned grid = static_cast<unsigned>(lanes * per);
    const auto s = static_cast<cudaStream_t>(stream);
    const auto* terms = static_cast<const GroupTerm*>(dev_terms);
    if (precision == MB2_C64)
        k_pauli_group_batch<float2><<<grid, kGroupThreads, mem.bytes, s>>>(static_cast<const float2*>(amps), n, c, d, dev_span,
                                                                 free_mask, terms, nterms, held, mem.paired, bindings, per, dev_partials);
    else
        k_pauli_group_batch<double2><<<grid, kGroupThreads, mem.bytes, s>>>(static_cast<const double2*>(amps), n, c, d,
                                                                  dev_span, free_mask, terms, nterms, held, mem.paired, bindings, per,
                                                                  dev_partials);
    note_launches(1);
    return launch_status();
}

int launch_batch_group_finish(const double* dev_partials, uint64_t bindings, uint32_t per, const uint64_t* dev_x,
                              const uint64_t* dev_z, const double* dev_coefs, uint32_t num_terms, double* dev_out,
                              void* stream) {
    const uint64_t blocks = (bindings + 127) / 128;
    k_batch_group_finish<<<static_cast<unsigned>(blocks < 1024 ? blocks : 1024), 128, 0,
                           static_cast<cudaStream_t>(stream)>>>(dev_partials, bindings, per, dev_x, dev_z, dev_coefs,
                                                                num_terms, dev_out);
    note_launches(1);
    return launch_status();
}

// ---- density matrices ---------------------------------------------------
// rho as a 2n-qubit vector, entry (r, c) at r | c << n.  Tr(P rho) partials:
// the sum over c of (-1)^popcount(c & z) rho[c | (c ^ x) << n] (the
// reference's trace_with_pauli, src/engines/density_matrix/
// density_matrix_engine.cpp); k_expectation_finish adds the partials in
// block order and applies i^popcount(x & z).
__global__ void __launch_bounds__(kThreads)
    k_dm_trace(const double2* __restrict__ rho, uint32_t n, const uint64_t* __restrict__ xs,
               const uint64_t* __restrict__ zs, double* __restrict__ partials) {
    const uint32_t term = blockIdx.y;
    const uint64_t x = xs[term], z = zs[term];
    const uint64_t dim = uint64_t{1} << n;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    double re = 0.0, im = 0.0;
    for (uint64_t c = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < dim; c += stride) {
        const double2 e = rho[c | ((c ^ x) << n)];
        if (__popcll(c & z) & 1) {
            re = __dsub_rn(re, e.x);
            im = __dsub_rn(im, e.y);
        } else {
            re = __dadd_rn(re, e.x);
            im = __dadd_rn(im, e.y);
        }
    }
    block_reduce2(re, im);
    if (threadIdx.x == 0) {
        double* p = partials + 2 * (static_cast<uint64_t>(term) * gridDim.x + blockIdx.x);
        p[0] = re;
        p[1] = im;
    }
}

// The reference's sort-then-walk over rho's diagonal (probabilities
// Re rho[x | x << n]), for the density matrices this path holds (n <= 15):
// 4096 shots at 11 qubits 1451 -> 31 us against one thread loading each entry
// and each uniform from memory as it came to them.
__global__ void __launch_bounds__(kWalkThreads)
    k_dm_walk(const double2* __restrict__ rho, uint32_t n, const double* __restrict__ u, uint64_t shots,
              uint64_t* __restrict__ basis) {
    const uint64_t step = (uint64_t{1} << n) + 1;
    walk_cta(1u << n, [&](uint32_t b) { return rho[b * step].x; }, u, shots, basis);
}

int launch_expectation_finish(const double* dev_partials, uint32_t blocks, const uint64_t* dev_x,
                              const uint64_t* dev_z, uint32_t num_terms, double* dev_out, void* stream) {
    k_expectation_finish<<<num_terms, kFinishThreads, 0, static_cast<cudaStream_t>(stream)>>>(dev_partials, blocks,
                                                                                              dev_x, dev_z, dev_out);
    note_launches(1);
    return launch_status();
}

int launch_dm_trace(const void* rho, uint32_t n, const uint64_t* dev_x, const uint64_t* dev_z, uint32_t num_terms,
                    double* dev_partials, double* dev_out, void* stream) {
    if (num_terms == 0) return MB2_OK;
    const auto s = static_cast<cudaStream_t>(stream);
    k_dm_trace<<<dim3(kExpBlocks, num_terms), kThreads, 0, s>>>(static_cast<const double2*>(rho), n, dev_x, dev_z,
                                                               dev_partials);
    note_launches(1);
    if (int rc = launch_status(); rc != MB2_OK) return rc;
    return launch_expectation_finish(dev_partials, kExpBlocks, dev_x, dev_z, num_terms, dev_out, stream);
}

int launch_dm_walk(const void* rho, uint32_t n, const double* dev_uniforms_sorted, uint64_t shots,
                   uint64_t* dev_basis, void* stream) {
    k_dm_walk<<<1, kWalkThreads, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const double2*>(rho), n,
                                                                         dev_uniforms_sorted, shots, dev_basis);
    note_launches(1);
    return launch_status();
}

int launch_expectation_partials(const void* amps, uint32_t n, const uint64_t* dev_x, const uint64_t* dev_z,
                                uint32_t num_terms, double* dev_partials, void* stream, int precision) {
    if (num_terms == 0) return MB2_OK;
    const auto s = static_cast<cudaStream_t>(stream);
    const dim3 grid(kExpBlocks, num_terms);
    if (precision == MB2_C64)
        k_expectation<float2><<<grid, kThreads, 0, s>>>(static_cast<const float2*>(amps), n, dev_x, dev_z, dev_partials);
    else
        k_expectation<double2><<<grid, kThreads, 0, s>>>(static_cast<const double2*>(amps), n, dev_x, dev_z,
                                                         dev_partials);
    note_launches(1);
    return launch_status();
}

int launch_expectation(const void* amps, uint32_t n, const uint64_t* dev_x, const uint64_t* dev_z,
                       uint32_t num_terms, double* dev_partials, double* dev_out, void* stream, int precision) {
    if (num_terms == 0) return MB2_OK;
    const auto s = static_cast<cudaStream_t>(stream);
    const dim3 grid(kExpBlocks, num_terms);
    if (precision == MB2_C64)
        k_expectation<float2><<<grid, kThreads, 0, s>>>(static_cast<const float2*>(amps), n, dev_x, dev_z, dev_partials);
    else
        k_expectation<double2><<<grid, kThreads, 0, s>>>(static_cast<const double2*>(amps), n, dev_x, dev_z,
                                                         dev_partials);
    k_expectation_finish<<<num_terms, kFinishThreads, 0, s>>>(dev_partials, kExpBlocks, dev_x, dev_z, dev_out);
    note_launches(2);
    return launch_status();
}

}  // namespace mb2

// ---------------------------------------------------------------------------
// The expectation reduction for callers that cannot allocate device memory.
//
// Some callers of this library must not call cudaMalloc: a serving process
// whose own pool allocator has reserved the GPU's memory up front (a
// cudaMalloc from here would fail or fragment that pool), or code running
// where allocation is not allowed at all (a latency-critical loop that must
// not stall on the driver's allocator).  mb2_expectation_noalloc gives them
// the Pauli-expectation reduction with every byte of scratch it needs --
// the Pauli masks, the per-block partial sums and the finished terms -- in
// the file-scope array below, a fixed 526,336 bytes that every GPU which
// loads this library holds until the process exits.
// ---------------------------------------------------------------------------
namespace mb2 {
namespace {

constexpr uint32_t kNoAllocTerms = MB2_NOALLOC_MAX_TERMS;
constexpr size_t kNoAllocMasks = kNoAllocTerms * sizeof(uint64_t);                 // x, then z
constexpr size_t kNoAllocPartials = size_t{kNoAllocTerms} * kExpBlocks * 2 * sizeof(double);
constexpr size_t kNoAllocOut = kNoAllocTerms * 2 * sizeof(double);
constexpr size_t kNoAllocBytes = 2 * kNoAllocMasks + kNoAllocPartials + kNoAllocOut;
static_assert(kNoAllocBytes == 526336, "the documented size");

__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {};

// The device address of g_noalloc_scratch on the current device.  In host
// code the symbol names a host-side stand-in, not device memory, so the
// address is looked up once per device (with that device current) and kept;
// `refresh` looks it up again (after a device reset the module is loaded
// anew and the kept address is stale).
int noalloc_scratch(unsigned char** out, bool refresh = false) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return MB2_ERR_NO_DEVICE;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (g_noalloc_ptr[dev] == nullptr || refresh) {
        void* p = nullptr;
        if (const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch); e != cudaSuccess)
            return record_cuda_error(e);
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return MB2_OK;
}

}  // namespace

}  // namespace mb2

extern "C" int mb2_expectation_noalloc(const void* dev_amps, uint32_t num_qubits, const uint64_t* x_masks,
                                       const uint64_t* z_masks, uint32_t num_terms, double* out, void* stream) {
    using namespace mb2;
    if (num_terms == 0) return MB2_OK;
    if (num_terms > kNoAllocTerms) return MB2_ERR_RESOURCE;
    if (dev_amps == nullptr || x_masks == nullptr || z_masks == nullptr || out == nullptr || num_qubits < 1 ||
        num_qubits > 40)
        return MB2_ERR_INVALID;
    const uint64_t lim = (uint64_t{1} << num_qubits) - 1;
    for (uint32_t t = 0; t < num_terms; ++t)
        if ((x_masks[t] | z_masks[t]) & ~lim) return MB2_ERR_INVALID;
    unsigned char* base = nullptr;
    if (int rc = noalloc_scratch(&base); rc != MB2_OK) return rc;
    auto* dx = reinterpret_cast<uint64_t*>(base);
    auto* dz = reinterpret_cast<uint64_t*>(base + kNoAllocMasks);
    auto* partials = reinterpret_cast<double*>(base + 2 * kNoAllocMasks);
    auto* dout = reinterpret_cast<double*>(base + 2 * kNoAllocMasks + kNoAllocPartials);
    const auto s = static_cast<cudaStream_t>(stream);
    const size_t mb = size_t{num_terms} * sizeof(uint64_t);
    cudaError_t e = cudaMemcpyAsync(dx, x_masks, mb, cudaMemcpyHostToDevice, s);
    if (e == cudaErrorInvalidValue) {
        // A kept address from before a device reset: look it up again, once.
        cudaGetLastError();
        if (int rc = noalloc_scratch(&base, true); rc != MB2_OK) return rc;
        dx = reinterpret_cast<uint64_t*>(base);
        dz = reinterpret_cast<uint64_t*>(base + kNoAllocMasks);
        partials = reinterpret_cast<double*>(base + 2 * kNoAllocMasks);
        dout = reinterpret_cast<double*>(base + 2 * kNoAllocMasks + kNoAllocPartials);
        e = cudaMemcpyAsync(dx, x_masks, mb, cudaMemcpyHostToDevice, s);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(dz, z_masks, mb, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return record_cuda_error(e);
    // Every partial and every output slot is written before it is read, so
    // nothing left in the array by an earlier call needs clearing.
    if (launch_expectation(dev_amps, num_qubits, dx, dz, num_terms, partials, dout, stream) != MB2_OK)
        return MB2_ERR_CUDA;
    e = cudaMemcpyAsync(out, dout, size_t{num_terms} * 2 * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return record_cuda_error(e);
}

