// A channel of the trajectory engine on the device, for a batch of
// trajectories at once (states back to back, trajectory t at t * 2^n): the
// reduced density matrix of the channel's qubits, the branch it selects for
// each trajectory's uniform, that branch's Kraus operator, and the scale by
// 1 / sqrt of the exact norm (kernels_sample.cu's chain between the last two).
//
// On the host this was a round trip per channel and trajectory -- the
// expectations of 4^k Pauli strings copied back, the branch chosen, the
// matrix sent, the norm copied back -- 115 us a channel at 14 qubits, of which
// the kernels were 60.  Here nothing returns before a trajectory's outputs,
// every launch serves the whole batch, and the scale is fused with the next
// channel's reduced density matrix (one read and one write of the state less).
#include <cuda_runtime.h>

#include <cstdint>

#include "device_math.cuh"
#include "mb2_internal.h"

namespace mb2 {
namespace {
using namespace dev;

constexpr int kThreads = 256;

// 1 / sqrt(norm), as the host computed it (both operations correctly rounded).
__device__ __forceinline__ double scale_of(const TrajNorm& w, uint32_t t, int* err) {
    const double norm = w.norms[static_cast<uint64_t>(t) * w.pitch];
    if (!(norm > 0.0) && blockIdx.x == 0 && threadIdx.x == 0 && err[t] == 0) err[t] = kTrajAnnihilated;
    return __ddiv_rn(1.0, __dsqrt_rn(norm));
}

__global__ void __launch_bounds__(kThreads) k_traj_scale(double2* __restrict__ st, uint32_t n, TrajNorm w,
                                                         int* __restrict__ err) {
    const uint32_t t = blockIdx.y;
    const double s = scale_of(w, t, err);
    const uint64_t na = uint64_t{1} << n;
    double2* const a = st + t * na;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; i < na;
         i += static_cast<uint64_t>(gridDim.x) * kThreads)
        a[i] = canon(cmul_re(s, a[i]));
}

// The index of group g's first amplitude: zeros inserted at the channel's
// qubits (ascending in `sorted`).
template <int K>
__device__ __forceinline__ uint64_t group_base(uint64_t g, const TrajQubits& q) {
#pragma unroll
    for (int j = 0; j < K; ++j) g = insert_zero(g, q.sorted[j]);
    return g;
}

// Element e's offset within a group: bit j of e on qubit q[j].
template <int K>
__device__ __forceinline__ uint64_t group_off(uint32_t e, const TrajQubits& q) {
    uint64_t o = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) o |= static_cast<uint64_t>((e >> j) & 1u) << q.q[j];
    return o;
}

// Partial sums of rho[r][c] = sum a[r] conj(a[c]) over the groups: D*D reals
// per block, the diagonal, then (re, im) of r < c row by row.  Bound by the
// read of the state; w.norms != nullptr: each amplitude is first scaled and
// written back.
template <int K>
__global__ void __launch_bounds__(kThreads) k_traj_rho(double2* __restrict__ st, uint32_t n, TrajQubits q, TrajNorm w,
                                                       int* __restrict__ err, double* __restrict__ partials) {
    constexpr int D = 1 << K;
    const uint32_t t = blockIdx.y;
    double2* const a = st + (static_cast<uint64_t>(t) << n);
    const bool scaled = w.norms != nullptr;
    const double s = scaled ? scale_of(w, t, err) : 1.0;
    const uint64_t groups = uint64_t{1} << (n - K);
    double acc[D * D];
#pragma unroll
    for (int i = 0; i < D * D; ++i) acc[i] = 0.0;
    for (uint64_t g = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; g < groups;
         g += static_cast<uint64_t>(gridDim.x) * kThreads) {
        const uint64_t b = group_base<K>(g, q);
        double2 v[D];
#pragma unroll
        for (int e = 0; e < D; ++e) v[e] = a[b | group_off<K>(e, q)];
        if (scaled) {
#pragma unroll
            for (int e = 0; e < D; ++e) {
                v[e] = canon(cmul_re(s, v[e]));
                a[b | group_off<K>(e, q)] = v[e];
            }
        }
        int i = D;
#pragma unroll
        for (int r = 0; r < D; ++r) {
            acc[r] += v[r].x * v[r].x + v[r].y * v[r].y;
#pragma unroll
            for (int c = r + 1; c < D; ++c) {
                acc[i] += v[r].x * v[c].x + v[r].y * v[c].y;
                acc[i + 1] += v[r].y * v[c].x - v[r].x * v[c].y;
                i += 2;
            }
        }
    }
    __shared__ double sh[kThreads / 32][D * D];
#pragma unroll
    for (int i = 0; i < D * D; ++i)
        for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_down_sync(0xffffffffu, acc[i], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int i = 0; i < D * D; ++i) sh[threadIdx.x >> 5][i] = acc[i];
    __syncthreads();
    if (threadIdx.x < D * D) {
        double v = 0.0;
        for (int x = 0; x < kThreads / 32; ++x) v += sh[x][threadIdx.x];
        partials[(static_cast<uint64_t>(t) * gridDim.x + blockIdx.x) * (D * D) + threadIdx.x] = v;
    }
}

// One CTA per trajectory: the partials added in a fixed order, then the
// branch as the reference chooses it (choose_branch,
// src/engines/trajectory/trajectory_engine.cpp:123-152): the first whose
// cumulative p_b = Re Tr(M_b rho) exceeds the uniform, else the last with
// p_b > 0.  products: `branches` matrices K^dagger K, D x D complex.
template <int K>
__global__ void __launch_bounds__(kThreads)
    k_traj_select(const double* __restrict__ partials, uint32_t blocks, const double2* __restrict__ products,
                  uint32_t branches, const double* __restrict__ uniforms, uint32_t pitch, uint32_t* __restrict__ chosen,
                  int* __restrict__ err) {
    constexpr int D = 1 << K, E = D * D, kParts = kThreads / E;
    __shared__ double sh[kThreads];
    __shared__ double2 rho[D][D];
    const uint32_t t = blockIdx.x, e = threadIdx.x % E, part = threadIdx.x / E;
    const double* p = partials + static_cast<uint64_t>(t) * blocks * E;
    double v = 0.0;
    for (uint32_t b = part; b < blocks; b += kParts) v += p[static_cast<uint64_t>(b) * E + e];
    sh[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < E) {
        v = sh[threadIdx.x];
        for (int x = 1; x < kParts; ++x) v += sh[x * E + threadIdx.x];
        sh[threadIdx.x] = v;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    int i = D;
    for (int r = 0; r < D; ++r) {
        rho[r][r] = make_double2(sh[r], 0.0);
        for (int c = r + 1; c < D; ++c, i += 2) {
            rho[r][c] = make_double2(sh[i], sh[i + 1]);
            rho[c][r] = make_double2(sh[i], -sh[i + 1]);
        }
    }
    const double u = uniforms[static_cast<uint64_t>(t) * pitch];
    double cumulative = 0.0;
    int64_t branch = -1, last = -1;
    for (uint32_t b = 0; b < branches && branch < 0; ++b) {
        double prob = 0.0;
        for (int a = 0; a < D; ++a)
            for (int c = 0; c < D; ++c) {
                const double2 m = products[(static_cast<uint64_t>(b) * D + a) * D + c], r = rho[c][a];
                prob += m.x * r.x - m.y * r.y;
            }
        if (prob > 0.0) {
            last = b;
            cumulative += prob;
            if (u < cumulative) branch = b;
        }
    }
    if (branch < 0) branch = last;
    if (branch < 0 && err[t] == 0) err[t] = kTrajNoBranch;
    chosen[t] = branch < 0 ? 0u : static_cast<uint32_t>(branch);
}

// The chosen branch's operator on every group: each output the products with
// the inputs in increasing order, every product and sum rounded (the
// reference's apply_matrix; an entry that is zero adds a zero, which
// changes at most the sign of a zero, and stored zeros are positive).
template <int K>
__global__ void __launch_bounds__(kThreads) k_traj_apply(double2* __restrict__ st, uint32_t n, TrajQubits q,
                                                         const double2* __restrict__ kraus,
                                                         const uint32_t* __restrict__ chosen) {
    constexpr int D = 1 << K;
    __shared__ double2 m[D * D];
    const uint32_t t = blockIdx.y;
    if (threadIdx.x < D * D) m[threadIdx.x] = kraus[static_cast<uint64_t>(chosen[t]) * (D * D) + threadIdx.x];
    __syncthreads();
    double2* const a = st + (static_cast<uint64_t>(t) << n);
    const uint64_t groups = uint64_t{1} << (n - K);
    for (uint64_t g = static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x; g < groups;
         g += static_cast<uint64_t>(gridDim.x) * kThreads) {
        const uint64_t b = group_base<K>(g, q);
        double2 v[D];
#pragma unroll
        for (int e = 0; e < D; ++e) v[e] = a[b | group_off<K>(e, q)];
#pragma unroll
        for (int o = 0; o < D; ++o) {
            double2 x = cmul(m[o * D].x, m[o * D].y, v[0]);
#pragma unroll
            for (int i = 1; i < D; ++i) x = cadd(x, cmul(m[o * D + i].x, m[o * D + i].y, v[i]));
            a[b | group_off<K>(o, q)] = canon(x);
        }
    }
}

// Enough blocks to fill the GPU, each thread some groups; a function of the
// sizes alone, so the sums do not depend on the batch.
uint32_t blocks_of(uint64_t groups) {
    const uint64_t b = groups / (4 * kThreads);
    return static_cast<uint32_t>(b < 1 ? 1 : b < 1184 ? b : 1184);
}

template <int K>
int channel_t(double2* st, uint32_t n, uint32_t batch, const TrajQubits& q, const TrajNorm& w, const TrajChannelData& c,
              void* scratch, int* err, cudaStream_t s) {
    const uint32_t nb = blocks_of(uint64_t{1} << (n - K));
    auto* chosen = static_cast<uint32_t*>(scratch);
    auto* partials = reinterpret_cast<double*>(static_cast<unsigned char*>(scratch) + ((batch * 4 + 255) & ~255u));
    const dim3 grid(nb, batch);
    k_traj_rho<K><<<grid, kThreads, 0, s>>>(st, n, q, w, err, partials);
    k_traj_select<K><<<batch, kThreads, 0, s>>>(partials, nb, static_cast<const double2*>(c.products), c.branches,
                                                c.uniforms, c.pitch, chosen, err);
    k_traj_apply<K><<<grid, kThreads, 0, s>>>(st, n, q, static_cast<const double2*>(c.kraus), chosen);
    note_launches(3);
    return launch_status();
}

}  // namespace

size_t traj_scratch_bytes(uint32_t n, uint32_t batch) {
    // k = 3 has the most sums per block, k = 1 the most blocks.
    size_t most = 0;
    for (uint32_t k = 1; k <= 3 && k <= n; ++k)
        most = most < (size_t{blocks_of(uint64_t{1} << (n - k))} << (2 * k))
                   ? size_t{blocks_of(uint64_t{1} << (n - k))} << (2 * k)
                   : most;
    return ((batch * 4 + 255) & ~255u) + most * batch * sizeof(double);
}

int launch_traj_channel(void* amps, uint32_t n, uint32_t batch, const uint32_t* qubits, uint32_t k, const TrajNorm& norm,
                        const TrajChannelData& c, void* scratch, int* dev_err, void* stream) {
    if (k < 1 || k > 3 || k > n || batch < 1 || batch > 65535) return MB2_ERR_INVALID;
    TrajQubits q{};
    for (uint32_t j = 0; j < k; ++j) q.q[j] = q.sorted[j] = qubits[j];
    for (uint32_t i = 0; i < k; ++i)
        for (uint32_t j = i + 1; j < k; ++j)
            if (q.sorted[j] < q.sorted[i]) {
                const uint32_t x = q.sorted[i];
                q.sorted[i] = q.sorted[j];
                q.sorted[j] = x;
            }
    auto* st = static_cast<double2*>(amps);
    const auto s = static_cast<cudaStream_t>(stream);
    return k == 1   ? channel_t<1>(st, n, batch, q, norm, c, scratch, dev_err, s)
           : k == 2 ? channel_t<2>(st, n, batch, q, norm, c, scratch, dev_err, s)
                    : channel_t<3>(st, n, batch, q, norm, c, scratch, dev_err, s);
}

int launch_traj_scale(void* amps, uint32_t n, uint32_t batch, const TrajNorm& norm, int* dev_err, void* stream) {
    if (batch < 1 || batch > 65535) return MB2_ERR_INVALID;
    k_traj_scale<<<dim3(blocks_of(uint64_t{1} << n), batch), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<double2*>(amps), n, norm, dev_err);
    note_launches(1);
    return launch_status();
}

}  // namespace mb2
