// Passes of a sweep launched behind one another on a stream: the next pass's
// CTAs may start while this one's last are at work, stage their program in
// shared memory and compute their offsets, and wait only before they touch
// the state (programmatic dependent launch).  What precedes the first pass
// (an upload, another kernel) is complete before it starts, as ever, and the
// program that a pass stages was uploaded before the sweep's first pass.
// What it saves is the gap between two launches, about 1.6 us a pass.  Beside
// long passes the waiting CTAs cost more than that, so a pass over more than
// 2^kBehindBits amplitudes is launched plainly.  Behind one another and plainly, ms:
// 20 brick layers at 14, 16 and 18 qubits 0.377 0.389, 0.442 0.455, 0.511 0.530;
// at 24 8.81 8.87; 10 layers at 26 19.13 19.18; 8 layers of RY and CZ at 27
// 24.81 24.79; 6 brick layers at 28 54.30 53.90; a sampled density matrix of 11
// qubits 1.22 1.26.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

namespace mb2 {

constexpr uint32_t kBehindBits = 26;

// Lets the next launch's CTAs start as slots free up.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Waits until everything the launches before this one wrote is visible.
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// bits: the amplitudes of the states that the pass runs over are 2^bits.
template <typename... P, typename... A>
void launch_behind(uint32_t bits, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &early;
    config.numAttrs = bits <= kBehindBits ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace mb2
