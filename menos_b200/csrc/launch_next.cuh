// Passes of a sweep launched behind one another on a stream: the next pass's
// CTAs may start while this one's last are at work, stage their program in
// shared memory and compute their offsets, and wait only before they touch
// the state (programmatic dependent launch).  What precedes the first pass
// (an upload, another kernel) is complete before it starts, as ever, and the
// program that a pass stages was uploaded before the sweep's first pass.
//
// What it saves is the gap between two launches, about 1.6 us a pass.  Beside
// long passes the waiting CTAs cost more than that, and where complex128 passes
// without and with blocks of three or more qubits follow one another, whose
// CTAs differ in size and last milliseconds, far more: so only passes over at
// most 64 MiB of states are, and not where those meet (TileLaunch::behind).
// Behind one another and plainly, ms, complex128: 20 brick layers at 14, 16
// and 18 qubits 0.377 0.389, 0.442 0.455, 0.511 0.530, at 24 8.81 8.87; 6 at 28
// 54.30 53.90; a sampled density matrix of 11 qubits 1.22 1.26; layers of H and
// four blocks of four qubits (passes without, then with them) at 18 qubits 1.04
// 1.01, at 22 5.07 4.93 (plainly only where they meet 4.88), at 26 75.8 71.5;
// the fused RY/RZ + CX ansatz of 12 layers (lean and full passes, no such
// blocks) at 16 qubits 0.517 0.551.  Complex64: the RY/RZ + CX ansatz of 10 layers
// at 23 qubits 2.21 2.24; layers of H and CCX (the full kernel) at 20 1.07
// 1.11, with CX at 26 94.9 88.0.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace mb2 {

// Lets the next launch's CTAs start as slots free up.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Waits until everything the launches before this one wrote is visible.
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... P, typename... A>
void launch_behind(bool behind, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &early;
    config.numAttrs = behind ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace mb2
