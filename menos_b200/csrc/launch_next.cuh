// Passes of a sweep launched behind one another on a stream: the next pass's
// CTAs may start while this one's last are at work, stage their program in
// shared memory and compute their offsets, and wait only before they touch
// the state (programmatic dependent launch).  What precedes the first pass
// (an upload, another kernel) is complete before it starts, as ever, and the
// program that a pass stages was uploaded before the sweep's first pass.
// What it saves is the gap between two launches, 1.6 us a pass: 21 passes over
// a density matrix of 11 qubits, sampled, 1.223 -> 1.190 ms a call (two runs
// of one side differ by 0.2 %).  Sweeps with much longer passes, or with host
// work beside short ones, are equal within the difference of two runs.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace mb2 {

// Lets the next launch's CTAs start as slots free up.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Waits until everything the launches before this one wrote is visible.
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... P, typename... A>
void launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &early;
    config.numAttrs = 1;
    cudaLaunchKernelEx(&config, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace mb2
