// Programmatic dependent launch: a kernel of a chain is brought up while the one before it runs, loads
// what no kernel of the chain writes (the matrix: offsets, columns, first values), and then waits.
// A multigrid cycle is 23-70 kernels of 2-3 us on small levels, and of those 2-3 us about half is
// the launch and the first dependent loads.  Measured (B200, us an iteration of the flexible CG without
// -> with): 52k edges 83 -> 66, 115k 93 -> 78, 404k 151 -> 137, 1.35M 288 -> 243, 3.2M 498 -> 456,
// 11M 2025 -> 1940 (all with FP32 vectors in the flexible CG, learned.cu).  Letting the next kernel come up behind the wait instead of before it gave 67, 78, 138,
// 247, 460, 1946; at the kernel's very start 67, 80, 139, 245, 459, 1942.
// The Chebyshev polynomial's steps: 28 -> 23 us an iteration (13k edges), 44 -> 38 (175k), 83 -> 73 (404k).
// Not the two kernels of plain CG: 65.4 -> 61.7 ms for a batch of four small systems, but 32.8 -> 34.1 us an
// iteration at 1.1M edges and 57.9 -> 59.9 (FP32) at 3.2M.
// The multigrid setup's small kernels are chained too, with nothing read ahead: 1.93 -> 1.62 ms (52k
// edges), 5.66 -> 5.16 (1.35M), 7.2 -> 6.6 (3.2M), 24.6 -> 23.3 (11M).
#pragma once
#include <cuda_runtime.h>

namespace mh {

// Lets the next kernel come up, and returns when everything the kernels before wrote is there.  Every
// thread calls it, on every path, before it reads or writes anything but such constants: a kernel
// ends only behind its own wait, so the wait for the last kernel is one for all before it.  A
// vector that a kernel of the chain writes must not be a __restrict__ argument of another, whose loads
// the compiler could move above the wait, nor be read by __ldg.  Does nothing in a kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// chained: the launch before on s is a kernel that writes nothing this one reads ahead of its wait.
template <typename... P, typename... A>
inline cudaError_t launch_chained(bool chained, void (*kernel)(P...), dim3 grid, unsigned block, cudaStream_t s,
                                  A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace mh
