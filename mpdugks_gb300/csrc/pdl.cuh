// Programmatic dependent launch: a step's kernels follow one another in one stream, each
// reading what the one before wrote.  Launched this way, a kernel's blocks are placed as soon
// as every block of the kernel before has started, and wait in pdl_wait() for that kernel to
// complete (its writes are then visible), so the launch and the block start-up of a kernel
// overlap the end of the one before.  pdl_wait() comes first in a kernel: completion is
// transitive (the kernel before has waited for its own predecessor).
// What such a kernel reads of an earlier kernel's writes it reads by ordinary loads: those of the
// read-only path (__ldg, const __restrict__ parameters) are for data that stays unwritten for
// the whole life of a kernel, which here begins before the last writes, and may be moved ahead
// of the wait.  (The streaming step's phi and aux by either kind of load: 81.3 us a step at
// 512x2048, 639 at 3072x3072.)
// Passes of steps, plain / programmatic launches: 128x128 HCZ FP32 storage 2.24 / 1.61 ms (200
// steps), UW 512x512 in four launches a step 7.71 / 6.97 (100), D2Q9PP 150x133 in three 4.29 /
// 3.95 (200), 32x24 AC FP64 1.86 / 1.69 (50).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace dugks {

__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// early: whether the launch may be brought forward; else it starts after the kernel before
template <typename... P, typename... A>
inline cudaError_t launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    return launch_after(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}

}  // namespace dugks
