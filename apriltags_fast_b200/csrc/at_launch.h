// Kernel launches of the detection path: a kernel may be set up while the
// one before it in its stream still runs (programmatic dependent launch).
// Every kernel of the path begins with kernel_begin(), before its first
// read or write of global memory: it waits until the one before has ended
// and its writes are visible, and, in grids that leave room on the GPU (at
// most 4 blocks an SM), first lets the next kernel be set up. A frame takes
// some 30 short kernels one after the other (40 when this was measured); the
// launch latency between two of them was 1 to 2 us (640 x 480: 437 us of
// kernels and gaps before, 394 us with it). In larger grids the next kernel's waiting blocks would only take
// room from running ones, of other streams above all (32 frames of 1920 x
// 1080 on three pipelines: 2.17 ms without, 2.40 ms with it everywhere).
#pragma once
#include <cuda_runtime.h>

#include <utility>

__device__ __forceinline__ void kernel_begin() {
    if (gridDim.x * gridDim.y <= 148 * 4) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
