// visg_launch.cuh — kernel launches that overlap the launch before them in the stream.
#pragma once
#include <cuda_runtime.h>

namespace visg {

// Launches overlap (launch_block): what earlier launches wrote (records, normals, trees) is
// read after this, and not through the read-only path, which need not see it; it also lets
// the next launch begin.  A no-op for a launch without the attribute.
__device__ __forceinline__ void wait_for_earlier_launches() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A launch that may begin while the kernel before it in the stream still runs (`overlap`):
// its blocks are placed and do what depends on nothing earlier, then wait
// (wait_for_earlier_launches).  For the short kernels of small simulations, where a launch's
// own latency is a fifth of a step: dragged 64 x 64 sheet 29.1 -> 22.0 us a frame, body moved
// before each of 4 steps 165 -> 154; with the queries begun before the wait, 200 steps of a
// 64 x 64 sheet in contact 1,677 -> 1,358 us, 20 of a 131 x 127 mesh 269 -> 229.  Large
// simulations in one chain of fused steps (SV_OVERLAP) gain the gaps between launches and
// the first tile's copy: 512 x 512 sheet 437 -> 430 us in 4 steps with as many rebuilds,
// 123 -> 114 in 4 steps with the output stage.
template <class... P, class... A>
cudaError_t launch_after(void (*fn)(P...), int grid, int block, int smem, cudaStream_t s, bool overlap, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, fn, (P)args...);
}

}  // namespace visg
