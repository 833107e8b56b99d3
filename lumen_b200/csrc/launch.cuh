// Launches that overlap the end of the kernel before them (programmatic dependent launch).
//
// A kernel launched with `launch_overlapped` may become resident as soon as every block of the kernel before it in its stream
// has ended, before that one's memory is flushed and its end has been reported: launch, block setup (barriers, tensor memory,
// descriptors) and the earlier kernel's last microsecond fall together. Every kernel launched this way calls `grid_wait` in
// every thread, before it reads or writes memory that another kernel may touch and before any wait with a bound: it returns
// once the kernels before it have completed and their writes are visible (and has no bound of its own). As each of them did the same, that holds for the
// whole stream before it, and what is launched in the ordinary way afterwards is ordered as ever.
//
// The wait is a barrier to ordinary loads and stores, but a compiler takes what is read through `const __restrict__` parameters
// (and __ldg) for constant while the kernel runs and may move such a load across it. `grid_wait` is therefore given those
// parameters (or what was computed from them) and makes them values that come out of the wait, so that the addresses computed from
// them do too. Pointers in a struct of arguments are read by ordinary loads.
//
// No kernel lets the next one come earlier (griddepcontrol.launch_dependents): its blocks would be dealt to the SMs that this
// one leaves idle, several to one SM, and stay there. Measured (us a pass, ordinary launches -> these -> these with the next
// kernel let in from the start): MLP forward and backward of 200 tokens x 1024 x 4096, bfloat16, eight kernels 81.6 -> 64.5 ->
// 65.7; a 2-layer float32 training step, 73 kernels replayed as a graph 324 -> 310 -> 400.
#pragma once
#include "device.h"

namespace lb {

template <class P>
__device__ __forceinline__ void behind_wait(P& pointer) {
    size_t at = __cvta_generic_to_global(pointer);
    asm volatile("" : "+l"(at)::"memory");
    pointer = (P)__cvta_global_to_generic(at);  // known to lead to global memory
}
template <class... P>
__device__ __forceinline__ void grid_wait(P&... read) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (behind_wait(read), ...);
}

// kernel<<<grid, block, smem, stream>>>(args...), overlapping the kernel before it; `cluster`: CTAs per cluster along x where
// the kernel does not fix them itself.
template <class... Params, class... Args>
void launch_overlapped(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, unsigned cluster, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cfg.attrs = attr, cfg.numAttrs = cluster ? 2 : 1;
    LB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

}  // namespace lb
