// qms_pdl.cuh -- launches that overlap the start of a kernel with the end of the one before it.
//
// A kernel launched with pdl_launch may start once every CTA of the kernel before it in the stream has
// called pdl_wait (or ended), before that kernel is complete: barrier set-up, index arithmetic and loads
// of data that no kernel of a solve writes run early.  pdl_wait then waits until the kernel before is
// complete and its writes are visible, and lets the next one start; EVERY kernel launched this way calls
// it, in every thread, before its first access to data that another kernel writes, so the order of a
// stream stays what it was.  Data that the kernel before writes is read with plain loads (not the
// read-only path, whose data must not change while a kernel runs).
// A cycle on a small grid is some 40 launches of 3-12 us with a gap of 1 us or more between two.  ms per run of
// steps without and with the overlap: 16x14x12 block 25.3 and 21.8, 96^3 ellipsoids 182 and 171, plate
// 141x97x53 97.8 and 76.5, steady 157x131x143 63.6 and 60.9.  Launches of more than 3000 CTAs do without: 256^3
// 642 ms with that line, 676 with the overlap everywhere, 660 with it nowhere (and a line at 1000 gives up
// most of the gain on the 97^3 grids).
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

#define QMS_PDL_CTAS 3000
// cluster: CTAs per cluster along x (0: none)
template <typename... P, typename... A>
static inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                     unsigned cluster, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim = {cluster, 1, 1};
    // a launch of many waves gains nothing from an early start
    const bool early = (unsigned long long)grid.x * grid.y * grid.z <= QMS_PDL_CTAS;
    cfg.attrs = early ? at : at + 1;
    cfg.numAttrs = (early ? 1 : 0) + (cluster ? 1 : 0);
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
