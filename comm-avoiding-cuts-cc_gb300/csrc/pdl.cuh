// Programmatic dependent launch of the kernels of a query that follow one another on one stream.
#pragma once
#include <cuda_runtime.h>

namespace cac {

// Programmatic dependent launch: a kernel launched with launch_pdl may start while its predecessor
// on the stream drains; pdl_wait() (griddepcontrol.wait) holds it until the predecessor has
// completed and its writes are visible, so every kernel calls it before its first dependent
// access. After an ordinary launch it returns at once. Measured on the CC query (17 kernels in
// one replayed graph, L2 flushed): BA n=1,024,000 184.7 -> 182.9 us, R-MAT scale 22 493 -> 491; on approx_cut (16 launches a
// level, no graph): G(10^6, M = 10^7) 446 -> 413 us.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace cac
