// Grid-stride loops over vertices. Vertex counts reach 2^32 - 1, so the counter has 64 bits: a 32-bit one
// wraps below n after the last step when n is within a stride of 2^32, and the loop starts over for ever.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CAC_LOOP_HD __host__ __device__ __forceinline__
#else
#define CAC_LOOP_HD inline
#endif

namespace cac {

// f(i) for i = first, first + stride, ... below n
template <typename F>
CAC_LOOP_HD void strided(uint32_t first, uint32_t stride, uint32_t n, F f) {
    for (uint64_t i = first; i < n; i += stride) f((uint32_t)i);
}

#ifdef __CUDACC__
// the calling thread's share of [0, n); every thread takes `per` strides at a time
template <typename F>
__device__ __forceinline__ void grid_stride(uint32_t n, F f, uint32_t per = 1) {
    strided(blockIdx.x * blockDim.x + threadIdx.x, per * gridDim.x * blockDim.x, n, f);
}
#endif

}  // namespace cac
