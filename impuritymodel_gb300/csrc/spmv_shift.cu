// The shifted products of spmv_kernels.cuh: Y = H X + shift X on the float copies.
#include "spmv_kernels.cuh"

namespace edgpu {

template int dispatch_lanes<float, true, true>(const edgpu_csr*, const float*, const int32_t*, int64_t, int, int, float,
                                               const void*, void*, int, cudaStream_t);
template int dispatch_lanes<float, false, true>(const edgpu_csr*, const float*, const int32_t*, int64_t, int, int, float,
                                                const void*, void*, int, cudaStream_t);
template int launch_pages<float, true, true>(int64_t, const void*, int, int, int, int, float, const void*, void*,
                                             cudaStream_t);
template int launch_pages<float, false, true>(int64_t, const void*, int, int, int, int, float, const void*, void*,
                                              cudaStream_t);

}  // namespace edgpu
