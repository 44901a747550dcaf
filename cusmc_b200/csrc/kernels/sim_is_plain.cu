// Launch entry points of the importance-sampling kernel of networks without
// invariants (sim_is_plain.cuh).
#include "sim_is_plain.cuh"

namespace csmc {

namespace {
using Kernel = void (*)(const IsParams);
Kernel pick(bool tc, bool trace) {
    if (tc) return trace ? detail::is_plain_kernel<true, true> : detail::is_plain_kernel<true, false>;
    return trace ? detail::is_plain_kernel<false, true> : detail::is_plain_kernel<false, false>;
}
}  // namespace

int is_plain_launch(bool tc, bool trace, const IsParams &p, int grid, int block, size_t smem, void *stream) {
    Kernel fn = pick(tc, trace);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    fn<<<grid, block, smem, static_cast<cudaStream_t>(stream)>>>(p);
    return static_cast<int>(cudaGetLastError());
}

int is_plain_max_active_ctas(bool tc, bool trace, int block, size_t smem, int *ctas) {
    Kernel fn = pick(tc, trace);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    return static_cast<int>(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, block, smem));
}

}  // namespace csmc
