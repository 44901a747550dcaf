// Launch entry points of the multi-network batch kernel; the instantiations
// with warp-per-run jobs are compiled in sim_batch_group.cu.
#include "sim_batch.cuh"

namespace csmc {

int batch_group_launch(bool verify, const BatchParams &p, int grid, int block, void *stream);
int batch_group_occupancy(bool verify, int block, size_t smem, int *ctas);

int batch_launch(bool verify, const BatchParams &p, int grid, int block, void *stream) {
    if (p.n_group_jobs > 0) return batch_group_launch(verify, p, grid, block, stream);
    return verify ? batch_launch_one<true, false>(p, grid, block, stream)
                  : batch_launch_one<false, false>(p, grid, block, stream);
}

int batch_max_active_ctas(bool verify, int group_k, int block, size_t smem, int *ctas) {
    if (group_k > 0) return batch_group_occupancy(verify, block, smem, ctas);
    return verify ? batch_occupancy_one<true, false>(block, smem, ctas)
                  : batch_occupancy_one<false, false>(block, smem, ctas);
}

}  // namespace csmc
