// Instantiations of the batch kernel with warp-per-run jobs.
#include "sim_batch.cuh"

namespace csmc {

int batch_group_launch(bool verify, const BatchParams &p, int grid, int block, void *stream) {
    return verify ? batch_launch_one<true, true>(p, grid, block, stream)
                  : batch_launch_one<false, true>(p, grid, block, stream);
}

int batch_group_occupancy(bool verify, int block, size_t smem, int *ctas) {
    return verify ? batch_occupancy_one<true, true>(block, smem, ctas)
                  : batch_occupancy_one<false, true>(block, smem, ctas);
}

}  // namespace csmc
