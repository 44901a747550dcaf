// Kernel instantiations for lane-group shapes: 16,2 2,4 4,4
#include "sim_impl.cuh"

namespace csmc {
CSMC_INSTANTIATE_SHAPE(16, 2)
CSMC_INSTANTIATE_SHAPE(2, 4)
CSMC_INSTANTIATE_SHAPE(4, 4)
}  // namespace csmc
