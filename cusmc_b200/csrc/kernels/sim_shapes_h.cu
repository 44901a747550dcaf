// Kernel instantiations for lane-group shapes: 8,4 16,4
#include "sim_impl.cuh"

namespace csmc {
CSMC_INSTANTIATE_SHAPE(8, 4)
CSMC_INSTANTIATE_SHAPE(16, 4)
}  // namespace csmc
