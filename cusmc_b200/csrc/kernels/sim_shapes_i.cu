// Kernel instantiations for lane-group shapes: 4,8 8,8
#include "sim_impl.cuh"

namespace csmc {
CSMC_INSTANTIATE_SHAPE(4, 8)
CSMC_INSTANTIATE_SHAPE(8, 8)
}  // namespace csmc
