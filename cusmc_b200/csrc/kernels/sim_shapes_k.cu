// Kernel instantiations for lane-group shapes: 8,16 16,16
#include "sim_impl.cuh"

namespace csmc {
CSMC_INSTANTIATE_SHAPE(8, 16)
CSMC_INSTANTIATE_SHAPE(16, 16)
}  // namespace csmc
