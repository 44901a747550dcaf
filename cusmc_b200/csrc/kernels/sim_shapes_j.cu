// Kernel instantiations for lane-group shapes: 16,8
#include "sim_impl.cuh"

namespace csmc {
CSMC_INSTANTIATE_SHAPE(16, 8)
}  // namespace csmc
