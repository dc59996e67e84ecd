// IC-GN solver instantiations for the quadratic model (see solver_impl.cuh).
#include "gbdic_kernels.h"
#include "solver_band.cuh"

namespace gbdic {
GBDIC_SOLVER_MODEL(kModelQuadratic)
}  // namespace gbdic
