// resident_f64_strict.cu -- the resident kernel of one precision tier (see lbm_step_resident.cuh).
#include "lbm_step_resident.cuh"

namespace hlbm {
cudaError_t resident_f64_strict(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<double, double, true>(a, walls, s);
}
}  // namespace hlbm
