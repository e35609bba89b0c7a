// resident_f64.cu -- the resident kernel and the observer of one precision tier (see
// lbm_step_resident.cuh, observe.cuh).
#include "lbm_step_resident.cuh"
#include "observe.cuh"

namespace hlbm {
cudaError_t resident_f64(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<double, double, false>(a, walls, s);
}
HLBM_OBSERVE_ENTRY(f64) {
  return launch_observe<double, double, false>(fin, fout, flags, p, blocks, partials, done, out, s);
}
}  // namespace hlbm
