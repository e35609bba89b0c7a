// resident_f64_strict.cu -- the resident kernel and the observer of one precision tier (see
// lbm_step_resident.cuh, observe.cuh).
#include "lbm_step_resident.cuh"
#include "observe.cuh"

namespace hlbm {
cudaError_t resident_f64_strict(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<double, double, true>(a, walls, s);
}
HLBM_OBSERVE_ENTRY(f64_strict) {
  return launch_observe<double, double, true>(fin, fout, flags, p, blocks, partials, done, out, s);
}
}  // namespace hlbm
