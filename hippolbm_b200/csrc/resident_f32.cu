// resident_f32.cu -- the resident kernel and the observer of one precision tier (see
// lbm_step_resident.cuh, observe.cuh).
#include "lbm_step_resident.cuh"
#include "observe.cuh"

namespace hlbm {
cudaError_t resident_f32(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<float, float, false>(a, walls, s);
}
HLBM_OBSERVE_ENTRY(f32) {
  return launch_observe<float, float, false>(fin, fout, flags, p, blocks, partials, done, out, s);
}
}  // namespace hlbm
