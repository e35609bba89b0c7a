// resident_f16.cu -- the resident kernel and the observer of one precision tier (see
// lbm_step_resident.cuh, observe.cuh).
#include "lbm_step_resident.cuh"
#include "observe.cuh"

namespace hlbm {
cudaError_t resident_f16(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<__half, float, false>(a, walls, s);
}
HLBM_OBSERVE_ENTRY(f16) {
  return launch_observe<__half, float, false>(fin, fout, flags, p, blocks, partials, done, out, s);
}
}  // namespace hlbm
