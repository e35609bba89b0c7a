// resident_bf16.cu -- the resident kernel and the observer of one precision tier (see
// lbm_step_resident.cuh, observe.cuh).
#include "lbm_step_resident.cuh"
#include "observe.cuh"

namespace hlbm {
cudaError_t resident_bf16(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<__nv_bfloat16, float, false>(a, walls, s);
}
HLBM_OBSERVE_ENTRY(bf16) {
  return launch_observe<__nv_bfloat16, float, false>(fin, fout, flags, p, blocks, partials, done, out, s);
}
}  // namespace hlbm
