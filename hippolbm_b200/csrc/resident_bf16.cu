// resident_bf16.cu -- the resident kernel of one precision tier (see lbm_step_resident.cuh).
#include "lbm_step_resident.cuh"

namespace hlbm {
cudaError_t resident_bf16(const ResidentArgs& a, int walls, cudaStream_t s) {
  return launch_resident<__nv_bfloat16, float, false>(a, walls, s);
}
}  // namespace hlbm
