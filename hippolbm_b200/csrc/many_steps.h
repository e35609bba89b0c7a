// many_steps.h -- the steps of one hlbm_step call as cooperative launches of many steps each.
//
// A cooperative launch can be refused where the same kernel's plain launches would run: a device that
// does not offer them, or a partition of one that holds fewer CTAs than the whole.  The call then goes on
// with one plain launch a step, as it does for lattices that no cooperative launch takes.
#pragma once
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdint>

namespace hlbm {

inline bool launch_refused(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorNotPermitted;
}

// launch(m) for m steps at a time, at most `chunk`, until nsteps are done or one is refused; the steps done in
// `done`.  `forget` drops the refusal from the runtime's last error.
template <class Launch, class Forget>
cudaError_t many_steps(int64_t nsteps, int64_t chunk, int64_t& done, Launch&& launch, Forget&& forget) {
  done = 0;
  while (done < nsteps) {
    const int m = int(std::min(nsteps - done, chunk));
    const cudaError_t e = launch(m);
    if (launch_refused(e)) {
      forget();
      return cudaSuccess;
    }
    if (e != cudaSuccess) return e;
    done += m;
  }
  return cudaSuccess;
}

}  // namespace hlbm
