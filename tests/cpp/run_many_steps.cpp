// many_steps (hippolbm_b200/csrc/many_steps.h) with launches that a device refuses, at once or after some,
// and launches that fail: refused ones leave the rest to the caller, failures are reported.
#include <cstdio>
#include <vector>

#include "many_steps.h"

int main() {
  struct Case {
    cudaError_t error;
    int after;  // launches that succeed first
    int64_t nsteps, done;
    cudaError_t result;
    int forgotten;
  };
  const Case cases[] = {{cudaSuccess, 1 << 20, 700, 700, cudaSuccess, 0},
                        {cudaErrorCooperativeLaunchTooLarge, 0, 700, 0, cudaSuccess, 1},
                        {cudaErrorNotSupported, 0, 1, 0, cudaSuccess, 1},
                        {cudaErrorNotPermitted, 2, 700, 512, cudaSuccess, 1},
                        {cudaErrorIllegalAddress, 1, 700, 256, cudaErrorIllegalAddress, 0}};
  for (const Case& c : cases) {
    std::vector<int> sizes;
    int forgotten = 0;
    int64_t done = -1, sum = 0;
    const auto launch = [&](int m) {
      if (int(sizes.size()) >= c.after) return c.error;
      sizes.push_back(m);
      sum += m;
      return cudaSuccess;
    };
    const cudaError_t e = hlbm::many_steps(c.nsteps, 256, done, launch, [&] { forgotten++; });
    if (e != c.result || done != c.done || sum != done || forgotten != c.forgotten) {
      std::printf("error %d: result %d, %lld steps done\n", int(c.error), int(e), static_cast<long long>(done));
      return 1;
    }
  }
  return 0;
}
