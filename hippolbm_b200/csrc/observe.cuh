// observe.cuh -- simulation_state of a lattice that has only its post-collision state, in one launch.
//
// A run that logs every few steps (print_log_freq) reads three numbers each time.  Streaming the state
// into the idle buffer, reading it back for the macro variables and folding the partial sums took three
// launches, some 22 us on a 31^3 lattice whose ten steps take 36 us, and on a large one wrote and
// re-read all populations.  Here a thread streams a node into registers (the gather and the boundary
// operators of the read-out), rounds it as the read-out would store it, and takes its macro variables;
// the last block to finish folds the partial sums.  Sums run in the order of k_macro_stats and
// k_reduce_partials (aux_kernels.cu), without contraction, so the values are the same.
//
// STORE: the rounded state is stored as the read-out would store it, so that another read-out of the same
// step finds it.  It costs a tenth to a fifth of the pass and saves one, which pays on large lattices:
// observe_stores.
#pragma once
#include <cuda_runtime.h>

#include "lbm_step.cuh"

namespace hlbm {

// what a read-out (MODE_FINISH) stores of direction I's value, as FP64
template <typename S, typename R, int I>
__device__ __forceinline__ double readout_value(R v, const StepPlan& p) {
  if constexpr (is_16bit<S>())
    return double(Codec<S, R>::template dec<I>(Codec<S, R>::template encd<I>(v, p), p));
  else
    return double(v);
}

// Whether simulation_state stores the state: lattices of a million nodes and more.  Measured (us, one step and
// simulation_state / those and moments; before this kernel, without, with storing): FP64 31^3 57, 46, 44 /
// 104, 92, 84; FP16 128^3 205, 167, 180 / 272, 291, 250; FP64 320^3 3873, 2843, 3209 / 5276, 5427, 4301; ten
// steps and simulation_state FP64 31^3 122, 78, 82; 64 x 60 x 61 224, 172, 176.
inline bool observe_stores(const StepPlan& p) { return p.ncell >= (int64_t(1) << 20); }

// out: {sum rho, min |u|, max |u|}; done: blocks finished, zero between launches
template <typename S, typename R, bool STRICT, bool WALLS, bool STORE>
__global__ void __launch_bounds__(256) k_observe(const S* fin, S* __restrict__ fout, const int8_t* __restrict__ flags,
                                                 const __grid_constant__ StepPlan p, double* __restrict__ partials,
                                                 unsigned* __restrict__ done, double* __restrict__ out) {
  double s = 0.0, vmin = 1.79769313486231570815e+308, vmax = -1.79769313486231570815e+308;
  const int64_t plane = int64_t(p.nx) * p.ny;
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < p.ncell; idx += int64_t(gridDim.x) * blockDim.x) {
    double rho = 0.0, ux = 0.0, uy = 0.0, uz = 0.0;
    const int8_t flag = flags[idx];
    if (STORE && WALLS && flag == FLAG_WALL) {
      Unroll<0, Q>::run([&]<int I>() { fout[I * p.stride + idx] = Codec<S, R>::template enc<I>(R(0), p); });
    } else if (STORE || flag >= FLAG_FLUID) {
      const int z = int(idx / plane);
      const int64_t rem = idx - z * plane;
      const int y = int(rem / p.nx), x = int(rem - int64_t(y) * p.nx);
      S raw[Q];
      node_pull<S, WALLS, LOAD_WAIT, true>(fin, flags, p, x, y, z, idx, raw, true);
      R v[Q];
      Unroll<0, Q>::run([&]<int I>() { v[I] = load_value<S, R, I>(raw[I], p); });
      node_update<S, R, STRICT, MODE_FINISH, 2>(v, fin, idx, x, y, z, flag, p, true, on_op_face(p, x, y, z));
      if constexpr (STORE) store_node<S, R, MODE_FINISH>(v, p, 0, idx, [&]<int I>(S s) { fout[I * p.stride + idx] = s; });
      if (!STORE || flag >= FLAG_FLUID) {
        double d[Q];
        Unroll<0, Q>::run([&]<int I>() { d[I] = readout_value<S, R, I>(v[I], p); });
        macro<double, true>(d, rho, ux, uy, uz);
      }
    }
    s = __dadd_rn(s, rho);
    const double n = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), __dmul_rn(uz, uz)));
    vmin = n < vmin ? n : vmin;
    vmax = n > vmax ? n : vmax;
  }
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, off);
    const double a = __shfl_down_sync(0xffffffffu, vmin, off);
    const double b = __shfl_down_sync(0xffffffffu, vmax, off);
    vmin = a < vmin ? a : vmin;
    vmax = b > vmax ? b : vmax;
  }
  __shared__ double sh[3][256];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    sh[0][warp] = s;
    sh[1][warp] = vmin;
    sh[2][warp] = vmax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = sh[0][0], b = sh[1][0], c = sh[2][0];
    for (int w = 1; w < 8; w++) {
      a += sh[0][w];
      b = sh[1][w] < b ? sh[1][w] : b;
      c = sh[2][w] > c ? sh[2][w] : c;
    }
    partials[3 * blockIdx.x + 0] = a;
    partials[3 * blockIdx.x + 1] = b;
    partials[3 * blockIdx.x + 2] = c;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  s = 0.0, vmin = 1.79769313486231570815e+308, vmax = -1.79769313486231570815e+308;
  for (int i = threadIdx.x; i < int(gridDim.x); i += 256) {
    s += __ldcg(partials + 3 * i);
    const double a = __ldcg(partials + 3 * i + 1), b = __ldcg(partials + 3 * i + 2);
    vmin = a < vmin ? a : vmin;
    vmax = b > vmax ? b : vmax;
  }
  sh[0][threadIdx.x] = s;
  sh[1][threadIdx.x] = vmin;
  sh[2][threadIdx.x] = vmax;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + h];
      sh[1][threadIdx.x] = sh[1][threadIdx.x + h] < sh[1][threadIdx.x] ? sh[1][threadIdx.x + h] : sh[1][threadIdx.x];
      sh[2][threadIdx.x] = sh[2][threadIdx.x + h] > sh[2][threadIdx.x] ? sh[2][threadIdx.x + h] : sh[2][threadIdx.x];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sh[0][0];
    out[1] = sh[1][0];
    out[2] = sh[2][0];
    *done = 0;
  }
}

template <typename S, typename R, bool STRICT, bool WALLS>
void launch_observe_walls(const void* fin, void* fout, const int8_t* flags, const StepPlan& p, int blocks,
                          double* partials, unsigned* done, double* out, cudaStream_t s) {
  const S* fi = static_cast<const S*>(fin);
  S* fo = static_cast<S*>(fout);
  if (fo)
    k_observe<S, R, STRICT, WALLS, true><<<blocks, 256, 0, s>>>(fi, fo, flags, p, partials, done, out);
  else
    k_observe<S, R, STRICT, WALLS, false><<<blocks, 256, 0, s>>>(fi, fo, flags, p, partials, done, out);
}

// fout: where the state is stored, or null
template <typename S, typename R, bool STRICT>
cudaError_t launch_observe(const void* fin, void* fout, const int8_t* flags, const StepPlan& p, int blocks,
                           double* partials, unsigned* done, double* out, cudaStream_t s) {
  if (p.walls)
    launch_observe_walls<S, R, STRICT, true>(fin, fout, flags, p, blocks, partials, done, out, s);
  else
    launch_observe_walls<S, R, STRICT, false>(fin, fout, flags, p, blocks, partials, done, out, s);
  return cudaGetLastError();
}

// one entry per precision tier (defined in resident_*.cu)
#define HLBM_OBSERVE_ENTRY(tier)                                                                                   \
  cudaError_t observe_##tier(const void* fin, void* fout, const int8_t* flags, const StepPlan& p, int blocks,      \
                             double* partials, unsigned* done, double* out, cudaStream_t s)
HLBM_OBSERVE_ENTRY(f64_strict);
HLBM_OBSERVE_ENTRY(f64);
HLBM_OBSERVE_ENTRY(f32);
HLBM_OBSERVE_ENTRY(f16);
HLBM_OBSERVE_ENTRY(bf16);

}  // namespace hlbm
