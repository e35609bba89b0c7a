// lbm_step_resident.cuh -- many time steps in one launch, for lattices whose two population
// buffers stay in L2.
//
// What bounds a small lattice stepped launch by launch is not its bytes: each launch starts with
// cold instruction and constant caches, runs one latency chain (index arithmetic, one round of
// loads, one collision, one round of stores) and drains, and the tiers with a fix-up launch do that
// twice a step.  Here one cooperative launch takes many steps: its CTAs step the lattice's nodes and a
// barrier (a counter in global memory) separates the steps.  Measured (us a step): FP64 31^3
// 6.3 -> 3.5, FP32 24^3 11.4 -> 2.6, FP16 24^3 20.6 -> 3.1, BF16 57 x 43 x 61 20 -> 8.4; the barrier alone
// takes 1.2 of them.
//
// A lattice of no more nodes than the launch has threads gets one node per thread for the whole launch,
// whose addresses to pull from are computed once.  Larger ones (16-bit tiers) work through items, whole
// warps of one kind:
//   faces     the nodes on the lattice's faces, each once, by the general one-node gather (periodic
//             wrap, on-node bounce-back) and the boundary operators;
//   interior  the node pairs (n, n + 1), n even, of every other kernel, whose sources are idx - d_I: one
//             offset per direction, packed FP32 and one 32-bit store per direction (a pair with one node
//             on a face stores its other half alone), so the stored bits are the same.
// Warps are dealt out across the CTAs first, so a lattice of few items still uses every SM; CTAs have no
// more warps than that takes, so that the launches of several small lattices, each on its stream, share the
// SMs (resident_shape).
//
// The buffers change hands between SMs inside the launch, so populations are read past L1 (ld_l2);
// flags and the near-wall map do not change and go through it.  Every wait is bounded by wait_limit
// polls and two seconds, after which the kernel records an error and returns.  A cooperative launch
// starts only when all its CTAs are resident, so they can wait for one another.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "group_barrier.cuh"
#include "lbm_step_vec.cuh"

namespace hlbm {

constexpr int RES_THREADS = 512;      // threads of a CTA at most: one CTA per SM, 128 registers a thread
constexpr int RES_BAR_STRIDE = 32;    // the barrier's counter lies 128 bytes past the count of CTAs that have left

struct ResidentArgs {
  const LatticeDesc* desc = nullptr;
  int nsteps = 0;
  int parity = 0;              // f[cur ^ parity] is read first
  uint32_t seed = 0;           // step number of the first step
  unsigned* left = nullptr;    // CTAs that have left the launch; zero between launches
  unsigned* bar = nullptr;     // the barrier's counter, zero between launches
  int* err = nullptr;
  int grid = 0, threads = RES_THREADS;
  long long wait_limit = TMA_WAIT_LIMIT;
};

// Whether the resident kernel steps a plan: no zero-gradient pass before the step, and
// 32-bit element offsets over all planes.
inline bool resident_plan(const StepPlan& p) {
  for (int o = 0; o < p.nops; o++)
    if (p.ops[o].kind == OP_ZERO_GRADIENT) return false;
  return int64_t(Q) * p.stride < (int64_t(1) << 31);
}

// CTAs and threads of a launch.  A lattice with a thread for each node takes as many warps as it has, spread
// over all SMs: as blocks of 512 threads it filled the register file of every SM with idle warps, and eight
// FP64 24^3 lattices, each on its stream, took 3.2 us a lattice step, against 0.9 with the warps they need.
inline void resident_shape(int64_t ncell, int sms, int& grid, int& threads) {
  grid = int(std::min<int64_t>(sms, (ncell + 63) / 64));
  const int64_t warps = (ncell + 32 * grid - 1) / (32 * int64_t(grid));
  threads = 32 * int(std::min<int64_t>(RES_THREADS / 32, warps));
}

// floor(n / d) = umul64hi(n, m) for n < 2^32, m = ceil(2^64 / d); d = 1 is marked by m = 0
__host__ __device__ inline uint64_t res_magic(uint64_t d) { return d <= 1 ? 0 : ~uint64_t(0) / d + 1; }
__device__ __forceinline__ uint32_t res_div(uint32_t n, uint64_t m) { return m == 0 ? n : uint32_t(__umul64hi(uint64_t(n), m)); }

// What the threads need of a lattice besides its plan, staged in shared memory.
struct ResidentGeometry {
  int off[Q];                      // element offset of direction I's source from the node's index
  uint32_t z_nodes, y_nodes, nface, nface_pad, nitems;  // face nodes in the z planes, then the y rows; all; padded
  uint32_t pair_begin;             // first pair's node: the last even index not above plane 1
  uint64_t m_nx, m_plane, m_yrow, m_ny2;
};

// pairs: the lattice runs node pairs (16-bit tiers, pair_kernels_apply); all_nodes: every node by
// the general path (16-bit lattices whose plan the pair form does not take)
__device__ inline void resident_geometry(const StepPlan& p, bool pairs, bool all_nodes, ResidentGeometry& g) {
  const uint32_t nx = p.nx, ny = p.ny, nz = p.nz;
  const uint32_t plane = nx * ny;
  const uint32_t yi = ny - 2, zi = nz - 2;  // every axis has at least two nodes
  g.z_nodes = 2 * plane;
  g.y_nodes = 2 * nx * zi;
  g.nface = all_nodes ? uint32_t(p.ncell) : g.z_nodes + g.y_nodes + 2 * yi * zi;
  g.nface_pad = (g.nface + 31u) & ~31u;
  g.pair_begin = plane & ~1u;
  const uint32_t inner = !pairs || zi == 0 ? 0 : (uint32_t(p.ncell) - plane - g.pair_begin + 1) / 2;
  g.nitems = g.nface_pad + inner;
  g.m_nx = res_magic(nx);
  g.m_plane = res_magic(plane);
  g.m_yrow = res_magic(2 * nx);
  g.m_ny2 = res_magic(2 * yi);
  Unroll<0, Q>::run([&]<int I>() {
    constexpr int ex = D3Q19::ex[I], ey = D3Q19::ey[I], ez = D3Q19::ez[I];
    g.off[I] = int(I * p.stride) - ((ez * int(ny) + ey) * int(nx) + ex);
  });
}

// The i-th face node: the planes z = 0 and nz - 1, then the rows y = 0 and ny - 1 of each inner
// plane, then x = nx - 1 and 0 of each inner row (neighbours in memory side by side).
__device__ __forceinline__ void resident_face_node(const StepPlan& p, const ResidentGeometry& g, uint32_t i, int& x,
                                                   int& y, int& z) {
  const uint32_t nx = p.nx;
  if (i < g.z_nodes) {
    const uint32_t plane = nx * uint32_t(p.ny);
    const bool last = i >= plane;
    if (last) i -= plane;
    z = last ? p.nz - 1 : 0;
    y = int(res_div(i, g.m_nx));
    x = int(i - uint32_t(y) * nx);
    return;
  }
  i -= g.z_nodes;
  if (i < g.y_nodes) {
    const uint32_t k = res_div(i, g.m_yrow), r = i - k * 2 * nx;
    z = int(k) + 1;
    y = r >= nx ? p.ny - 1 : 0;
    x = int(r >= nx ? r - nx : r);
    return;
  }
  i -= g.y_nodes;
  const uint32_t k = res_div(i, g.m_ny2), r = i - k * 2 * uint32_t(p.ny - 2);
  z = int(k) + 1;
  y = int(r >> 1) + 1;
  x = (r & 1) ? p.nx - 1 : 0;
}

struct ResidentNode {
  int x, y, z;
  uint32_t idx;
  int8_t flag;
};

// The node of face item i (every_node: of all nodes), and its stored values by the general gather.
template <typename S, bool WALLS>
__device__ __forceinline__ void resident_face(const S* fin, const int8_t* __restrict__ flags, const StepPlan& p,
                                              const ResidentGeometry& g, bool walls, bool every_node, uint32_t i,
                                              ResidentNode& it, S (&raw)[Q]) {
  if (every_node) {
    it.z = int(res_div(i, g.m_plane));
    const uint32_t rem = i - uint32_t(it.z) * uint32_t(p.nx) * uint32_t(p.ny);
    it.y = int(res_div(rem, g.m_nx));
    it.x = int(rem - uint32_t(it.y) * uint32_t(p.nx));
  } else {
    resident_face_node(p, g, i, it.x, it.y, it.z);
  }
  it.idx = (uint32_t(it.z) * uint32_t(p.ny) + uint32_t(it.y)) * uint32_t(p.nx) + uint32_t(it.x);
  it.flag = flags[it.idx];
  node_pull<S, WALLS, LOAD_LIVE, false>(fin, flags, p, it.x, it.y, it.z, it.idx, raw, walls);
}

// The update and store of a fetched node (a wall node keeps its scratch).
template <typename S, typename R, bool STRICT, bool WALLS>
__device__ __forceinline__ void resident_finish(const S* fin, S* fout, const StepPlan& p, bool walls,
                                                const ResidentNode& it, const S (&raw)[Q], bool edge) {
  if (WALLS && walls && it.flag == FLAG_WALL) return;
  R v[Q];
  Unroll<0, Q>::run([&]<int I>() { v[I] = load_value<S, R, I>(raw[I], p); });
  node_update<S, R, STRICT, MODE_FUSED, 2, LOAD_LIVE>(v, fin, it.idx, it.x, it.y, it.z, it.flag, p, true, edge);
  store_node<S, R, MODE_FUSED>(v, p, p.seed, it.idx, [&]<int I>(S s) { fout[I * p.stride + it.idx] = s; });
}

// Where a node pulls each direction from, as element offsets over all planes: node_pull with its
// bounces decided (they depend on the faces and the flags alone).
template <bool WALLS>
__device__ __forceinline__ void resident_sources(const int8_t* __restrict__ flags, const StepPlan& p, bool walls,
                                                 const ResidentNode& it, int (&src)[Q]) {
  const bool near = WALLS && walls && p.nearwall[it.idx] == 1;
  Unroll<0, Q>::run([&]<int I>() {
    constexpr int ex = D3Q19::ex[I], ey = D3Q19::ey[I], ez = D3Q19::ez[I], O = D3Q19::opp(I);
    int sx = it.x - ex, sy = it.y - ey, sz = it.z - ez;
    bool bounce = false;
    if (sx < 0 || sx >= p.nx) { if (p.periodic[0]) sx = sx < 0 ? sx + p.nx : sx - p.nx; else bounce = true; }
    if (sy < 0 || sy >= p.ny) { if (p.periodic[1]) sy = sy < 0 ? sy + p.ny : sy - p.ny; else bounce = true; }
    if (sz < 0 || sz >= p.nz) { if (p.periodic[2]) sz = sz < 0 ? sz + p.nz : sz - p.nz; else bounce = true; }
    const int n = (sz * p.ny + sy) * p.nx + sx;
    if (I != 0 && near && !bounce) bounce = flags[n] == FLAG_WALL;
    src[I] = bounce ? O * int(p.stride) + int(it.idx) : I * int(p.stride) + n;
  });
}

// The pair (n, n + 1), n even, of a 16-bit tier: the nodes off the faces.
template <typename S, bool WALLS>
__device__ __forceinline__ void resident_pair(const S* fin, S* fout, const int8_t* __restrict__ flags,
                                              const StepPlan& p, const ResidentGeometry& g, bool walls, uint32_t n) {
  const int z = int(res_div(n, g.m_plane));
  const uint32_t rem = n - uint32_t(z) * uint32_t(p.nx) * uint32_t(p.ny);
  const int y = int(res_div(rem, g.m_nx));
  const int x = int(rem - uint32_t(y) * uint32_t(p.nx));
  if (y == 0 && x + 1 < p.nx) return;  // both nodes on a y face
  // the second node is in the same row unless the first is a row's last, i.e. on a face itself
  bool a = x >= 1 && x <= p.nx - 2 && y >= 1 && y <= p.ny - 2 && z >= 1 && z <= p.nz - 2;
  bool b = x + 1 <= p.nx - 2 && y >= 1 && y <= p.ny - 2 && z >= 1 && z <= p.nz - 2;
  if (!a && !b) return;
  const uint32_t* words = reinterpret_cast<const uint32_t*>(fin);
  uint32_t w[Q];
  Unroll<0, Q>::run([&]<int I>() {
    const int e = g.off[I] + int(n);  // planes start at even elements, so parity is the offset's
    const uint32_t w0 = ld_pop<LOAD_LIVE>(words + (e >> 1));
    w[I] = (e & 1) ? __byte_perm(w0, ld_pop<LOAD_LIVE>(words + (e >> 1) + 1), 0x5432) : w0;
  });
  const unsigned short fl = __ldg(reinterpret_cast<const unsigned short*>(flags + n));
  const int8_t fa = int8_t(fl & 0xff), fb = int8_t(fl >> 8);
  if constexpr (WALLS) {
    if (walls) {
      const unsigned short near = __ldg(reinterpret_cast<const unsigned short*>(p.nearwall + n));
      S raw[Q];
      if (a && (near & 0xff) == 1) {
        node_pull<S, true, LOAD_LIVE, false>(fin, flags, p, x, y, z, n, raw, true);
        Unroll<0, Q>::run([&]<int I>() { w[I] = (w[I] & 0xffff0000u) | uint32_t(PackedChunk<S, 2>::bits(raw[I])); });
      }
      if (b && (near >> 8) == 1) {
        node_pull<S, true, LOAD_LIVE, false>(fin, flags, p, x + 1, y, z, n + 1, raw, true);
        Unroll<0, Q>::run([&]<int I>() { w[I] = (w[I] & 0xffffu) | uint32_t(PackedChunk<S, 2>::bits(raw[I])) << 16; });
      }
    }
  }
  float2 v[Q];
  Unroll<0, Q>::run([&]<int I>() { v[I] = unpack2<S>(w[I]); });
  pair_update<S, MODE_FUSED, 2>(v, p, fa, fb);
  uint32_t h = 0, h2 = 0;
  if (p.rounding) {
    h = node_hash(n, p.seed);
    h2 = second_hash(h);
  }
  if (a && b)
    pack_pair<S>(v, p.rounding != 0, h, h2,
                 [&]<int I>(uint32_t r) { *reinterpret_cast<uint32_t*>(fout + I * p.stride + n) = r; });
  else
    pack_pair<S>(v, p.rounding != 0, h, h2, [&]<int I>(uint32_t r) {
      reinterpret_cast<unsigned short*>(fout + I * p.stride + n)[a ? 0 : 1] = (unsigned short)(a ? r & 0xffffu : r >> 16);
    });
}

template <typename S, typename R, bool STRICT, bool WALLS>
__global__ void __launch_bounds__(RES_THREADS, 1)
    k_step_resident(const LatticeDesc* __restrict__ desc, int nsteps, int parity, uint32_t seed, unsigned* left,
                    unsigned* bar, int* err, long long wait_limit) {
  __shared__ StepPlan p;
  __shared__ ResidentGeometry g;
  __shared__ int bail;
  const LatticeDesc L = *desc;
  const uint32_t* from = reinterpret_cast<const uint32_t*>(L.plan);
  uint32_t* to = reinterpret_cast<uint32_t*>(&p);
  for (int w = threadIdx.x; w < int(sizeof(StepPlan) / 4); w += blockDim.x) to[w] = from[w];
  __syncthreads();
  const bool pairs = is_16bit<S>() && p.nsets == 0 && (!p.wall_flags || p.walls);
  if (threadIdx.x == 0) {
    bail = 0;
    resident_geometry(p, pairs, is_16bit<S>() && !pairs, g);
    p.seed = seed;
  }
  __syncthreads();
  const bool walls = WALLS && p.walls;
  const uint32_t nthreads = gridDim.x * blockDim.x;
  const uint32_t me = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
  const int cur0 = L.cur ^ parity;
  auto step_done = [&](int k) {  // false when the launch gives up
    if (k + 1 == nsteps) return true;
    if (!group_barrier(bar, gridDim.x * unsigned(k + 1), wait_limit, err, &bail)) return false;
    if (threadIdx.x == 0) p.seed++;
    __syncthreads();
    return true;
  };
  bool ok = true;
  if (uint32_t(p.ncell) <= nthreads) {
    // one node per thread for the whole launch: where it pulls from stays in registers
    ResidentNode it;
    int src[Q];
    S raw[Q];
    const bool live = me < uint32_t(p.ncell);
    bool edge = false;
    if (live) {
      it.idx = me;
      it.z = int(res_div(me, g.m_plane));
      const uint32_t rem = me - uint32_t(it.z) * uint32_t(p.nx) * uint32_t(p.ny);
      it.y = int(res_div(rem, g.m_nx));
      it.x = int(rem - uint32_t(it.y) * uint32_t(p.nx));
      it.flag = L.flags[me];
      resident_sources<WALLS>(L.flags, p, walls, it, src);
      edge = on_op_face(p, it.x, it.y, it.z);
    }
    for (int k = 0; k < nsteps && ok; k++) {
      const S* fin = static_cast<const S*>(L.f[cur0 ^ (k & 1)]);
      S* fout = static_cast<S*>(L.f[cur0 ^ (k & 1) ^ 1]);
      if (live) {
        Unroll<0, Q>::run([&]<int I>() { raw[I] = ld_pop<LOAD_LIVE>(fin + src[I]); });
        resident_finish<S, R, STRICT, WALLS>(fin, fout, p, walls, it, raw, edge);
      }
      ok = step_done(k);
    }
  } else if constexpr (is_16bit<S>()) {
    for (int k = 0; k < nsteps && ok; k++) {
      const S* fin = static_cast<const S*>(L.f[cur0 ^ (k & 1)]);
      S* fout = static_cast<S*>(L.f[cur0 ^ (k & 1) ^ 1]);
      uint32_t i = me;
      for (; i < g.nface_pad; i += nthreads) {
        if (i >= g.nface) continue;
        ResidentNode it;
        S raw[Q];
        resident_face<S, WALLS>(fin, L.flags, p, g, walls, !pairs, i, it, raw);
        resident_finish<S, R, STRICT, WALLS>(fin, fout, p, walls, it, raw, on_op_face(p, it.x, it.y, it.z));
      }
      for (; i < g.nitems; i += nthreads)
        resident_pair<S, WALLS>(fin, fout, L.flags, p, g, walls, g.pair_begin + 2 * (i - g.nface_pad));
      ok = step_done(k);
    }
  }
  group_leave(left, bar);
}

template <typename S, typename R, bool STRICT>
cudaError_t launch_resident(const ResidentArgs& a, int walls, cudaStream_t s) {
  ResidentArgs c = a;
  void* args[] = {&c.desc, &c.nsteps, &c.parity, &c.seed, &c.left, &c.bar, &c.err, &c.wait_limit};
  const void* kern = walls ? (const void*)k_step_resident<S, R, STRICT, true> : (const void*)k_step_resident<S, R, STRICT, false>;
  return cudaLaunchCooperativeKernel(kern, dim3(c.grid), dim3(c.threads), args, 0, s);
}

// one entry per precision tier (defined in resident_*.cu)
cudaError_t resident_f64_strict(const ResidentArgs& a, int walls, cudaStream_t s);
cudaError_t resident_f64(const ResidentArgs& a, int walls, cudaStream_t s);
cudaError_t resident_f32(const ResidentArgs& a, int walls, cudaStream_t s);
cudaError_t resident_f16(const ResidentArgs& a, int walls, cudaStream_t s);
cudaError_t resident_bf16(const ResidentArgs& a, int walls, cudaStream_t s);

}  // namespace hlbm
