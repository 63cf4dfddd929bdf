// Device helpers shared by the step and adjoint kernels (internal).
#pragma once
#include "epi_kernels.h"

namespace epi {
namespace {

inline int blocks_for(int64_t n, int b) { return (int)((n + b - 1) / b); }
inline int stride_blocks(int64_t n, int b, const LaunchCfg& lc) {
  const int need = blocks_for(n, b);
  const int cap = lc.num_sms * 8;
  return need < cap ? (need > 0 ? need : 1) : cap;
}

// One count per kernel launch (the first thread of the first block).
__device__ __forceinline__ void count_launch(unsigned long long* launches) {
  if (launches && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) atomicAdd(launches, 1ull);
}

template <typename... Params, typename... Args>
void launch_pdl(void (*kernel)(Params...), int grid, int block, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

#define GRID_STRIDE(i, lo, hi) \
  for (int64_t i = (lo) + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (hi); \
       i += (int64_t)gridDim.x * blockDim.x)

// Has a particle of tissue T at (x, y, z) moved skin/2 from b, its position at
// the tissue's last candidate rebuild? (The margin covers the float rounding
// of b; NaN counts as moved.)
__device__ __forceinline__ bool moved_too_far(double skin, const TissueDev& T, double x, double y,
                                              double z, const float4& b) {
  double ex = x - (double)b.x, ey = y - (double)b.y;
  if (ex > T.hlx) ex -= T.lx;
  else if (ex < -T.hlx) ex += T.lx;
  if (ey > T.hly) ey -= T.ly;
  else if (ey < -T.hly) ey += T.ly;
  const double ez = z - (double)b.z;
  const double lim = 0.5 * skin - 1e-3;
  return !(xfma(ez, ez, xfma(ey, ey, xmul(ex, ex))) <= xmul(lim, lim));
}

// Separation of a pair as cell_interaction_apply computes it for its c1
// (:56-58), seen from particle i: the reference adds +d to c1, -d to c2.
__device__ __forceinline__ void pair_sep(const double4& p, const double4& pq, bool i_is_c1,
                                         const TissueDev& T, double& dx, double& dy, double& dz) {
  if (i_is_c1) {
    dx = pdiff(p.x, pq.x, T.lx);
    dy = pdiff(p.y, pq.y, T.ly);
    dz = p.z - pq.z;
  } else {
    dx = -pdiff(pq.x, p.x, T.lx);
    dy = -pdiff(pq.y, p.y, T.ly);
    dz = -(pq.z - p.z);
  }
}

template <typename R>
struct Vec3 {
  R x, y, z;
};
// Offset of a lattice neighbour from the particle (minimum image).
template <typename R>
__device__ __forceinline__ Vec3<R> offset_of(const double4& q, const double4& p,
                                             const TissueDev& T) {
  return Vec3<R>{R(pdiff_h(q.x, p.x, T.lx, T.hlx)), R(pdiff_h(q.y, p.y, T.ly, T.hly)),
                 R(q.z - p.z)};
}
}  // namespace
}  // namespace epi
