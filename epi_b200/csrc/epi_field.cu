// Cell maps and external-stimulus diffusion, FP64: the rest of the
// reference's per-step loop before its chemistry (epi5_MT/proc.cpp:152-157).
//
// Per tissue, on an (nx+1) x (ny+1) x (nz+1) grid (z fastest, the layout of
// FArr3D, define.h:243), three kernels:
//   k_field_begin    both maps cleared; calc_zzmax (proc.cpp:34-43): highest
//                    DEAD / ALIVE / MUSUME / FIX cell
//   k_field_stamp    setup_map_lat (map.cpp:24-167): every cell marks the
//                    grid points inside its radius in cmap1 and, for ALIVE /
//                    FIX / MUSUME, inside FAC_MAP times its radius in cmap2.
//                    Where spheres overlap the reference (in index order)
//                    keeps the highest-index cell; atomicMax on index + 1
//                    gives the same answer in any order. Points of the first
//                    x and y planes are marked in the periodic copies
//                    (map.cpp:156-166) too.
//   k_ext_stim       calc_ext_stim (ext_stim.cpp:18-69): 7-point diffusion
//                    with cmap2 as the conductance mask and the cornification
//                    source fB, below the z bound, periodic copies included;
//                    evaluated with the reference's operation order and no
//                    fused multiply-adds, so results are bit-identical.
// A step of the 36,864-particle tissue on 129 x 129 x 65 points took nine
// kernels and 95 us (the stamp alone 59, walking every column of the widest
// window), now 35.5.
#include "epi_kernels.h"

#include <algorithm>

#include "epi_device.cuh"

namespace epi {
namespace {

constexpr double kRad = 1.4;          // Rad, map.cpp:26
constexpr double kFacMap = 2.0;       // FAC_MAP, define.h:184
constexpr double kRMax = 1.4;         // R_max, define.h:116
constexpr double kDtCa = 0.01;        // DT_Ca, define.h:89
constexpr double kDB = 0.0009;        // DB, ext_stim.cpp:20
constexpr double kKb = 0.025;         // kb, ext_stim.cpp:10
constexpr double kDurAlive = 0.5;     // ext_stim.cpp:11
constexpr double kDurDead = 2.0;      // ext_stim.cpp:12
constexpr double kThreshDead = 22.0;  // THRESH_DEAD, define.h:156

__device__ __forceinline__ int64_t fidx(const FieldDev& F, int32_t a, int32_t b, int32_t c) {
  return F.base + ((int64_t)a * (F.ny + 1) + b) * (F.nz + 1) + c;
}

__device__ __forceinline__ bool afm_state(uint32_t s) {
  return s == ST_ALIVE || s == ST_FIX || s == ST_MUSUME;
}

// zzmax of every tissue: the z of its qualifying cells folded in with
// atomicMax on the bit patterns (non-negative doubles order like their
// bits; zzmax starts at 0), so the result does not depend on the order.
// Lanes of a warp holding the same tissue first fold their values with
// shuffles, so one atomic per (warp, tissue) run reaches memory. The maps are
// cleared 16 bytes at a time (their arrays start 256-byte aligned).
__global__ void __launch_bounds__(256) k_field_begin(DevState S, FieldState FS) {
  {
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const int64_t n1 = FS.nvox / 4, n2 = FS.nvox / 16;
    GRID_STRIDE(v, 0, n1) reinterpret_cast<uint4*>(FS.cmap1)[v] = zero;
    GRID_STRIDE(v, 0, n2) reinterpret_cast<uint4*>(FS.cmap2)[v] = zero;
    GRID_STRIDE(v, 4 * n1, FS.nvox) FS.cmap1[v] = 0;
    GRID_STRIDE(v, 16 * n2, FS.nvox) FS.cmap2[v] = 0;
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t base0 = (int64_t)blockIdx.x * blockDim.x;
  for (int64_t base = base0; base < S.n_total; base += stride) {
    const int64_t i = base + threadIdx.x;
    int32_t t = -1;
    unsigned long long z = 0;
    if (i < S.n_total) {
      const uint32_t a = S.attr[i];
      const uint32_t st = attr_state(a);
      t = attr_tissue(a);
      if (st == ST_DEAD || st == ST_ALIVE || st == ST_MUSUME || st == ST_FIX) {
        const double zd = S.pos_cur[i].z;
        if (zd > 0.0) z = (unsigned long long)__double_as_longlong(zd);
      }
    }
    const int lane = threadIdx.x & 31;
    // same-tissue lanes form contiguous runs (particles are grouped by tissue)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long zo = __shfl_down_sync(0xffffffffu, z, o);
      const int32_t to = __shfl_down_sync(0xffffffffu, t, o);
      if (lane + o < 32 && to == t && zo > z) z = zo;
    }
    const int32_t tprev = __shfl_up_sync(0xffffffffu, t, 1);
    if (t >= 0 && z > 0 && (lane == 0 || tprev != t))
      atomicMax(reinterpret_cast<unsigned long long*>(&FS.zzmax[t]), z);
  }
}

// The diffusion's z bound of a tissue, (int)((zzmax + FAC_MAP R_max) inv_dz)
// (ext_stim.cpp:22).
__device__ __forceinline__ int32_t field_bound(const FieldDev& F, double zz) {
  return (int32_t)(__dmul_rn(__dadd_rn(zz, kFacMap * kRMax), F.inv_dz));
}

// set_lattice and the two branches of setup_map_lat: kStampLanes lanes per
// particle share the (x, y) columns of its window, each walking its column's
// z. The window is the reference's (lat +- ir, twice that for ALIVE / FIX /
// MUSUME), cut to the points its sphere can reach (at unit density 36 of 81
// columns, 6 of 9 heights); the exact tests decide.
constexpr int kStampLanes = 8;
__global__ void __launch_bounds__(256) k_field_stamp(DevState S, FieldState FS) {
  pdl_entry();
  const int sub = (int)threadIdx.x & (kStampLanes - 1);
  const int64_t groups = (int64_t)gridDim.x * blockDim.x / kStampLanes;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kStampLanes; i < S.n_total;
       i += groups) {
    const uint32_t a = S.attr[i];
    const int32_t t = attr_tissue(a);
    const TissueDev& T = S.tissues[t];
    const FieldDev& F = FS.fd[t];
    const double4 p = S.pos_cur[i];
    const int32_t lat0 = ((int32_t)(p.x * F.inv_dx) + F.nx) % F.nx;
    const int32_t lat1 = ((int32_t)(p.y * F.inv_dy) + F.ny) % F.ny;
    const int32_t lat2 = ((int32_t)(p.z * F.inv_dz) + F.nz) % F.nz;
    const bool afm = afm_state(attr_state(a));
    const int32_t rx = afm ? 2 * F.irx : F.irx, ry = afm ? 2 * F.iry : F.iry;
    const int32_t rz = afm ? 2 * F.irz : F.irz;
    const double normal_radSq = __dmul_rn(p.w, p.w);
    const double crad = __dmul_rn(kFacMap, p.w);
    const double cradSq = __dmul_rn(crad, crad);
    const double reach = afm ? crad : p.w, reachSq = afm ? cradSq : normal_radSq;
    // grid points a distance below reach away lie within `reach / d` of the
    // coordinate in grid units; lat is the coordinate's floor (modulo the
    // grid), so they lie from lat - g to lat + 1 + g, g = floor(reach / d)
    // (one more for rounding)
    auto cut = [&](int32_t r, double inv) {
      const double g = reach * inv;
      return g < (double)r ? (int32_t)g + 1 : r;
    };
    const int32_t gx = cut(rx, F.inv_dx), gy = cut(ry, F.inv_dy), gz = cut(rz, F.inv_dz);
    const int32_t x0 = lat0 - gx, nxc = (gx + 1 < rx ? gx + 1 : rx) + gx + 1;
    const int32_t y0 = lat1 - gy, nyc = (gy + 1 < ry ? gy + 1 : ry) + gy + 1;
    const int32_t z_b = lat2 - gz, z_u = lat2 + (gz + 1 < rz ? gz + 1 : rz);
    const int32_t zmin = z_b >= 1 ? z_b : 1;
    const int32_t zmax = z_u < F.nz ? z_u : F.nz - 1;
    const int32_t mark = (int32_t)i - T.pbase + 1;
    for (int32_t c = sub; c < nxc * nyc; c += kStampLanes) {
      const int32_t ox = c / nyc, oy = c - ox * nyc;
      const int32_t kx = x0 + ox, ky = y0 + oy;
      const double diffx = pdiff(__dmul_rn((double)kx, F.dx), p.x, T.lx);
      const double diffy = pdiff(__dmul_rn((double)ky, F.dy), p.y, T.ly);
      const double tmps = __dadd_rn(__dmul_rn(diffx, diffx), __dmul_rn(diffy, diffy));
      if (!(tmps < reachSq)) continue;  // (the heights only add to it)
      // the window does not wrap onto itself: at most one box off
      const int32_t ipx = kx < 0 ? kx + F.nx : (kx >= F.nx ? kx - F.nx : kx);
      const int32_t ipy = ky < 0 ? ky + F.ny : (ky >= F.ny ? ky - F.ny : ky);
      const int64_t v0 = fidx(F, ipx, ipy, 0);
      // the periodic copies of the first planes
      const int64_t copy_y = ipy == 0 ? (int64_t)F.ny * (F.nz + 1) : 0;
      const int64_t copy_x = ipx == 0 ? (int64_t)F.nx * (F.ny + 1) * (F.nz + 1) : 0;
      for (int32_t mz = zmin; mz <= zmax; ++mz) {
        const double diffz = __dsub_rn(__dmul_rn((double)mz, F.dz), p.z);
        const double distSq = __dadd_rn(tmps, __dmul_rn(diffz, diffz));
        if (!(distSq < reachSq)) continue;
        const bool in = distSq < normal_radSq;
        auto put = [&](int64_t v) {
          if (afm) FS.cmap2[v] = 1;
          if (in) atomicMax(&FS.cmap1[v], mark);
        };
        const int64_t v = v0 + mz;
        put(v);
        if (copy_y) put(v + copy_y);
        if (copy_x) put(v + copy_x);
        if (copy_x && copy_y) put(v + copy_x + copy_y);
      }
    }
  }
}

// fB, ext_stim.cpp:8-16
__device__ __forceinline__ double source_fB(double age, double B, bool cornif) {
  const bool on = cornif && age > kThreshDead - kDurAlive && age <= kThreshDead + kDurDead;
  return __dsub_rn(on ? 1.0 : 0.0, __dmul_rn(kKb, B));
}

// calc_ext_stim's update, one thread per grid point below the z bound, and the
// periodic copies (ext_stim.cpp:63-66) of the first planes. blockIdx.y =
// tissue.
template <typename Index>
__global__ void __launch_bounds__(256) k_ext_stim(DevState S, FieldState FS) {
  pdl_entry();
  const int32_t t = blockIdx.y;
  const TissueDev& T = S.tissues[t];
  const FieldDev& F = FS.fd[t];
  const int32_t bound = field_bound(F, FS.zzmax[t]);
  // beyond the grid the reference would read outside its arrays
  if (bound > F.nz && blockIdx.x == 0 && threadIdx.x == 0)
    raise_error(S.status, E_UNSUPPORTED, T.pbase, -1, FS.zzmax[t]);
  const int32_t izb = bound > F.nz ? F.nz : bound;
  if (izb <= 0) return;
  const Index m = (Index)F.nx * (Index)F.ny * (Index)izb;
  for (Index e = (Index)blockIdx.x * blockDim.x + threadIdx.x; e < m;
       e += (Index)gridDim.x * blockDim.x) {
    const Index r = e / (Index)izb;
    const int32_t l = (int32_t)(e - r * (Index)izb);
    const int32_t j = (int32_t)(r / (Index)F.ny), k = (int32_t)(r - (Index)j * (Index)F.ny);
    const int32_t px = j == 0 ? F.nx - 1 : j - 1, nx = j + 1 == F.nx ? 0 : j + 1;
    const int32_t py = k == 0 ? F.ny - 1 : k - 1, ny = k + 1 == F.ny ? 0 : k + 1;
    const int32_t pz = l == 0 ? 1 : l - 1, nz = l + 1 == F.nz ? F.nz - 1 : l + 1;
    const double* c = FS.cur;
    const int64_t v = fidx(F, j, k, l);
    const double cext = c[v];
    auto term = [&](int64_t w) {
      return __dmul_rn((double)FS.cmap2[w], __dsub_rn(c[w], cext));
    };
    double sum = term(fidx(F, px, k, l));
    sum = __dadd_rn(sum, term(fidx(F, j, py, l)));
    sum = __dadd_rn(sum, term(fidx(F, j, k, pz)));
    sum = __dadd_rn(sum, term(fidx(F, j, k, nz)));
    sum = __dadd_rn(sum, term(fidx(F, j, ny, l)));
    sum = __dadd_rn(sum, term(fidx(F, nx, k, l)));
    double age = 0.0;
    bool cornif = false;
    const int32_t cm = FS.cmap1[v] - 1;
    if (cm >= 0) {
      const int32_t ci = T.pbase + cm;
      const uint32_t st = attr_state(S.attr[ci]);
      if (st == ST_DEAD || st == ST_ALIVE) {
        age = FS.agek[ci];
        cornif = true;
      }
    }
    const double diff = __dmul_rn(__dmul_rn(__dmul_rn(kDB, sum), F.inv_dz), F.inv_dz);
    const double next =
        __dadd_rn(cext, __dmul_rn(kDtCa, __dadd_rn(diff, source_fB(age, cext, cornif))));
    FS.nxt[v] = next;
    if (k == 0) FS.nxt[fidx(F, j, F.ny, l)] = next;
    if (j == 0) FS.nxt[fidx(F, F.nx, k, l)] = next;
    if (j == 0 && k == 0) FS.nxt[fidx(F, F.nx, F.ny, l)] = next;
  }
}

}  // namespace

void field_params(FieldDev& F, double lx, double ly, double lz, int32_t nx, int32_t ny,
                  int32_t nz) {
  F.nx = nx;
  F.ny = ny;
  F.nz = nz;
  // cdefd dx = LX / NX; inv_dx = NX / LX (define.h:111-113)
  F.dx = lx / (double)nx;
  F.dy = ly / (double)ny;
  F.dz = lz / (double)nz;
  F.inv_dx = (double)nx / lx;
  F.inv_dy = (double)ny / ly;
  F.inv_dz = (double)nz / lz;
  // irx = (int)(Rad * NX / LX), map.cpp:28-30
  F.irx = (int32_t)(kRad * (double)nx / lx);
  F.iry = (int32_t)(kRad * (double)ny / ly);
  F.irz = (int32_t)(kRad * (double)nz / lz);
}

void launch_field_step(const DevState& S, const FieldState& FS, const LaunchCfg& lc,
                       cudaStream_t s) {
  const int nt = S.ntissues;
  const int grid = lc.num_sms * 8;
  cudaMemsetAsync(FS.zzmax, 0, sizeof(double) * nt, s);
  k_field_begin<<<grid, 256, 0, s>>>(S, FS);
  if (S.n_total > 0)
    launch_pdl(k_field_stamp, stride_blocks(S.n_total * kStampLanes, 256, lc), 256, s, S, FS);
  // enough blocks for the batch, spread over its tissues; 32-bit index
  // arithmetic whenever a tissue's points and a stride fit
  const dim3 g((unsigned)std::max(grid / std::max(nt, 1), 1) + 1, (unsigned)nt);
  const int64_t stride = (int64_t)g.x * 256;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = g;
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (FS.nvox / std::max(nt, 1) + stride < (int64_t)UINT32_MAX)
    cudaLaunchKernelEx(&cfg, k_ext_stim<uint32_t>, S, FS);
  else
    cudaLaunchKernelEx(&cfg, k_ext_stim<uint64_t>, S, FS);
}

}  // namespace epi
