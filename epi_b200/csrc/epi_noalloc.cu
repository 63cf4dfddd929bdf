// connect_cell for one tissue without any device allocation.
//
// Some callers cannot let this library call cudaMalloc: applications whose
// device memory all belongs to another allocator (a framework's caching
// allocator, or a pool sized once at start-up against a fixed memory budget)
// and loops that must not allocate once they run. For them,
// epi_connect_noalloc reads caller-owned device inputs, writes caller-owned
// device outputs, and keeps its working storage in one file-scope device
// array of fixed size. That array exists on every GPU that loads the
// library, from load until process exit.
//
// The scratch holds the bin counts, bin offsets, the sorted particle indices
// of the counting sort and a sorted FP32 copy of positions and radii. It is
// shared by every call on a device and keeps the last call's contents; each
// call clears the counts it uses before binning. Two calls whose work
// overlaps on the GPU (different streams, or different host threads) race on
// it.
#include "epi_mech.h"
#include "epi_common.cuh"

#include <cuda_runtime.h>
#include <cmath>
#include <mutex>

namespace {

using namespace epi;

constexpr int32_t kMaxP = EPI_NOALLOC_MAX_PARTICLES;
constexpr int32_t kMaxB = EPI_NOALLOC_MAX_BINS;
// scratch layout, in int32 words, each part 64-word aligned
constexpr int32_t kOffCounts = 0;
constexpr int32_t kOffStarts = kOffCounts + kMaxB;
constexpr int32_t kOffBin = kOffStarts + ((kMaxB + 1 + 63) / 64) * 64;
constexpr int32_t kOffRank = kOffBin + kMaxP;
constexpr int32_t kOffSorted = kOffRank + kMaxP;
constexpr int32_t kOffCopy = kOffSorted + kMaxP;  // float4 per sorted particle
constexpr int32_t kOffRmax = kOffCopy + 4 * kMaxP;   // bits of the largest FP32 |radius|
constexpr int32_t kScratchWords = kOffRmax + 64;
static_assert(kOffCopy % 4 == 0 && kOffStarts % 4 == 0, "16-byte aligned parts");

static __device__ __align__(256) int32_t g_noalloc_scratch[kScratchWords];

struct Args {
  const double* x;
  const double* y;
  const double* z;
  const double* r;
  int32_t n, nmemb, nmx, nmy;
  double lx, ly, lz, lt;
  int32_t anx, any, anz;
  int32_t max_conn;
  float tol;  // bound on the FP32 error of a separation (see na_connect)
  int32_t* conn;
  int32_t* count;
  int32_t* scratch;  // device address of g_noalloc_scratch
};

constexpr int kThreads = 256;
constexpr int kScanThreads = 1024;

// Clears the bin counts this call uses.
__global__ void na_init(Args A) {
  if (blockIdx.x == 0 && threadIdx.x == 0) A.scratch[kOffRmax] = 0;
  const int32_t nb = A.anx * A.any * A.anz;
  for (int32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x)
    A.scratch[kOffCounts + b] = 0;
}

// grid_init's bin (cell_connection.cpp:44-53); -1 marks the range assert.
// Also the row heads: membrane rows start with their four lattice links in
// the order _memb_init pushes them (cellmanager.cpp:160-163), and the largest
// radius of the particles inside the grid (non-negative floats order like
// their bits; a NaN orders above infinity).
__device__ __forceinline__ uint32_t bin_particle(const Args& A, int32_t i) {
  if (i < A.nmemb) {
    const Lattice L = lattice_of(i, A.nmx, A.nmy);
    int32_t* row = A.conn + (int64_t)i * A.max_conn;
    const int32_t links[4] = {L.l, L.r, L.b, L.u};
    for (int k = 0; k < kMembAdj && k < A.max_conn; ++k) row[k] = links[k];
  }
  const double x = A.x[i], y = A.y[i], z = A.z[i];
  // Coordinates are converted to bin numbers only once they are finite and
  // within a few boxes of the grid, so every conversion is in int32 range.
  const double big = 4.0 * (A.lx + A.ly + A.lz);
  bool bad = !isfinite(x) || !isfinite(y) || !isfinite(z) || fabs(x) > big || fabs(y) > big ||
             fabs(z) > big;
  int32_t aix = 0, aiy = 0, aiz = 0;
  if (!bad) {
    aix = (int32_t)((0.5 * A.lx - pdiff(0.5 * A.lx, x, A.lx)) / kAreaGrid);
    aiy = (int32_t)((0.5 * A.ly - pdiff(0.5 * A.ly, y, A.ly)) / kAreaGrid);
    aiz = (int32_t)(fmax(z, 0.0) / kAreaGrid);
    bad = aix >= A.anx || aiy >= A.any || aiz >= A.anz || aix < 0 || aiy < 0 || aiz < 0;
  }
  if (!bad && i >= A.nmemb) {  // connect_proc's assert for the searching cells (:95-99)
    const int32_t cx = (int32_t)(x / kAreaGrid), cy = (int32_t)(y / kAreaGrid),
                  cz = (int32_t)(z / kAreaGrid);
    bad = cx >= A.anx || cy >= A.any || cz >= A.anz || cx < 0 || cy < 0 || cz < 0;
  }
  // -1: the range assert of grid_init / connect_proc
  A.count[i] = bad ? -1 : (i < A.nmemb ? kMembAdj : 0);
  if (bad) {
    A.scratch[kOffBin + i] = -1;
    return 0u;
  }
  const int32_t b = (aix * A.any + aiy) * A.anz + aiz;
  A.scratch[kOffBin + i] = b;
  A.scratch[kOffRank + i] = atomicAdd(&A.scratch[kOffCounts + b], 1);
  return __float_as_uint(fabsf((float)A.r[i]));
}
__global__ void na_bin(Args A) {
  pdl_entry();
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t rmax = __reduce_max_sync(0xffffffffu, i < A.n ? bin_particle(A, i) : 0u);
  if ((threadIdx.x & 31) == 0 && rmax)
    atomicMax(reinterpret_cast<uint32_t*>(A.scratch + kOffRmax), rmax);
}

// One block: exclusive scan of the bin counts into the bin offsets. 1024
// threads of eight bins each cover 8192 bins per pass (two 16-byte loads and
// stores a thread), so the largest grid takes four passes; the former 256
// bins per pass took 44 us on 16,384 bins, this 6 us.
__global__ void __launch_bounds__(kScanThreads) na_scan(Args A) {
  pdl_entry();
  __shared__ int32_t wsum[kScanThreads / 32];
  const int32_t nb = A.anx * A.any * A.anz;
  const int32_t* in = A.scratch + kOffCounts;
  int32_t* out = A.scratch + kOffStarts;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t carry = 0;
  for (int32_t base = 0; base < nb; base += 8 * kScanThreads) {
    // the count and offset parts hold kMaxB >= nb rounded up to 8 entries
    const int32_t b = base + 8 * (int32_t)threadIdx.x;
    int4 lo = make_int4(0, 0, 0, 0), hi = lo;
    if (b < nb) {
      lo = *reinterpret_cast<const int4*>(in + b);
      hi = *reinterpret_cast<const int4*>(in + b + 4);
    }
    int32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    int32_t sum = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (b + k >= nb) v[k] = 0;
      const int32_t t = v[k];
      v[k] = sum;
      sum += t;
    }
    int32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      int32_t w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    const int32_t run = carry + (wid ? wsum[wid - 1] : 0) + incl - sum;
    if (b < nb) {
      *reinterpret_cast<int4*>(out + b) = make_int4(run + v[0], run + v[1], run + v[2], run + v[3]);
      *reinterpret_cast<int4*>(out + b + 4) =
          make_int4(run + v[4], run + v[5], run + v[6], run + v[7]);
    }
    carry += wsum[kScanThreads / 32 - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[nb] = carry;
}

__global__ void na_scatter(Args A) {
  pdl_entry();
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const int32_t b = A.scratch[kOffBin + i];
  if (b < 0) return;
  const int32_t s = A.scratch[kOffStarts + b] + A.scratch[kOffRank + i];
  A.scratch[kOffSorted + s] = i;
  reinterpret_cast<float4*>(A.scratch + kOffCopy)[s] =
      make_float4((float)A.x[i], (float)A.y[i], (float)A.z[i], (float)A.r[i]);
}

__device__ __forceinline__ void push(const Args& A, int32_t row, int32_t v) {
  const int32_t k = atomicAdd(&A.count[row], 1);
  if (k < A.max_conn) A.conn[(int64_t)row * A.max_conn + k] = v;
}

__device__ __forceinline__ float pdiff_f(float a, float b, float L) {
  const float d = a - b;
  return d > 0.5f * L ? d - L : (d <= -0.5f * L ? d + L : d);
}

// connect_proc (cell_connection.cpp:70-129): every non-membrane cell scans
// the 5x5x5 bins around (int)(x/AREA_GRID) with wrap in x, y and z and
// connects to each lower-index particle within LJ_THRESH*(r_c+r_o),
// pushing each into the other's row.
//
// One warp per cell. The z bins of an (x, y) column are one run of sorted
// slots (two where the window wraps in z). Lane k looks at column k: a column
// farther than R = LJ_THRESH (|r_c| + the largest |r|) in x and y holds no
// partner and is left out, and R cuts the run's z bins too, so of the 25
// columns and about 750 slots of the window some 7 and 110 remain at unit
// density. The kept runs are laid out in shared memory; eight lanes take a
// run, so a warp sweeps four at a time with coalesced loads. A slot costs a
// 16-byte load and an FP32 test that rejects what is certainly out of reach.
// What it passes is held in shared memory until the sweep is done; then the
// lanes read the partners' FP64 data, decide and push all at once, so a warp
// waits for its atomics once and not after every slot.
//
// Both tests only reject. A bin's particles lie in [k AG, (k+1) AG) of the
// grid's coordinate, bin 0 also below it (grid_init truncates towards 0),
// and p_diff's difference is never shorter than the nearest image's. With M
// the bound na_bin puts on coordinates and u = 2^-24, an FP32 separation is
// off by at most 6 M u per axis (two roundings of coordinates, the
// difference, the +-L), so a pair within D = LJ_THRESH |r_c + r_o| has an
// FP32 distance below D + 11 M u; A.tol is 16 M u, and 1e-5 covers the
// relative rounding of sums and squares. NaN passes every test.
//
// Bound by issue and by the latency of a warp's few dependent loads. 36,864
// particles, whole call: 1353 us with a thread per cell testing every slot
// in FP64 through four strided loads, 103 us with this sweep over all 25
// columns, 65 us with the kept ones, 53 us with the partners held (this kernel 39 of them).
constexpr int kRunLanes = 8;
constexpr int kHeld = 64;  // partners a warp holds until its sweep is done
// distance of v from [lo, hi] or its images a box away
__device__ __forceinline__ float gap_f(float v, float lo, float hi, float L) {
  float g = fmaxf(fmaxf(lo - v, v - hi), 0.f);
  g = fminf(g, fmaxf(fmaxf(lo - L - v, v - (hi - L)), 0.f));
  return fminf(g, fmaxf(fmaxf(lo + L - v, v - (hi + L)), 0.f));
}
__global__ void __launch_bounds__(kThreads) na_connect(Args A) {
  pdl_entry();
  __shared__ int2 s_runs[kThreads / 32][50];
  __shared__ int32_t s_list[kThreads / 32][kHeld], s_held[kThreads / 32];
  const int32_t c = A.nmemb + (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (c >= A.n) return;
  if (A.scratch[kOffBin + c] < 0) return;
  int2* runs = s_runs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, sub = lane & (kRunLanes - 1), grp = lane / kRunLanes;
  const double x = A.x[c], y = A.y[c], z = A.z[c], r = A.r[c];
  const float xf = (float)x, yf = (float)y, zf = (float)z, rf = (float)r;
  const float lxf = (float)A.lx, lyf = (float)A.ly, ltf = (float)A.lt * (1.f + 1e-5f);
  const float agf = (float)kAreaGrid;
  const float R = fmaf(ltf, fabsf(rf) + __int_as_float(A.scratch[kOffRmax]), A.tol);
  const int32_t cx = (int32_t)(x / kAreaGrid), cy = (int32_t)(y / kAreaGrid),
                cz = (int32_t)(z / kAreaGrid);
  // z bins [z0, z1] and, where the window wraps (at most on one side:
  // ANZ >= 5), [w0, w1]
  const float tz = R + A.tol;
  int32_t z0 = cz < 2 ? 0 : cz - 2, z1 = cz + 2 < A.anz ? cz + 2 : A.anz - 1;
  while (z0 < cz && zf - (float)(z0 + 1) * agf > tz) ++z0;
  while (z1 > cz && (float)z1 * agf - zf > tz) --z1;
  int32_t w0 = 0, w1 = -1;
  if (cz < 2) {
    if (!((float)(A.anz + cz - 2) * agf - zf > tz)) {
      w0 = A.anz + cz - 2;
      w1 = A.anz - 1;
    }
  } else if (cz + 2 >= A.anz && !(zf - (float)(cz + 3 - A.anz) * agf > tz)) {
    w1 = cz + 2 - A.anz;
  }
  const bool wraps = w1 >= w0;
  const int32_t* starts = A.scratch + kOffStarts;
  const float4* copy = reinterpret_cast<const float4*>(A.scratch + kOffCopy);
  int32_t nruns;
  {
    bool keep = false;
    int2 main = make_int2(0, 0), wrap = main;
    if (lane < 25) {
      int32_t aix = cx - 2 + lane / 5, aiy = cy - 2 + lane % 5;
      aix += aix < 0 ? A.anx : (aix >= A.anx ? -A.anx : 0);
      aiy += aiy < 0 ? A.any : (aiy >= A.any ? -A.any : 0);
      const float gx = gap_f(xf, (float)(aix - (aix == 0)) * agf, (float)(aix + 1) * agf, lxf);
      const float gy = gap_f(yf, (float)(aiy - (aiy == 0)) * agf, (float)(aiy + 1) * agf, lyf);
      keep = !(gx * gx + gy * gy > tz * tz);
      if (keep) {
        const int32_t b = (aix * A.any + aiy) * A.anz;
        main = make_int2(starts[b + z0], starts[b + z1 + 1]);
        if (wraps) wrap = make_int2(starts[b + w0], starts[b + w1 + 1]);
      }
    }
    if (lane == 0) s_held[threadIdx.x >> 5] = 0;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    const int at = __popc(m & ((1u << lane) - 1u));
    nruns = __popc(m);
    if (keep) {
      runs[at] = main;
      if (wraps) runs[nruns + at] = wrap;
    }
    if (wraps) nruns *= 2;
    __syncwarp();
  }
  int32_t* list = s_list[threadIdx.x >> 5];
  int32_t* held = &s_held[threadIdx.x >> 5];
  // the exact predicate, and the pushes of both rows
  auto decide = [&](int32_t o) {
    const double d2 = dist_sq_exact(pdiff(x, A.x[o], A.lx), pdiff(y, A.y[o], A.ly), z - A.z[o]);
    if (connected_pred(d2, A.lt, r, A.r[o])) {
      push(A, c, o);
      push(A, o, c);
    }
  };
  for (int32_t k = grp; k < nruns; k += 32 / kRunLanes) {
    const int2 run = runs[k];
    for (int32_t s = run.x + sub; s < run.y; s += kRunLanes) {
      const float4 q = copy[s];
      const float dx = pdiff_f(xf, q.x, lxf), dy = pdiff_f(yf, q.y, lyf), dz = zf - q.z;
      const float reach = fmaf(ltf, fabsf(rf + q.w), A.tol);
      if (dx * dx + dy * dy + dz * dz > reach * reach) continue;
      const int32_t o = A.scratch[kOffSorted + s];
      if (c <= o) continue;
      const int32_t at = atomicAdd(held, 1);
      if (at < kHeld) list[at] = o;
      else decide(o);
    }
  }
  __syncwarp();
  const int32_t nh = *held < kHeld ? *held : kHeld;
  for (int32_t k = lane; k < nh; k += 32) decide(list[k]);
}

// Each row sorted ascending (the rows' push order depends on thread timing).
// One warp per row: a lane holds one entry and stores it at its rank, the
// number of smaller entries; rows longer than a warp (rare) are sorted in
// place by one lane.
__global__ void __launch_bounds__(kThreads) na_sort_rows(Args A) {
  pdl_entry();
  const int32_t i = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= A.n) return;
  const int lane = threadIdx.x & 31;
  const int32_t c = A.count[i];
  const int32_t m = c < 0 ? 0 : (c < A.max_conn ? c : A.max_conn);
  int32_t* row = A.conn + (int64_t)i * A.max_conn;
  if (m <= 32) {
    const int32_t v = lane < m ? row[lane] : 0x7fffffff;
    int32_t rank = 0;
    for (int k = 0; k < m; ++k) {
      const int32_t o = __shfl_sync(0xffffffffu, v, k);
      rank += (o < v || (o == v && k < lane)) ? 1 : 0;
    }
    if (lane < m) row[rank] = v;
    return;
  }
  if (lane != 0) return;
  for (int32_t s = 1; s < m; ++s) {
    const int32_t v = row[s];
    int32_t k = s - 1;
    while (k >= 0 && row[k] > v) {
      row[k + 1] = row[k];
      --k;
    }
    row[k + 1] = v;
  }
}

// Launches kernel k with `grid` blocks of `block` threads on stream s and
// returns that launch's own status. pdl: the kernel may be scheduled while
// its predecessor (this call's previous kernel) drains; it waits for it in
// pdl_entry().
cudaError_t launch(void (*k)(Args), int grid, int block, bool pdl, cudaStream_t s,
                   const Args& A) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, A);
}

// Device address of the scratch array, looked up once per device.
constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
int32_t* g_scratch_addr[kMaxDevices] = {};

int scratch_of_current_device(int32_t** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return EPI_ERR_NO_DEVICE;
  if (dev < 0 || dev >= kMaxDevices) return EPI_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) return EPI_ERR_CUDA;
    g_scratch_addr[dev] = static_cast<int32_t*>(p);
  }
  *out = g_scratch_addr[dev];
  return EPI_OK;
}

}  // namespace

extern "C" int epi_connect_noalloc(const double* x, const double* y, const double* z,
                                   const double* radius, int32_t n, int32_t nmemb, int32_t nmx,
                                   int32_t nmy, double lx, double ly, double lz,
                                   double lj_thresh, int32_t max_conn, int32_t* conn,
                                   int32_t* count, void* stream) {
  try {
    if (n < 0 || nmemb < 0 || nmemb > n || max_conn < kMembAdj) return EPI_ERR_INVALID_ARG;
    if (n > 0 && (!x || !y || !z || !radius || !conn || !count))
      return EPI_ERR_INVALID_ARG;
    if (!(lx > 0) || !(ly > 0) || !(lz > 0) || !(lj_thresh > 0)) return EPI_ERR_INVALID_ARG;
    if (nmemb != nmx * nmy || (nmemb > 0 && (nmx < 3 || nmy < 3))) return EPI_ERR_UNSUPPORTED;
    Args A;
    A.anx = (int32_t)(lx / 2.0 + 0.5);  // ANX / ANY / ANZ, cell_connection.cpp:22-26
    A.any = (int32_t)(ly / 2.0 + 0.5);
    A.anz = (int32_t)(lz / 2.0);
    // a window of 5 bins that wrapped onto itself would push pairs twice
    if (A.anx < 5 || A.any < 5 || A.anz < 5) return EPI_ERR_UNSUPPORTED;
    // the fixed scratch bounds every call
    if (n > kMaxP || (int64_t)A.anx * A.any * A.anz > kMaxB) return EPI_ERR_INVALID_ARG;
    if (n == 0) return EPI_OK;
    int rc = scratch_of_current_device(&A.scratch);
    if (rc != EPI_OK) return rc;
    A.x = x;
    A.y = y;
    A.z = z;
    A.r = radius;
    A.n = n;
    A.nmemb = nmemb;
    A.nmx = nmx;
    A.nmy = nmy;
    A.lx = lx;
    A.ly = ly;
    A.lz = lz;
    A.lt = lj_thresh;
    A.max_conn = max_conn;
    A.conn = conn;
    A.count = count;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    A.tol = (float)(16.0 * 4.0 * (lx + ly + lz) * std::ldexp(1.0, -24));
    const int nb = A.anx * A.any * A.anz;
    const int per_warp = kThreads / 32;  // rows (cells) of a warp-per-row block
    const int gp = (n + kThreads - 1) / kThreads;
    // Each launch reports its own status, so an error that earlier, unrelated
    // work left pending on this thread is neither reported here nor cleared.
    cudaError_t e = launch(na_init, (nb + kThreads - 1) / kThreads, kThreads, false, s, A);
    if (e == cudaSuccess) e = launch(na_bin, gp, kThreads, true, s, A);
    if (e == cudaSuccess) e = launch(na_scan, 1, kScanThreads, true, s, A);
    if (e == cudaSuccess) e = launch(na_scatter, gp, kThreads, true, s, A);
    if (e == cudaSuccess && n > nmemb)
      e = launch(na_connect, (n - nmemb + per_warp - 1) / per_warp, kThreads, true, s, A);
    if (e == cudaSuccess)
      e = launch(na_sort_rows, (n + per_warp - 1) / per_warp, kThreads, true, s, A);
    return e == cudaSuccess ? EPI_OK : EPI_ERR_CUDA;
  } catch (...) {
    return EPI_ERR_CUDA;
  }
}
