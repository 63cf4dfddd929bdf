// Mechanics kernels for sm_100a.
//
// One step of the reference (epi5_MT/proc.cpp:22-32 without state renewal)
// runs as the sequence below (small batches: as phases of one resident kernel,
// epi_resident.cu)
//   [rebuild]  Verlet candidate rebuild of the tissues that need one
//              (bin -> scan -> scatter -> per-bin sort -> candidate search);
//              every kernel of it exits at once when no tissue does
//   k_memb_force  bending, lattice springs and wall of the membrane
//              (_memb_bend_calc1..3, tri_memb_bend, _MEMB_interaction)
//   k_dermis   the dermis of FIX / MUSUME cells (find_dermis)
//   k_step     connect_proc's exact predicate over the candidates, every
//              force of cell_interaction, pos_copy and the periodic wrap,
//              fused; flags tissues whose particles moved more than skin/2
//              since their last rebuild
//
// The reference rebuilds its connection lists from scratch every step
// (connect_cell, cell_connection.cpp:191-203). Here a tissue's candidate list
// holds every partner within LJ_THRESH*(r_i+r_j) + skin at the last rebuild;
// while no particle has moved more than skin/2 since, every pair that can
// satisfy the reference's predicate is a candidate, and k_step evaluates that
// predicate exactly (same rounding as the reference) on the current
// positions. The connection set of every step is therefore the reference's.
//
// Forces are gathered, not scattered: each particle sums every interaction it
// takes part in (the reference adds +d to c1 and -d to c2 with CAS atomics,
// cell_interaction.cpp:48-66). No atomics touch positions, so a step is
// deterministic and repeatable bit for bit.
#include "epi_kernels.h"

#include <algorithm>

#include "epi_device.cuh"
#include "epi_rebuild.cuh"
#include "epi_step.cuh"

namespace epi {

const char* const kKernelClassNames[KC_COUNT] = {
    "step", "prepass", "rebuild_bin", "rebuild_scan", "rebuild_sort", "rebuild_search", "gate"};

namespace {

// ---------------------------------------------------------------------------
// Scan (reduce -> top-level scan -> down-sweep). No inter-block waiting.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool closed(const int32_t* gate) { return gate && *gate == 0; }

__global__ void k_scan_partial(const int32_t* __restrict__ in, int32_t n,
                               int32_t* __restrict__ partial, const int32_t* gate) {
  if (closed(gate)) return;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += in[base + k];
  int32_t tot;
  block_excl_scan<kScanThreads>(s, &tot);
  if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

__global__ void k_set1(int32_t* out, int32_t v, const int32_t* gate) {
  if (closed(gate)) return;
  *out = v;
}

__global__ void k_scan_top(int32_t* partial, int32_t nb, const int32_t* gate) {
  if (closed(gate)) return;
  int32_t carry = 0;
  for (int32_t base = 0; base < nb; base += kScanThreads) {
    const int32_t i = base + threadIdx.x;
    const int32_t v = i < nb ? partial[i] : 0;
    int32_t tot;
    const int32_t ex = block_excl_scan<kScanThreads>(v, &tot);
    if (i < nb) partial[i] = carry + ex;
    carry += tot;
  }
}

__global__ void k_scan_final(const int32_t* __restrict__ in, int32_t* __restrict__ out,
                             int32_t n, const int32_t* __restrict__ partial, int32_t init,
                             const int32_t* gate) {
  if (closed(gate)) return;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int32_t v[kScanItems];
  int32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    s += v[k];
  }
  int32_t tot;
  int32_t run = block_excl_scan<kScanThreads>(s, &tot) + partial[blockIdx.x] + init;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) out[n] = run;
}

__global__ void k_gate_compact(DevState S, int32_t t0, int32_t t1) {
  pdl_entry();
  count_launch(S.launches);
  gate_compact<kScanThreads>(S, t0, t1, S.gate[0] != 0, t0 == 0 && t1 == S.ntissues);
}

__global__ void k_bin(DevState S) {
  pdl_entry();
  count_launch(S.launches);
  rebuild_bin(S);
}

constexpr int kTissueScanThreads = 1024;
__global__ void __launch_bounds__(kTissueScanThreads) k_scan_tissue(DevState S) {
  pdl_entry();
  count_launch(S.launches);
  rebuild_scan<kTissueScanThreads>(S);
}

__global__ void k_scatter(DevState S) {
  pdl_entry();
  count_launch(S.launches);
  rebuild_scatter(S);
}

__global__ void k_binsort(DevState S) {
  pdl_entry();
  count_launch(S.launches);
  rebuild_sort(S);
}

template <bool k16>
__global__ void __launch_bounds__(256, 4) k_cand_search(DevState S, int32_t thread_from) {
  pdl_entry();
  count_launch(S.launches);
  rebuild_search<k16>(S, thread_from);
}

// Condition of the rebuild node in the captured step graph: builds the work
// list of [t0, t1) (as k_gate_compact) and runs the rebuild kernels only
// when it is not empty.
__global__ void k_rebuild_condition(DevState S, int32_t t0, int32_t t1,
                                    cudaGraphConditionalHandle h) {
  pdl_entry();
  count_launch(S.launches);
  gate_compact<kScanThreads>(S, t0, t1, S.gate[0] != 0, t0 == 0 && t1 == S.ntissues);
  __syncthreads();
  if (threadIdx.x == 0) cudaGraphSetConditional(h, S.rl_count[0] > 0 ? 1u : 0u);
}

__global__ void k_gate_set_all(DevState S, int32_t ntissues) {
  GRID_STRIDE(t, 0, ntissues) S.gate[1 + t] = 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) S.gate[0] = 1;
}

// ---------------------------------------------------------------------------
// find_dermis for the FIX / MUSUME cells in prep[f0, f1), from the current
// positions, one warp per cell: 64 all-states tissues (640 such cells) took
// 68 us with a thread per cell, 128 take 8.
// ---------------------------------------------------------------------------
__global__ void k_dermis(DevState S, int32_t f0, int32_t f1) {
  pdl_entry();
  count_launch(S.launches);
  const int lane = threadIdx.x & 31;
  const int32_t warps = (int32_t)((gridDim.x * blockDim.x) >> 5);
  for (int32_t e = f0 + (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); e < f1; e += warps)
    dermis_cell(S, S.prep[e], lane);
}

// ---------------------------------------------------------------------------
// Step: cell_interaction (cell_interaction.cpp:648-685) gathered per
// particle, pos_copy (cellmanager.cpp:19-26), the single periodic wrap of
// cell_pos_periodic_fix (:395-414), and the range checks the next
// connect_cell would make. R is the arithmetic type of the force laws
// (double: FP64 path; float: mixed path). Sums and positions stay double.
// ---------------------------------------------------------------------------

// The membrane sum of memb_force for the prep list's membrane particles
// [m0, m1), into S.fmemb for k_step. Computing it inside k_step instead
// spills the step kernel's registers and costs more than this launch. The
// mixed path is held to 64 registers (four blocks per SM; a few bytes spill)
// and runs about a quarter faster than at its natural 80; the FP64 path to
// 128 (two blocks per SM, no spill; 40 % faster than at its natural 138).
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 4 : 2) k_memb_force(DevState S, int32_t m0, int32_t m1) {
  pdl_entry();
  count_launch(S.launches);
  GRID_STRIDE(e, m0, m1) {
    const int32_t i = S.prep[e];
    const double3 f = memb_force<R>(S, i);
    S.fmemb[i] = make_double4(f.x, f.y, f.z, 0.0);
  }
}

template <typename Pos>
__device__ __forceinline__ const Pos* gather_source(const DevState& S);
template <>
__device__ __forceinline__ const double4* gather_source<double4>(const DevState& S) {
  return S.pos_cur;
}
template <>
__device__ __forceinline__ const float4* gather_source<float4>(const DevState& S) {
  return S.posf_cur;
}

// Entry e of a candidate row from its first chunks held in registers (e a
// constant once the caller's loop is unrolled). 16-bit entries: half e % 2
// of word (e % 8) / 2 of chunk e / 8; 32-bit: word e % 4 of chunk e / 4.
template <bool k16, int NC>
__device__ __forceinline__ uint32_t row_entry(const uint4 (&c)[NC], int e) {
  const uint4& ch = c[k16 ? e / 8 : e / 4];
  const int w = k16 ? (e % 8) / 2 : e % 4;
  const uint32_t word = w == 0 ? ch.x : (w == 1 ? ch.y : (w == 2 ? ch.z : ch.w));
  return k16 ? ((e & 1) ? word >> 16 : word & 0xffffu) : word;
}

// The candidates of particle i, from the first chunks of its row in c (kPre
// entries after the count) and the rest of the row from memory, passed to
// P.candidate with their positions. Positions are gathered kG at a time:
// all kG loads are issued before the first is used.
template <bool k16, int kPre, int kG, typename Part, int NC>
__device__ __forceinline__ void gather_candidates(const DevState& S, Part& P, const uint4 (&c)[NC],
                                                  int64_t i) {
  using Pos = typename Part::Pos;
  const int32_t pbase = P.T.pbase;
  const Pos* src = gather_source<Pos>(S) + pbase;
  const int32_t nc = (int32_t)row_entry<k16>(c, 0);
#pragma unroll
  for (int b = 1; b <= kPre; b += kG) {
    if (b > nc) break;
    int32_t q[kG];
    Pos pq[kG];
#pragma unroll
    for (int u = 0; u < kG; ++u) {
      q[u] = 0;
      if (b + u <= kPre) {
        q[u] = (int32_t)row_entry<k16>(c, b + u);
        if (b + u <= nc && EPI_CHECKED(q[u] < P.T.n, S.status, (int32_t)i, q[u]))
          pq[u] = src[q[u]];
      }
    }
#pragma unroll
    for (int u = 0; u < kG; ++u)
      if (b + u <= kPre && b + u <= nc && (q[u] < P.T.n || !kCheck))
        P.candidate(pbase + q[u], pq[u]);
  }
  for (int32_t e = kPre + 1; e <= nc; ++e) {
    const int32_t q = (int32_t)cand_entry(S, i, e);
    if (!EPI_CHECKED(q < P.T.n, S.status, (int32_t)i, q)) continue;
    P.candidate(pbase + q, src[q]);
  }
}

// One thread per particle. The first chunks of the particle's candidate row
// (15 candidates with 16-bit entries, 15 with 32-bit) are loaded up front,
// independent of each other and of the particle's own data, so the index
// stream costs one memory latency per particle rather than one per
// candidate. The neighbours' positions are then gathered kG at a time (all
// kG loads issued before the first is used). Rows longer than that (rare)
// finish with one load per entry. kMinBlocks bounds the registers so that
// that many 256-thread blocks stay resident per SM.
//
// The kernel is bound by the latency of its gathers and by issue, not by
// bytes, so what counts is how many warps an SM holds and how few
// instructions a candidate takes. What only the commit needs (the FP64
// position, the rebuild position, the membrane sums) is loaded after the
// loop, so the mixed path's registers hold the FP32 copy, the sums and the
// gathers alone: 64 registers with two gathers in flight and almost no
// spill, four blocks per SM. On 6.56M particles (512 tissues): 0.333 ms with
// three blocks and four gathers and all inputs loaded first, 0.329 ms with
// the late loads, 0.291 ms with four blocks and two gathers (0.309 with one,
// 0.308 with three, 0.326 with four; five blocks 0.326 to 0.338 with spills);
// 0.294 ms with the laws' roundings of the plain expressions.
// FP64 forces, 96 tissues: three blocks with one gather 91 us, with two 97;
// two blocks without spills 110.
// Streaming loads that do not allocate in L1 (the particle's own inputs,
// read once), leaving L1 to the neighbours' gathered positions.
__device__ __forceinline__ uint4 ld_na(const uint4* p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_na(const float4* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ double4 ld_na(const double4* p) {
  double a, b, c, d;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0,%1}, [%2];" : "=d"(a), "=d"(b) : "l"(p));
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0,%1}, [%2];"
      : "=d"(c), "=d"(d) : "l"(reinterpret_cast<const double2*>(p) + 1));
  return make_double4(a, b, c, d);
}
__device__ __forceinline__ uint32_t ld_na(const uint32_t* p) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Loads that stay where they are written, after the candidate loop (an
// ordinary load would be moved ahead of it, into registers the loop needs).
__device__ __forceinline__ double4 ld_late(const double4* p) {
  double a, b, c, d;
  asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(a), "=d"(b) : "l"(p) : "memory");
  asm volatile("ld.global.v2.f64 {%0,%1}, [%2];"
               : "=d"(c), "=d"(d) : "l"(reinterpret_cast<const double2*>(p) + 1) : "memory");
  return make_double4(a, b, c, d);
}
__device__ __forceinline__ float4 ld_late(const float4* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}

template <typename Part>
__device__ __forceinline__ void finish_particle(const DevState& S, Part& P, int64_t i) {
  double4 p;
  if constexpr (Part::kFloatPos) p = ld_late(S.pos_cur + i);
  else p = P.p;
  P.finish(p, ld_late(S.bpos + i),
           P.st == ST_MEMB ? ld_late(S.fmemb + i) : make_double4(0.0, 0.0, 0.0, 0.0));
}

template <typename R, bool kSimple, bool kOld, bool k16, int kG>
__device__ __forceinline__ void step_particle(const DevState& S, int64_t i) {
  const int64_t N = S.n_total;
  constexpr int kChunks = k16 ? 2 : 4;               // chunks loaded up front
  constexpr int kPre = kChunks * (k16 ? 8 : 4) - 1;  // candidates they hold
  uint4 c[kChunks];
#pragma unroll
  for (int k = 0; k < kChunks; ++k) c[k] = ld_na(S.cand + k * N + i);
  const uint32_t a = ld_na(S.attr + i);
  using Part = Particle<R, kSimple, kOld>;
  Part P(S, (int32_t)i, a, ld_na(S.pos_cur + i));
  gather_candidates<k16, kPre, kG>(S, P, c, i);
  finish_particle(S, P, i);
}

// The same loop with the gathers copied into shared memory asynchronously
// (cp.async, cached in L1): a thread issues the copies of kS neighbours'
// positions at once -- all 15 candidates its first two chunks hold when
// kS = 15 -- holding no register for data in flight, waits once for its own
// copies, then evaluates the candidates from its own slots (thread t's slot
// k at slots[k * kStepThreads + t]: conflict-free, no barrier needed).
constexpr int kStepThreads = 256;
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
template <typename Pos>
__device__ __forceinline__ void cp_async_pos(Pos* dst, const Pos* src) {
#pragma unroll
  for (int h = 0; h < (int)(sizeof(Pos) / 16); ++h)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(
                     reinterpret_cast<char*>(dst) + 16 * h)),
                 "l"(reinterpret_cast<const char*>(src) + 16 * h)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <bool k16, int kPre, int kS, typename Part, int NC>
__device__ __forceinline__ void gather_candidates_async(const DevState& S, Part& P,
                                                        const uint4 (&c)[NC], int64_t i,
                                                        typename Part::Pos* slots) {
  using Pos = typename Part::Pos;
  const int32_t pbase = P.T.pbase;
  const Pos* src = gather_source<Pos>(S) + pbase;
  const int32_t nc = (int32_t)row_entry<k16>(c, 0);
#pragma unroll
  for (int b = 1; b <= kPre; b += kS) {
    if (b > nc) break;
#pragma unroll
    for (int u = 0; u < kS; ++u) {
      const int e = b + u;
      if (e <= kPre && e <= nc) {
        const int32_t q = (int32_t)row_entry<k16>(c, e);
        if (EPI_CHECKED(q < P.T.n, S.status, (int32_t)i, q))
          cp_async_pos(slots + u * kStepThreads, src + q);
      }
    }
    cp_async_wait_all();
#pragma unroll
    for (int u = 0; u < kS; ++u) {
      const int e = b + u;
      if (e <= kPre && e <= nc) {
        const int32_t q = (int32_t)row_entry<k16>(c, e);
        if (q < P.T.n || !kCheck) P.candidate(pbase + q, slots[u * kStepThreads]);
      }
    }
  }
  for (int32_t e = kPre + 1; e <= nc; ++e) {
    const int32_t q = (int32_t)cand_entry(S, i, e);
    if (!EPI_CHECKED(q < P.T.n, S.status, (int32_t)i, q)) continue;
    P.candidate(pbase + q, src[q]);
  }
}

template <typename R, bool kSimple, bool kOld, int kMinBlocks, bool k16, int kS>
__global__ void __launch_bounds__(kStepThreads, kMinBlocks) k_step_async(DevState S, Range r) {
  pdl_entry();
  count_launch(S.launches);
  using Part = Particle<R, kSimple, kOld>;
  using Pos = typename Part::Pos;
  extern __shared__ __align__(16) unsigned char gather_smem[];
  Pos* slots = reinterpret_cast<Pos*>(gather_smem) + threadIdx.x;
  const int64_t i = r.p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= r.p1) return;
  const int64_t N = S.n_total;
  constexpr int kChunks = k16 ? 2 : 4;
  constexpr int kPre = kChunks * (k16 ? 8 : 4) - 1;
  uint4 c[kChunks];
#pragma unroll
  for (int k = 0; k < kChunks; ++k) c[k] = ld_na(S.cand + k * N + i);
  Part P(S, (int32_t)i, ld_na(S.attr + i), ld_na(S.pos_cur + i));
  gather_candidates_async<k16, kPre, kS>(S, P, c, i, slots);
  finish_particle(S, P, i);
}

template <typename R, bool kSimple, bool kOld, int kMinBlocks, bool k16>
__global__ void __launch_bounds__(256, kMinBlocks) k_step(DevState S, Range r) {
  pdl_entry();
  count_launch(S.launches);
  const int64_t i = r.p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= r.p1) return;
  constexpr int kG = sizeof(R) == 4 ? (kMinBlocks == 4 ? 2 : 4) : (kMinBlocks == 3 ? 1 : 2);
  step_particle<R, kSimple, kOld, k16, kG>(S, i);
}


// connect_cell's lists (for export): the exact predicate over the candidates.
__global__ void k_exact_lists(DevState S, Range r) {
  GRID_STRIDE(i, r.p0, r.p1) {
    const uint32_t a = S.attr[i];
    const TissueDev& T = S.tissues[attr_tissue(a)];
    const double4 p = S.pos_cur[i];
    const int32_t nc = cand_count(S, i);
    const double lt = T.P.lj_thresh;
    int32_t count = 0;
    for (int32_t k = 0; k < nc; ++k) {
      const int32_t q = T.pbase + (int32_t)cand_entry(S, i, k + 1);
      const double4 pq = S.pos_cur[q];
      const double d2 =
          dist_sq_exact(pdiff(p.x, pq.x, T.lx), pdiff(p.y, pq.y, T.ly), p.z - pq.z);
      if (!connected_pred(d2, lt, p.w, pq.w)) continue;
      if (count < S.max_conn) S.nbr[(int64_t)count * S.n_total + i] = q;
      ++count;
    }
    if (count > S.max_conn) raise_error(S.status, E_LIST_OVERFLOW, (int32_t)i, -1, (double)count);
    S.nn[i] = count < S.max_conn ? count : S.max_conn;
  }
}

// ---------------------------------------------------------------------------
// Export helpers (not on the per-step path).
// ---------------------------------------------------------------------------
__global__ void k_rowlen(DevState S, int32_t* rowlen, int32_t n) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t a = S.attr[i];
  rowlen[i] = S.nn[i] + (attr_state(a) == ST_MEMB ? S.tissues[attr_tissue(a)].nadj : 0);
}

__global__ void k_fill_csr(DevState S, const int32_t* rowoff, int32_t* idx, int32_t n) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t a = S.attr[i];
  const TissueDev& T = S.tissues[attr_tissue(a)];
  int32_t o = rowoff[i];
  const int32_t o0 = o;
  if (attr_state(a) == ST_MEMB)  // push order of _memb_init, cellmanager.cpp:70-166
    for (int k = 0; k < T.nadj; ++k) idx[o++] = lattice_link(T, i - T.pbase, k);
  const int32_t nn = S.nn[i];
  for (int32_t k = 0; k < nn; ++k) idx[o++] = S.nbr[(int64_t)k * S.n_total + i] - T.pbase;
  for (int32_t s = o0 + 1; s < o; ++s) {
    const int32_t v = idx[s];
    int32_t k = s - 1;
    while (k >= o0 && idx[k] > v) {
      idx[k + 1] = idx[k];
      --k;
    }
    idx[k + 1] = v;
  }
}

__global__ void k_dermis_local(DevState S, int32_t* out, int32_t n) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t a = S.attr[i];
  const uint32_t st = attr_state(a);
  const int32_t d = (st == ST_FIX || st == ST_MUSUME) ? S.dermis[i] : -1;
  out[i] = d < 0 ? -1 : d - S.tissues[attr_tissue(a)].pbase;
}

__global__ void k_unpack(DevState S, double* x, double* y, double* z, int32_t n) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4 p = S.pos_cur[i];
  x[i] = p.x;
  y[i] = p.y;
  z[i] = p.z;
}

__global__ void k_pack(DevState S, const double* x, const double* y, const double* z,
                       int32_t n) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double r = S.pos_cur[i].w;
  const double4 p = make_double4(x[i], y[i], z[i], r);
  if (!isfinite(p.x) || !isfinite(p.y) || !isfinite(p.z))
    raise_error(S.status, E_NONFINITE, (int32_t)i, -1, p.z);
  S.pos_cur[i] = p;
  S.pos_nxt[i] = p;
  const float4 f = make_float4((float)p.x, (float)p.y, (float)p.z, (float)r);
  S.posf_cur[i] = f;
  S.posf_nxt[i] = f;
}

// Particles [p0, p1) of a host step: positions from the staged host arrays
// into both buffers and both FP32 copies (as k_pack), and the displacement
// test of the candidate rows (as k_gate_check).
__global__ void k_pack_gate(DevState S, const double* x, const double* y, const double* z,
                            int32_t p0, int32_t p1) {
  GRID_STRIDE(i, p0, p1) {
    const double r = S.pos_cur[i].w;
    const double4 p = make_double4(x[i], y[i], z[i], r);
    if (!isfinite(p.x) || !isfinite(p.y) || !isfinite(p.z))
      raise_error(S.status, E_NONFINITE, (int32_t)i, -1, p.z);
    S.pos_cur[i] = p;
    S.pos_nxt[i] = p;
    const float4 f = make_float4((float)p.x, (float)p.y, (float)p.z, (float)r);
    S.posf_cur[i] = f;
    S.posf_nxt[i] = f;
    const uint32_t t = attr_tissue(S.attr[i]);
    const TissueDev& T = S.tissues[t];
    const float4 b = S.bpos[i];
    if (moved_too_far(S.skin, T, p.x, p.y, p.z, b)) {
      S.gate[1 + t] = 1;
      S.gate[0] = 1;
    }
  }
}

__global__ void k_unpack_range(DevState S, double* x, double* y, double* z, int32_t p0,
                               int32_t p1) {
  GRID_STRIDE(i, p0, p1) {
    const double4 p = S.pos_cur[i];
    x[i] = p.x;
    y[i] = p.y;
    z[i] = p.z;
  }
}

__global__ void k_posf(DevState S) {
  GRID_STRIDE(i, 0, S.n_total) {
    const double4 p = S.pos_cur[i];
    S.posf_cur[i] = make_float4((float)p.x, (float)p.y, (float)p.z, (float)p.w);
  }
}

}  // namespace

void launch_posf(const DevState& S, const LaunchCfg& lc, cudaStream_t s) {
  if (S.n_total > 0) k_posf<<<stride_blocks(S.n_total, lc.block, lc), lc.block, 0, s>>>(S);
}

void launch_scan(const int32_t* in, int32_t* out, int32_t n, int32_t init,
                 const ScanScratch& sc, const int32_t* gate, const LaunchCfg&,
                 cudaStream_t s) {
  const int32_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb == 0) {
    k_set1<<<1, 1, 0, s>>>(out, init, gate);
    return;
  }
  k_scan_partial<<<nb, kScanThreads, 0, s>>>(in, n, sc.partial, gate);
  k_scan_top<<<1, kScanThreads, 0, s>>>(sc.partial, nb, gate);
  k_scan_final<<<nb, kScanThreads, 0, s>>>(in, out, n, sc.partial, init, gate);
}

void launch_rebuild(const DevState& S, const Range& r, const ScanScratch&,
                    const LaunchCfg& lc, cudaStream_t s, Timer* tm, bool listed) {
  const int B = lc.block;
  const int grid = lc.num_sms * 8;
  if (!listed) {
    timer_begin(tm, KC_GATE, s);
    launch_pdl(k_gate_compact, 1, kScanThreads, s, S, r.t0, r.t1);
    timer_end(tm, KC_GATE, s);
  }
  timer_begin(tm, KC_REBUILD_BIN, s);
  launch_pdl(k_bin, grid, B, s, S);
  timer_end(tm, KC_REBUILD_BIN, s);
  timer_begin(tm, KC_REBUILD_SCAN, s);
  const int nt = r.t1 - r.t0;
  const int64_t units = (int64_t)nt * S.scan_chunks;
  launch_pdl(k_scan_tissue, (int)std::max<int64_t>(1, std::min<int64_t>(units, lc.num_sms * 4)),
             kTissueScanThreads, s, S);
  timer_end(tm, KC_REBUILD_SCAN, s);
  timer_begin(tm, KC_REBUILD_SORT, s);
  launch_pdl(k_scatter, grid, B, s, S);
  launch_pdl(k_binsort, grid, B, s, S);
  timer_end(tm, KC_REBUILD_SORT, s);
  timer_begin(tm, KC_REBUILD_SEARCH, s);
  if (S.cand16) launch_pdl(k_cand_search<true>, grid, B, s, S, (int32_t)lc.search_switch);
  else launch_pdl(k_cand_search<false>, grid, B, s, S, (int32_t)lc.search_switch);
  timer_end(tm, KC_REBUILD_SEARCH, s);
}

void launch_memb_force(const DevState& S, int32_t m0, int32_t m1, int precision,
                       const LaunchCfg& lc, cudaStream_t s, Timer* tm) {
  if (m1 <= m0) return;
  timer_begin(tm, KC_PREPASS, s);
  const int gm = stride_blocks(m1 - m0, lc.block, lc);
  if (precision == 1)
    launch_pdl(k_memb_force<float>, gm, lc.block, s, S, m0, m1);
  else
    launch_pdl(k_memb_force<double>, gm, lc.block, s, S, m0, m1);
  timer_end(tm, KC_PREPASS, s);
}

void launch_dermis(const DevState& S, int32_t f0, int32_t f1, const LaunchCfg& lc,
                   cudaStream_t s, Timer* tm) {
  if (f1 <= f0) return;
  timer_begin(tm, KC_PREPASS, s);
  launch_pdl(k_dermis, stride_blocks((int64_t)(f1 - f0) * 32, lc.block, lc), lc.block, s, S, f0,
             f1);
  timer_end(tm, KC_PREPASS, s);
}

void launch_prepass(const DevState& S, int32_t m0, int32_t m1, int32_t f0, int32_t f1,
                    int precision, const LaunchCfg& lc, cudaStream_t s, Timer* tm) {
  launch_memb_force(S, m0, m1, precision, lc, s, tm);
  launch_dermis(S, f0, f1, lc, s, tm);
}

// The asynchronous-gather kernel with kS shared-memory slots per thread.
template <typename R, bool kSimple, bool kOld, bool k16, int kS, int kMinBlocks>
void launch_step_async(const DevState& S, const Range& r, const LaunchCfg& lc, cudaStream_t s) {
  using Pos = typename std::conditional<sizeof(R) == 4, float4, double4>::type;
  auto kern = k_step_async<R, kSimple, kOld, kMinBlocks, k16, kS>;
  constexpr int smem = kS * kStepThreads * (int)sizeof(Pos);
  // once per context (and so per device) and form; every context sets the same
  constexpr int form = (k16 ? 1 : 0) + (kS > 128 / (int)sizeof(Pos) ? 2 : 0) +
                       4 * (kSimple ? (kOld ? 1 : 0) : 2) + (sizeof(R) == 4 ? 12 : 0);
  if (!(lc.step_sized >> form & 1u)) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    lc.step_sized |= 1u << form;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks_for(r.p1 - r.p0, kStepThreads));
  cfg.blockDim = dim3((unsigned)kStepThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, S, r);
}

// Tuning variants: 1 and 2, gathers copied asynchronously into shared
// memory, 8 (FP64: 4) and 15 (FP64: 8) slots per thread; 3 and 4, gathers
// into registers at two register budgets: 3, three resident 256-thread blocks
// per SM and four gathers at a time (FP64: one; the FP64 default); 4, four
// blocks and two gathers (the mixed path's default; FP64: two blocks).
template <typename R, bool kSimple, bool kOld, bool k16>
void launch_step_w(const DevState& S, const Range& r, const LaunchCfg& lc, cudaStream_t s) {
  const int grid = blocks_for(r.p1 - r.p0, 256);
  constexpr bool kF = sizeof(R) == 4;
  switch (lc.variant) {
    case 1: launch_step_async<R, kSimple, kOld, k16, kF ? 8 : 4, kF ? 4 : 3>(S, r, lc, s); break;
    case 2: launch_step_async<R, kSimple, kOld, k16, kF ? 15 : 8, 3>(S, r, lc, s); break;
    case 3: launch_pdl(k_step<R, kSimple, kOld, 3, k16>, grid, 256, s, S, r); break;
    default: launch_pdl(k_step<R, kSimple, kOld, kF ? 4 : 2, k16>, grid, 256, s, S, r); break;
  }
}

template <typename R, bool kSimple, bool kOld>
void launch_step_v(const DevState& S, const Range& r, const LaunchCfg& lc, cudaStream_t s) {
  if (S.cand16) launch_step_w<R, kSimple, kOld, true>(S, r, lc, s);
  else launch_step_w<R, kSimple, kOld, false>(S, r, lc, s);
}

template <typename R>
void launch_step_r(const DevState& S, const Range& r, const LaunchCfg& lc, cudaStream_t s) {
  if (lc.simple && lc.any_old)
    launch_step_v<R, true, true>(S, r, lc, s);
  else if (lc.simple)
    launch_step_v<R, true, false>(S, r, lc, s);
  else
    launch_step_v<R, false, true>(S, r, lc, s);
}

void launch_step(const DevState& S, const Range& r, int precision, const LaunchCfg& lc,
                 cudaStream_t s, Timer* tm) {
  const int32_t np = r.p1 - r.p0;
  if (np <= 0) return;
  timer_begin(tm, KC_STEP, s);
  if (precision == 1)
    launch_step_r<float>(S, r, lc, s);
  else
    launch_step_r<double>(S, r, lc, s);
  timer_end(tm, KC_STEP, s);
}

void launch_exact_lists(const DevState& S, const Range& r, const LaunchCfg& lc,
                        cudaStream_t s) {
  const int32_t np = r.p1 - r.p0;
  if (np > 0) k_exact_lists<<<stride_blocks(np, lc.block, lc), lc.block, 0, s>>>(S, r);
}

// Loop counter of the step graph's WHILE node: one pass of the body (two
// steps) done; run another while pairs remain.
__global__ void k_loop_tick(int32_t* remaining, cudaGraphConditionalHandle h,
                            unsigned long long* launches) {
  pdl_entry();
  count_launch(launches);
  const int32_t left = *remaining - 1;
  *remaining = left;
  cudaGraphSetConditional(h, left > 0 ? 1u : 0u);
}

void launch_loop_tick(int32_t* remaining, cudaGraphConditionalHandle h,
                      unsigned long long* launches, cudaStream_t s) {
  launch_pdl(k_loop_tick, 1, 1, s, remaining, h, launches);
}

void launch_set_counter(int32_t* remaining, int32_t value, cudaStream_t s) {
  k_set1<<<1, 1, 0, s>>>(remaining, value, nullptr);
}

void launch_rebuild_condition(const DevState& S, const Range& r, cudaGraphConditionalHandle h,
                              cudaStream_t s) {
  launch_pdl(k_rebuild_condition, 1, kScanThreads, s, S, r.t0, r.t1, h);
}

void launch_set_gates(const DevState& S, int32_t ntissues, cudaStream_t s) {
  k_gate_set_all<<<(ntissues + 255) / 256 + 1, 256, 0, s>>>(S, ntissues);
}

void launch_rowlen(const DevState& S, int32_t* rowlen, int32_t n, cudaStream_t s) {
  if (n > 0) k_rowlen<<<blocks_for(n, 256), 256, 0, s>>>(S, rowlen, n);
}
void launch_fill_csr(const DevState& S, const int32_t* rowoff, int32_t* idx, int32_t n,
                     cudaStream_t s) {
  if (n > 0) k_fill_csr<<<blocks_for(n, 256), 256, 0, s>>>(S, rowoff, idx, n);
}
void launch_dermis_local(const DevState& S, int32_t* out, int32_t n, cudaStream_t s) {
  if (n > 0) k_dermis_local<<<blocks_for(n, 256), 256, 0, s>>>(S, out, n);
}
void launch_unpack_positions(const DevState& S, double* x, double* y, double* z, int32_t n,
                             cudaStream_t s) {
  if (n > 0) k_unpack<<<blocks_for(n, 256), 256, 0, s>>>(S, x, y, z, n);
}
void launch_pack_gate(const DevState& S, const double* x, const double* y, const double* z,
                      int32_t p0, int32_t p1, const LaunchCfg& lc, cudaStream_t s) {
  if (p1 > p0) k_pack_gate<<<stride_blocks(p1 - p0, lc.block, lc), lc.block, 0, s>>>(S, x, y, z, p0, p1);
}
void launch_unpack_range(const DevState& S, double* x, double* y, double* z, int32_t p0,
                         int32_t p1, const LaunchCfg& lc, cudaStream_t s) {
  if (p1 > p0)
    k_unpack_range<<<stride_blocks(p1 - p0, lc.block, lc), lc.block, 0, s>>>(S, x, y, z, p0, p1);
}
void launch_pack_positions(const DevState& S, const double* x, const double* y,
                           const double* z, int32_t n, cudaStream_t s) {
  if (n > 0) k_pack<<<blocks_for(n, 256), 256, 0, s>>>(S, x, y, z, n);
}

}  // namespace epi
