// Resident stepping: one cooperative kernel that runs a whole sequence of
// steps of a small batch.
//
// A small batch (a tissue or a few dozen) does not fill the GPU: a step of
// the kernel sequence is then a chain of launches and of dependent loads by
// few threads -- 768 particles took 55 us per call, 36,864 took 19 us per
// step of the replayed graph, of which the arithmetic is under 2. Here every
// block stays on its SM for all steps:
//   * every term of a step -- a candidate of a particle, a bending term or a
//     lattice spring of a membrane particle -- is a task of its own thread,
//     so the chain of a step is one gather and one evaluation deep whatever
//     the row's length;
//   * the terms meet in shared memory and one thread per particle sums them
//     in the row's order and commits: the same operations in the same order
//     as the thread-per-particle kernels, so the same bits;
//   * the block's own positions, rows and constants stay in shared memory;
//   * blocks meet at a grid barrier after every step (and between the phases
//     of a candidate rebuild, which runs in the same kernel when some tissue
//     is flagged).
// Bound by latency: per step one barrier (about 1.5 us), one gather from L2
// (0.4 us), and the evaluation, summing and committing chains. A step costs
// 4.9 us for 768 particles (FP64; 21 in the graph), 6.9 for 36,864 (13.5),
// 11.7 for 92,160 (16.1), and meets the sequence at 147,456 (17 both); FP64
// forces 9.9 for 36,864 (18.1). Batches: 9 tissues of 106,112 particles 18.0
// (20.6), 64 small ones of 49,152 17.5 (20.5); with every cell state and FP64
// forces 16 tissues of 17,360 particles 20 (97), 64 53 (104), 118 97 (117).
#include "epi_kernels.h"

#include <algorithm>

#include "epi_device.cuh"
#include "epi_rebuild.cuh"
#include "epi_step.cuh"

namespace epi {
namespace {

constexpr int kTile = 8;  // consecutive particles dealt to a block at a time

// Positions the run works on: step k reads pos(k), writes pos(k + 1).
struct ResidentArgs {
  int32_t nsteps;
  int32_t slots;            // particles per block
  int32_t membs;            // membrane particles a block may hold
  int32_t turn;             // of which it holds the terms at a time
  int32_t tasks;            // pair terms a block holds at a time
  int32_t terms;            // bending threads per membrane particle
  int32_t group;            // blocks that deal their range's tiles of particles among them
  int32_t thread_from;      // candidate search: a thread per particle from here on
  unsigned* bar;            // barrier arrivals (zero at launch)
  unsigned* other;          // the next run's (zeroed here)
  int32_t* abort;           // set when a barrier wait gave up
  int32_t* flags;           // RunFlags::words
  int32_t polls;            // limit of a barrier wait
  DevStatus* post;          // non-null: pinned host memory the status is put in
  int32_t per_step, per_pair, per_rebuild;  // kernels stood for (see ResidentCfg)
  double4* hist;            // non-null: step k's positions go to hist + k n_total
};

// Waits of thread 0 of every block; a wait that is not met within the limit
// gives up: the error is recorded and every block leaves at its next check.
struct GridBarrier {
  unsigned* bar;
  int32_t* abort;
  DevStatus* status;
  int32_t limit;  // polls
  unsigned target;
  // word: read by thread 0 after the barrier and returned to all threads of
  // the block (the same value in every block: see RunFlags). False: some
  // block gave up.
  __device__ __forceinline__ bool sync(const int32_t* word, int32_t* value) {
    __shared__ int32_t s_word, s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
      target += gridDim.x;
      // release: the block's writes (ordered before by the block barrier)
      // are visible to whoever sees the count; acquire: and the other way
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      unsigned seen;
      int spins = 0;
      int32_t ok = 1;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        if ((int32_t)(seen - target) >= 0) break;
        if (++spins >= limit || ((spins & 1023) == 0 && *(volatile int32_t*)abort)) {
          if (spins >= limit) {
            raise_error(status, E_TIMEOUT, (int32_t)blockIdx.x, -1, (double)seen);
            *(volatile int32_t*)abort = 1;
          }
          ok = 0;
          break;
        }
      }
      s_ok = ok;
      s_word = word ? *(volatile const int32_t*)word : 0;
    }
    __syncthreads();
    if (value) *value = s_word;
    return s_ok != 0;
  }
};

// The candidate rebuild of the flagged tissues, the phases of launch_rebuild
// between barriers. The word every block acted on, *flag, is cleared once all
// blocks are past the first barrier here (RunFlags).
template <int NT>
__device__ __noinline__ bool resident_rebuild(const DevState& S0, double4* pos, int32_t thread_from,
                                              int32_t* flag, GridBarrier& B) {
  DevState S = S0;
  S.pos_cur = pos;
  if (blockIdx.x == 0) gate_compact<NT>(S, 0, S.ntissues, true, false);
  if (!B.sync(nullptr, nullptr)) return false;
  if (blockIdx.x == 0 && threadIdx.x == 0) *flag = 0;
  rebuild_bin(S);
  if (!B.sync(nullptr, nullptr)) return false;
  rebuild_scan<NT>(S);
  if (!B.sync(nullptr, nullptr)) return false;
  rebuild_scatter(S);
  if (!B.sync(nullptr, nullptr)) return false;
  rebuild_sort(S);
  if (!B.sync(nullptr, nullptr)) return false;
  if (S.cand16) rebuild_search<true>(S, thread_from);
  else rebuild_search<false>(S, thread_from);
  return B.sync(nullptr, nullptr);
}

constexpr int kLinks = kMembAdjTri + 1;  // springs of a membrane particle, and its wall
constexpr int kTissues = 8;  // tissues of a group whose constants its blocks keep

// What a block keeps of its particles (slots) in shared memory between steps:
// an L2 load costs 700 cycles and more here, and after a barrier L1 holds
// nothing. R: the arithmetic type of the forces.
template <typename R>
struct Slots {
  using Pos = typename SiteOffsets<R>::Pos;
  double4* pos;     // positions
  double* sum;      // pair sums, 3 per slot
  double* msum;     // membrane sums, 3 per membrane slot
  Pos* own;         // the same as the forces see them (FP64 path: pos itself)
  float4* bpos;     // positions at the last candidate rebuild
  R* term;          // pair terms x | y | z (tasks each)
  R* bend;          // bending terms t, g: 4 x terms per membrane slot of a turn
  R* link;          // spring terms and the wall: 3 x kLinks of the same
  uint32_t* attr;
  int32_t* off;     // slots + 1: first pair task of each slot
  int32_t* at;      // membrane slot: its place in list
  int32_t* list;    // slots of membrane particles
  uint32_t* jk;     // their lattice column and row (16 bits each: a membrane is three
                    // wide or more, so of kResidentParticles it has under 65,536 rows)
  uint32_t* task;   // pair tasks: partner (global index, 20 bits) | slot << 20
  static constexpr bool kOwn = sizeof(R) == 4;
  // terms: bending threads per membrane particle (kTriTerms, or with square
  // lattices only kSquareTerms + 2)
  static __host__ __device__ constexpr size_t bytes(int slots, int membs, int turn, int tasks,
                                                    int terms) {
    return (size_t)slots * (sizeof(double4) + 24 + (kOwn ? sizeof(float4) : 0) + sizeof(float4) + 8) +
           (size_t)membs * 24 +
           sizeof(R) * 3 * tasks + sizeof(R) * (4 * terms + 3 * kLinks) * turn +
           4 * (slots + 4 + 2 * membs + tasks);
  }
  __device__ Slots(unsigned char* m, int slots, int membs, int turn, int tasks, int terms) {
    pos = reinterpret_cast<double4*>(m);
    bpos = reinterpret_cast<float4*>(pos + slots);
    unsigned char* rest = reinterpret_cast<unsigned char*>(bpos + slots);
    if constexpr (kOwn) {
      own = reinterpret_cast<float4*>(rest);
      rest += sizeof(float4) * slots;
    } else {
      own = pos;
    }
    sum = reinterpret_cast<double*>(rest);
    msum = sum + 3 * slots;
    bend = reinterpret_cast<R*>(msum + 3 * membs);
    link = bend + 4 * terms * turn;
    term = link + 3 * kLinks * turn;
    attr = reinterpret_cast<uint32_t*>(term + 3 * tasks);
    off = reinterpret_cast<int32_t*>(attr + slots);
    at = off + slots + 1;
    list = at + slots;
    jk = reinterpret_cast<uint32_t*>(list + membs);
    task = reinterpret_cast<uint32_t*>(jk + membs);
  }
};

// Bending term e of membrane particle i, evaluated by all lanes of a warp for
// the terms they hold (live: this lane holds one). Square terms (square_term's
// order) are taken over three consecutive sites of the row or column, s[0] ->
// s[1] and s[1] -> s[2]; the last one (e = 5) takes its cosine from the row
// two below (the reference reads memb_bb's ipn, :380), which the next lane
// (e = 6) forms. Triangular ones (tri_term1, tri_term2) over three
// neighbours. All sites are loaded before one is used.
template <typename R>
__device__ __forceinline__ BendTerm<R> bend_task(const DevState& S, int32_t i,
                                                 const SiteOffsets<R>& off, const MembSites& M,
                                                 bool tri, int e, bool live) {
  using Pos = typename SiteOffsets<R>::Pos;
  int32_t site[3] = {i, i, i};
  const int kind = square_kind(e < 6 ? e : 0);
  if (!live) {
  } else if (tri) {
    const int k = e < 6 ? e : e - 6;
    site[0] = M.tri(S, k);
    site[1] = M.tri(S, k == 5 ? 0 : k + 1);
    site[2] = e < 6 ? M.tri_ring(S, k) : M.tri(S, k >= 4 ? k - 4 : k + 2);
  } else {
    const bool col = e >= 3 && e < 6;
    const int d = e == 6 ? 0 : (kind == 0 ? -1 : (kind == 1 ? 0 : -2));
#pragma unroll
    for (int k = 0; k < 3; ++k)
      site[k] = M.square(S, col ? 0 : d + k, col ? d + k : (e == 6 ? -2 : 0));
  }
  Pos at[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) at[k] = off.at(site[k]);
  const Vec3<R> a = off.from(at[0]), b = off.from(at[1]), c = off.from(at[2]);
  BendTerm<R> t{Vec3<R>{R(0), R(0), R(0)}, R(0)};
  if (live && tri) t = e < 6 ? tri_term1(a, b, c) : tri_term2(a, b, c);
  if (__any_sync(0xffffffffu, live && !tri)) {
    const Unit<R> u = unit_ab(a, b), v = unit_ab(b, c);
    R cs = v3_dot(u.v, v.v);
    const R next = __shfl_down_sync(0xffffffffu, cs, 1);
    if (e == 5) cs = next;
    if (live && !tri && e < 6)
      t = square_term(kind, kind == 0 ? v : u, kind == 0 ? u : v, cs);
  }
  return t;
}

// NT threads per block, one block per SM (more threads would halve their
// registers: at 64 a thread spilled 45 words a step, and a reload misses L1
// after a barrier: 9.2 us per step on 36,864 particles against 7.0). A group
// of blocks holds consecutive particles of about kTissues tissues, whose
// constants each block has in shared memory (those of a single one, kOne, are
// arguments), and deals them round in tiles of kTile particles, so that every
// block gets its share of the membrane and of the long rows.
template <typename R, bool kSimple, bool kOld, bool kOne, int NT>
__global__ void __launch_bounds__(NT, 1) k_resident(const __grid_constant__ DevState S0,
                                                       const __grid_constant__ ResidentArgs A,
                                                       const __grid_constant__ TissueDev T0) {
  using Part = Particle<R, kSimple, kOld>;
  using Pos = typename Part::Pos;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) unsigned char s_tissue[kTissues][sizeof(TissueDev)];
  __shared__ int32_t s_nm, s_t0;
  const int slots = A.slots;
  const Slots<R> K(smem, slots, A.membs, A.turn, A.tasks, A.terms);
  const int32_t n = (int32_t)S0.n_total;
  const int tid = (int)threadIdx.x;
  DevState S = S0;
  if (A.hist) S.pos_cur = A.hist;
  if (A.hist) S.pos_nxt = A.hist + n;
  GridBarrier B{A.bar, A.abort, S0.status, A.polls, 0u};
  unsigned long long counted = 0;
  const RunFlags flags{S0.gate, A.flags};
  int32_t flagged = *(volatile const int32_t*)flags.read_by(0);
  // this block's group: its first particle, its blocks, the block's place
  const int32_t lead = kOne ? 0 : (int32_t)blockIdx.x / A.group * A.group;
  const int32_t deal = kOne ? (int32_t)gridDim.x : min(A.group, (int32_t)gridDim.x - lead);
  auto particle = [&](int slot) {
    return lead * slots + (slot / kTile * deal + (int32_t)blockIdx.x - lead) * kTile + slot % kTile;
  };
  // once: the slots' attributes, positions and membrane list, and the
  // constants of the block's first tissues
  if (tid == 0) {
    if (blockIdx.x == 0) *A.other = 0u;
    s_nm = 0;
    s_t0 = !kOne && lead * slots < n ? (int32_t)attr_tissue(S0.attr[lead * slots]) : 0;
  }
  __syncthreads();
  for (int s = tid; s < slots; s += NT) {
    const int32_t i = particle(s);
    K.off[s] = 0;
    if (i >= n) continue;
    const uint32_t a = S0.attr[i];
    const double4 p = S.pos_cur[i];
    const int32_t nc = cand_count(S, i);
    const float4 b = S.bpos[i];
    K.attr[s] = a;
    K.pos[s] = p;
    K.off[s] = nc;
    K.bpos[s] = b;
    if constexpr (Slots<R>::kOwn) K.own[s] = Part::own(p);
    if (attr_state(a) == ST_MEMB) {
      const TissueDev& T = kOne ? T0 : S0.tissues[attr_tissue(a)];
      const int32_t j = i - T.pbase, at = atomicAdd(&s_nm, 1);
      if (!EPI_CHECKED(at < A.membs, S0.status, i, at)) continue;
      K.list[at] = s;
      K.jk[at] = (uint32_t)(j % T.nmx) | (uint32_t)(j / T.nmx) << 16;
      K.at[s] = at;
    }
  }
  if constexpr (!kOne) {
    for (int t = 0; t < kTissues && s_t0 + t < S0.ntissues; ++t) {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(S0.tissues + s_t0 + t);
      for (int w = tid; w < (int)(sizeof(TissueDev) / 4); w += NT)
        reinterpret_cast<uint32_t*>(s_tissue[t])[w] = from[w];
    }
  }
  auto tissue = [&](uint32_t a) -> const TissueDev& {
    if constexpr (kOne) return T0;
    const int32_t t = (int32_t)attr_tissue(a) - s_t0;
    return t < kTissues ? *reinterpret_cast<const TissueDev*>(s_tissue[t])
                        : S0.tissues[attr_tissue(a)];
  };
  // slots [c0, c1) hold the pair tasks listed in K.task
  int c0 = 0, c1 = 0;
  bool fresh = true, rebuilt = false;  // rows are to be listed, to be read first
  bool done = false;
  for (int32_t step = 0; step < A.nsteps; ++step) {
    counted += A.per_step + ((step & 1) ? A.per_pair : 0);
    S.flag = flags.raised_by(step);
    if (flagged) {
      counted += A.per_rebuild;
      if (!resident_rebuild<NT>(S0, S.pos_cur, A.thread_from, flags.read_by(step), B)) break;
      fresh = rebuilt = true;
    }
    if (fresh) {
      fresh = false;
      // first task of each slot, from the row lengths (in K.off after the
      // set-up, read again after a rebuild)
      int32_t carry = 0;
      for (int base = 0; base < slots; base += NT) {
        const int s = base + tid;
        int32_t nc = 0;
        if (s < slots) {
          const int32_t i = particle(s);
          if (!rebuilt) {
            nc = K.off[s];  // written by this thread
          } else if (i < n) {
            nc = cand_count(S, i);
            K.bpos[s] = S.bpos[i];
          }
        }
        int32_t total;
        const int32_t before = block_excl_scan<NT>(nc, &total);
        if (s < slots) K.off[s] = carry + before;
        carry += total;
      }
      if (tid == 0) K.off[slots] = carry;
      c0 = c1 = 0;
      __syncthreads();
    }
    if (!kSimple && S.nprep > S.nprep_memb) {
      const int warps = (int)(gridDim.x * NT) >> 5;
      for (int32_t e = S.nprep_memb + (int32_t)((blockIdx.x * NT + tid) >> 5); e < S.nprep;
           e += warps)
        dermis_cell(S, S.prep[e], tid & 31);
      if (!B.sync(nullptr, nullptr)) break;
    }
    // in turns: pair terms of the slots from `from` on, membrane terms of the
    // membrane slots from `m0` on, as many as fit (kSimple: all of them)
    const int held = min(s_nm, A.membs);  // (the same: the host counted them)
    int from = 0, m0 = 0;
    do {
      const bool pairs = kSimple || from < slots;
      // the slots whose pair tasks fit; listed once per rebuild when all do
      if (pairs && (c0 != from || c1 == from)) {
        c0 = from;
        int lo = from + 1, hi = slots;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (K.off[mid] - K.off[c0] <= A.tasks) lo = mid;
          else hi = mid - 1;
        }
        c1 = lo;
        const int32_t t0 = K.off[c0], nt = K.off[c1] - t0;
        for (int t = tid; t < nt; t += NT) {
          int a = c0, b = c1;  // the slot of task t: off[a] <= t0 + t < off[b]
          while (b - a > 1) {
            const int mid = (a + b) >> 1;
            if (K.off[mid] <= t0 + t) a = mid;
            else b = mid;
          }
          const int32_t i = particle(a);
          const int32_t q = tissue(K.attr[a]).pbase +
                            (int32_t)cand_entry(S, i, t0 + t - K.off[a] + 1);
          K.task[t] = (uint32_t)(EPI_CHECKED(q >= 0 && q < n, S.status, i, q) ? q : i) |
                      (uint32_t)a << 20;
        }
        __syncthreads();
      }
      // every term of these slots: a thread each
      const int32_t t0 = K.off[c0], np = pairs ? K.off[c1] - t0 : 0;
      R *tx = K.term, *ty = tx + A.tasks, *tz = ty + A.tasks;
      const Pos* src;
      if constexpr (Part::kFloatPos) src = S.posf_cur;
      else src = S.pos_cur;
      constexpr int kU = Part::kFloatPos ? 4 : 2;  // gathers in flight per thread
      for (int base = tid; base < np; base += kU * NT) {
        uint32_t w[kU];
        Pos pq[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          if (base + u * NT < np) {
            w[u] = K.task[base + u * NT];
            pq[u] = src[w[u] & 0xfffffu];
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int t = base + u * NT;
          if (t < np) {
            const int slot = (int)(w[u] >> 20);
            const uint32_t a = K.attr[slot];
            Part P(S, particle(slot), a, K.own[slot], tissue(a));
            const Vec3<R> v = P.term((int32_t)(w[u] & 0xfffffu), pq[u]);
            P.report_bad();
            tx[t] = v.x;
            ty[t] = v.y;
            tz[t] = v.z;
          }
        }
      }
      const int nm = kSimple && from > 0 ? 0 : min(held - m0, A.turn);
      if (nm > 0) {
        // the membrane: bending terms, then lattice springs, A.terms and
        // kLinks threads per particle, from the first warp on that took
        // no or one pair task less
        const int nb32 = (nm * A.terms + 31) & ~31, nl = nm * kLinks;
        for (int t = (tid + NT - (np & ~31) % NT) % NT; t < nb32 + nl; t += NT) {
          const bool spring = t >= nb32;
          const int r = spring ? t - nb32 : t;
          const int m = r / (spring ? kLinks : A.terms);
          const int e = r - m * (spring ? kLinks : A.terms);
          const bool in = m < nm;
          const int slot = in ? K.list[m0 + m] : 0;
          const int32_t i = particle(slot);
          const TissueDev& T = tissue(K.attr[slot]);
          const bool tri = T.lattice == kLatticeTriangular;
          const SiteOffsets<R> off(S, K.own[slot], T);
          const uint32_t jk = in ? K.jk[m0 + m] : 0u;
          const MembSites M(T, i, (int32_t)(jk & 0xffffu), (int32_t)(jk >> 16));
          if (spring) {
            if (!in) continue;
            if (e == kMembAdjTri) {  // the wall
              const double4 p = K.pos[slot];
              K.link[3 * r] = p.z < p.w ? T.laws<R>().wall(R(T.P.dt), R(p.z), R(p.w)) : R(0);
              continue;
            }
            if (e >= T.nadj) continue;
            const int32_t q = M.link(S, tri, e);
            const Vec3<R> v = link_term<R>(S, off, T, T.laws<R>(), R(T.P.dt), i, q, off.at(q));
            R* o = K.link + 3 * r;
            o[0] = v.x;
            o[1] = v.y;
            o[2] = v.z;
          } else {
            const bool live = in && e < (tri ? kTriTerms : kSquareTerms + 1);
            const BendTerm<R> b = bend_task<R>(S, i, off, M, tri, e, live);
            if (!live) continue;
            R* o = K.bend + 4 * r;
            o[0] = b.t.x;
            o[1] = b.t.y;
            o[2] = b.t.z;
            o[3] = b.g;
          }
        }
      }
      __syncthreads();
      // sums in the order of the thread-per-particle kernels, a thread per
      // component: the slots' pair terms, then the membrane's
      const int ns = pairs ? c1 - c0 : 0;
      for (int r = tid; r < 3 * (ns + nm); r += NT) {
        if (r < 3 * ns) {
          const int s = c0 + r / 3, c = r % 3;
          const R* v = K.term + c * A.tasks;
          double sum = 0.0;
          const int end = K.off[s + 1] - t0;
#pragma unroll 4
          for (int t = K.off[s] - t0; t < end; ++t) sum = xadd(sum, double(v[t]));
          K.sum[3 * s + c] = sum;
        } else {
          const int m = (r - 3 * ns) / 3, c = (r - 3 * ns) % 3, slot = K.list[m0 + m];
          const TissueDev& T = tissue(K.attr[slot]);
          const int nb = T.lattice == kLatticeTriangular ? kTriTerms : kSquareTerms;
          const R* b = K.bend + 4 * A.terms * m;
          R v = R(0);
#pragma unroll 4
          for (int e = 0; e < nb; ++e) v = xfma(b[4 * e + 3], b[4 * e + c], v);
          double sum = double(xmul(R(T.P.dt * T.P.kbend), v));
          const R* l = K.link + 3 * kLinks * m + c;
#pragma unroll 2
          for (int e = 0; e < T.nadj; ++e) sum = xadd(sum, double(l[3 * e]));
          // (adding no wall, +0, changes nothing: the sum is not -0)
          if (c == 2) sum = xadd(sum, double(l[3 * kMembAdjTri - 2]));
          K.msum[3 * (m0 + m) + c] = sum;
        }
      }
      __syncthreads();
      if (pairs) from = c1;
      if (!kSimple) m0 += nm;
    } while (from < slots || (!kSimple && m0 < held));
    // the commit, a thread per particle
    for (int s = tid; s < slots; s += NT) {
      const int32_t i = particle(s);
      if (i >= n) continue;
      const uint32_t a = K.attr[s];
      const double4 p = K.pos[s];
      Part P(S, i, a, K.own[s], tissue(a));
      P.ax = K.sum[3 * s];
      P.ay = K.sum[3 * s + 1];
      P.az = K.sum[3 * s + 2];
      double4 f = make_double4(0.0, 0.0, 0.0, 0.0);
      if (attr_state(a) == ST_MEMB) {
        const double* v = K.msum + 3 * K.at[s];
        f = make_double4(v[0], v[1], v[2], 0.0);
      }
      const double4 q = P.finish(p, K.bpos[s], f);
      K.pos[s] = q;
      if constexpr (Slots<R>::kOwn) K.own[s] = Part::own(q);
    }
    if (A.hist) {
      S.pos_cur = S.pos_nxt;
      S.pos_nxt += n;
    } else {
      double4* t = S.pos_cur;
      S.pos_cur = S.pos_nxt;
      S.pos_nxt = t;
    }
    float4* tf = S.posf_cur;
    S.posf_cur = S.posf_nxt;
    S.posf_nxt = tf;
    done = step + 1 == A.nsteps;
    if (!B.sync(done ? nullptr : flags.read_by(step + 1), &flagged)) {
      done = false;
      break;
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    if (S0.launches) {
      atomicAdd(S0.launches, counted);
      atomicAdd(S0.launches + 1, 1ull);
      atomicAdd(S0.launches + 2, counted);
    }
    // past the last barrier every block has raised what it had to: the host
    // finds the status after its wait for the stream, without a copy. (All is
    // read before anything is written: one trip to L2.)
    if (done) {
      const int32_t raised = *(const volatile int32_t*)flags.read_by(A.nsteps);
      const volatile DevStatus* from = S0.status;
      const DevStatus s{from->flags | kStatusPosted, from->code, from->a, from->b, from->v};
      if (raised) flags.hand_on(A.nsteps);
      if (A.post) {
        volatile DevStatus* to = A.post;
        to->code = s.code;
        to->a = s.a;
        to->b = s.b;
        to->v = s.v;
        to->flags = s.flags;
      }
    }
  }
}

// Kernel of a batch's form, and the form's number (0 to 11).
constexpr int kThreads = 512;
template <typename R, bool kOne>
const void* kernel_of(const LaunchCfg& lc, int* form) {
  const int kind = lc.simple ? (lc.any_old ? 1 : 0) : 2;
  *form = kind + (kOne ? 3 : 0) + (sizeof(R) == 4 ? 6 : 0);
  if (kind == 1) return (const void*)k_resident<R, true, true, kOne, kThreads>;
  if (kind == 0) return (const void*)k_resident<R, true, false, kOne, kThreads>;
  return (const void*)k_resident<R, false, true, kOne, kThreads>;
}

// Of 227 KB, less the static parts. The limit that every kernel is given,
// whatever a plan needs of it: the attribute belongs to the kernel, not to a
// context, so contexts in other threads may be between setting and launching.
constexpr size_t kSmemPerBlock = 216 * 1024;
static_assert(kResidentParticles / 3 < 65536, "rows of a membrane fit 16 bits");
constexpr int kLeastSlots = 16;
// pair terms per slot a block must have room for: all of a step's at unit
// density, a part of them for batches of every cell state, whose membrane rows
// are short and cell rows long (the rest of a step's follow in turns)
constexpr int kLeastTasks = 8, kLeastTasksGeneral = 3;
// Where the resident step is the faster one. A block walks its slots and its
// membrane terms; a step of the sequence costs its launches whatever the batch
// holds, and with every cell state as long as the longest row takes one
// thread. So the resident step gains `base` and `row` per candidate of that
// row, and loses `slot` per slot and `memb` per membrane particle of a block.
// Nanoseconds, fitted to 8,512 batches of one to 420 tissues with both routes
// timed (50-step runs); of 1,313 other ones two take the resident route and
// lose more than 2 % by it (2.4 at most), and of the fitted ones 1 % take the
// sequence and leave more than 5 %.
// With 144 membrane particles per block as the only limit, and none in batches
// of every state, 20 % lost more than 2 %, up to 2.5 times: 28 us a step
// against 22 for six tissues of 63,116 particles under triangular membranes
// (mixed), 118 against 99 for 105 small tissues of every state. (A rebuild
// costs a resident run more, 0.8 ns per particle, 5 with every state: of 3,046
// resident runs from a jittered start, which rebuild most, 8 % lose more than
// 2 %, up to 1.5 times in runs of four steps. Sizes do not tell how often a
// run rebuilds; a line for those runs would leave as much in the others.)
struct Gain {
  int32_t base, row, slot, memb;
};
// What a run saves once: its launches, eight against one (a call of one step
// near the line: 4 us, between 0 and 12).
constexpr int32_t kGainRun = 4000;
constexpr Gain kGain[2][2][2] = {  // [every state][triangular][mixed]
    {{{15000, 0, 16, 50}, {9800, 0, 10, 34}}, {{22800, 0, 31, 95}, {14200, 0, 15, 92}}},
    {{{20900, 350, 30, 55}, {17700, 300, 23, 43}}, {{27400, 335, 46, 97}, {21000, 300, 27, 94}}}};
// Turns that the membrane terms of a batch of every state may take.
constexpr int kMostTurns = 8;

}  // namespace

bool resident_plan(const TissueDev* T, int32_t ntissues, int64_t n, int precision, int max_cand,
                   int32_t nsteps, const LaunchCfg& lc, ResidentPlan* out) {
  if (n <= 0 || n > kResidentParticles) return false;
  ResidentPlan P{};
  // an even share of the particles over all SMs, one block each
  const int64_t share = ((n + lc.num_sms - 1) / lc.num_sms + kTile - 1) / kTile * kTile;
  P.slots = (int32_t)std::max<int64_t>(share, kLeastSlots);
  P.grid = (int32_t)((n + P.slots - 1) / P.slots);
  // the largest group whose particles are of kTissues tissues at most: more
  // tissues than that hold all of the ones between their first and last
  int64_t range = (int64_t)P.grid * P.slots;
  for (int32_t t = kTissues; t < ntissues; ++t)
    range = std::min<int64_t>(range, T[t].pbase - T[t - kTissues + 1].pbase + 1);
  P.group = (int32_t)std::max<int64_t>(range / P.slots, 1);
  // membrane particles of a block, group by group: the tiles that a tissue's
  // membrane touches, dealt round
  bool tri = false;
  int64_t membs = 0, most = 0, of = 0;
  double row = 0.0;  // membrane particles within reach of the largest cell
  for (int32_t t = 0; t < ntissues; ++t) {
    tri |= T[t].lattice == kLatticeTriangular;
    if (!T[t].nmemb) continue;
    const double reach = T[t].P.lj_thresh * (T[t].rmax_nm + T[t].rmax);
    row = std::max(row, 3.14159265 * reach * reach * T[t].nmemb / (T[t].lx * T[t].ly));
    const int64_t per = (int64_t)P.group * P.slots, end = T[t].pbase + T[t].nmemb;
    for (int64_t g = T[t].pbase / per; g <= (end - 1) / per; ++g) {
      if (g != of) membs = 0;
      of = g;
      const int64_t deal = std::min<int64_t>(P.group, P.grid - g * P.group);
      const int64_t lo = std::max<int64_t>(T[t].pbase, g * per), hi = std::min(end, (g + 1) * per);
      const int64_t tiles = (hi + kTile - 1) / kTile - lo / kTile;
      membs += (tiles + deal - 1) / deal * kTile;
      most = std::max(most, membs);
    }
  }
  P.membs = (int32_t)std::min<int64_t>(P.slots, most);
  const Gain& gain = kGain[lc.simple ? 0 : 1][tri ? 1 : 0][precision == 1 ? 1 : 0];
  if (gain.base + kGainRun / nsteps + gain.row * std::min(row, (double)max_cand) <
      (double)gain.slot * P.slots + (double)gain.memb * P.membs)
    return false;
  P.terms = tri ? kTriTerms : kSquareTerms + 2;
  P.turn = P.membs;
  auto bytes = [&](int tasks) {
    return precision == 1 ? Slots<float>::bytes(P.slots, P.membs, P.turn, tasks, P.terms)
                          : Slots<double>::bytes(P.slots, P.membs, P.turn, tasks, P.terms);
  };
  // room for the pair terms of all slots at 24 partners each, as far as it
  // goes, and for the longest row
  const int least =
      std::max(P.slots * (lc.simple ? kLeastTasks : kLeastTasksGeneral), max_cand);
  for (int turns = 2; !lc.simple && turns <= kMostTurns && bytes(least) > kSmemPerBlock; ++turns)
    P.turn = (P.membs + turns - 1) / turns;
  P.tasks = std::max(P.slots * 24, max_cand);
  while (P.tasks > least && bytes(P.tasks) > kSmemPerBlock) P.tasks -= std::min(64, P.tasks - least);
  P.smem = (int32_t)bytes(P.tasks);
  if (bytes(P.tasks) > kSmemPerBlock || P.slots > 4095) return false;
  *out = P;
  return true;
}

cudaError_t launch_resident(const DevState& S, const ResidentPlan& P, const TissueDev& first,
                            int32_t nsteps, int precision, const ResidentCfg& rc,
                            const LaunchCfg& lc, cudaStream_t s) {
  const bool one = S.ntissues == 1;
  int form;
  const void* kernel =
      precision == 1 ? (one ? kernel_of<float, true>(lc, &form) : kernel_of<float, false>(lc, &form))
                     : (one ? kernel_of<double, true>(lc, &form) : kernel_of<double, false>(lc, &form));
  cudaError_t e = cudaSuccess;
  if (!(*rc.sized >> form & 1u)) {  // once per context and form: a driver call
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSmemPerBlock);
    if (e != cudaSuccess) return e;
    *rc.sized |= 1u << form;
  }
  ResidentArgs A;
  A.nsteps = nsteps;
  A.slots = P.slots;
  A.membs = P.membs;
  A.turn = P.turn;
  A.tasks = P.tasks;
  A.terms = P.terms;
  A.group = P.group;
  A.thread_from = lc.search_switch;
  A.bar = reinterpret_cast<unsigned*>(rc.sync) + rc.runs->own();
  A.other = reinterpret_cast<unsigned*>(rc.sync) + rc.runs->next();
  A.abort = rc.sync + 2;
  A.flags = rc.sync + 3;
  A.polls = rc.polls;
  A.post = rc.post;
  A.per_step = rc.per_step;
  A.per_pair = rc.per_pair;
  A.per_rebuild = rc.per_rebuild;
  A.hist = rc.hist;
  DevState S1 = S;
  TissueDev T0 = first;
  void* args[] = {&S1, &A, &T0};
  e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)P.grid), dim3((unsigned)kThreads), args,
                                  (size_t)P.smem, s);
  if (e == cudaSuccess) ++rc.runs->launched;
  return e;
}

}  // namespace epi
