// Candidate rebuild of the flagged tissues, as device functions a kernel of
// any grid calls: the work list, binning, the per-tissue scan, the counting
// sort and the candidate search. The kernels of the step sequence run one of
// them each; the resident kernel runs them between grid barriers.
#pragma once
#include "epi_device.cuh"

namespace epi {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = kScanTile / kScanThreads;  // 8

__device__ __forceinline__ int32_t warp_incl_scan(int32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Block-wide exclusive scan of one value per thread over NT threads (a multiple
// of 32, at most 1024); returns the prefix and writes the block total to *total.
template <int NT>
__device__ __forceinline__ int32_t block_excl_scan(int32_t v, int32_t* total) {
  __shared__ int32_t wsum[NT / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int32_t incl = warp_incl_scan(v);
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int32_t w = lane < NT / 32 ? wsum[lane] : 0;
    w = warp_incl_scan(w);
    if (lane < NT / 32) wsum[lane] = w;
  }
  __syncthreads();
  const int32_t before = wid == 0 ? 0 : wsum[wid - 1];
  *total = wsum[NT / 32 - 1];
  __syncthreads();
  return before + incl - v;
}

// ---------------------------------------------------------------------------
// Reference grid checks: grid_init's bin (cell_connection.cpp:44-53) and the
// range assert of connect_proc (:95-99). Returns the tissue-local bin or -1.
// ---------------------------------------------------------------------------
// (int)(v / AREA_GRID) of the IEEE division, by a multiplication wherever the
// quotient is not within 1e-9 of an integer.
__device__ __forceinline__ int32_t grid_index(double v) {
  const double q = v * (1.0 / kAreaGrid);
  const int32_t k = (int32_t)q;
  const double f = q - (double)k;
  return f > 1e-9 && f < 1.0 - 1e-9 ? k : (int32_t)(v / kAreaGrid);
}
__device__ __forceinline__ int32_t ref_bin(const TissueDev& T, double x, double y, double z,
                                           bool memb) {
  const int32_t aix = grid_index(0.5 * T.lx - pdiff(0.5 * T.lx, x, T.lx));
  const int32_t aiy = grid_index(0.5 * T.ly - pdiff(0.5 * T.ly, y, T.ly));
  const int32_t aiz = grid_index(fmax(z, 0.0));  // min0, utils.h:55-57
  bool bad = aix >= T.anx || aiy >= T.any || aiz >= T.anz || aix < 0 || aiy < 0 || aiz < 0;
  if (!memb) {
    const int32_t cx = grid_index(x), cy = grid_index(y), cz = grid_index(z);
    bad |= cx >= T.anx || cy >= T.any || cz >= T.anz || cx < 0 || cy < 0 || cz < 0;
  }
  return bad ? -1 : (aix * T.any + aiy) * T.anz + aiz;
}

// ---------------------------------------------------------------------------
// Rebuild work list. k_gate_compact lists the gated tissues of [t0, t1) with
// prefix sums of their particle and bin counts; every other rebuild kernel
// then strides over the gated particles (or bins) only, mapping a running
// index back to (tissue, local index) by binary search in the prefix sums.
// With nothing gated the list is empty and each kernel exits at once.
// ---------------------------------------------------------------------------
// Run by one block of NT threads. any: the "some tissue" word. clear (whole
// batch): gate[0] is cleared once the list is built; the step sets it again
// for the next step.
template <int NT>
__device__ __forceinline__ void gate_compact(const DevState& S, int32_t t0, int32_t t1, bool any,
                                             bool clear) {
  if (!any) {
    if (threadIdx.x == 0) {
      S.rl_count[0] = 0;
      S.rl_ppre[0] = 0;
      S.rl_bpre[0] = 0;
    }
    return;
  }
  if (t1 - t0 == 1) {  // one tissue: no scan
    if (threadIdx.x == 0) {
      const TissueDev& T = S.tissues[t0];
      const bool g = S.gate[1 + t0] != 0;
      if (clear) S.gate[0] = 0;
      S.rl_count[0] = g ? 1 : 0;
      S.rl_list[0] = t0;
      S.rl_ppre[0] = S.rl_bpre[0] = 0;
      S.rl_ppre[g ? 1 : 0] = g ? T.n : 0;
      S.rl_bpre[g ? 1 : 0] = g ? T.anx * T.any * T.anz : 0;
    }
    return;
  }
  __syncthreads();  // every thread has read the word before it is cleared
  if (clear && threadIdx.x == 0) S.gate[0] = 0;
  int32_t cc = 0, cp = 0, cb = 0;
  for (int32_t base = t0; base < t1; base += NT) {
    const int32_t t = base + threadIdx.x;
    const bool g = t < t1 && S.gate[1 + t] != 0;
    int32_t np = 0, nb = 0;
    if (g) {
      const TissueDev& T = S.tissues[t];
      np = T.n;
      nb = T.anx * T.any * T.anz;
    }
    int32_t tc, tp, tb;
    const int32_t oc = block_excl_scan<NT>(g ? 1 : 0, &tc);
    const int32_t op = block_excl_scan<NT>(np, &tp);
    const int32_t ob = block_excl_scan<NT>(nb, &tb);
    if (g) {
      S.rl_list[cc + oc] = t;
      S.rl_ppre[cc + oc] = cp + op;
      S.rl_bpre[cc + oc] = cb + ob;
    }
    cc += tc;
    cp += tp;
    cb += tb;
  }
  if (threadIdx.x == 0) {
    S.rl_count[0] = cc;
    S.rl_ppre[cc] = cp;
    S.rl_bpre[cc] = cb;
  }
}

// Once the work list is built nothing of the rebuild reads the flags: clear
// the listed tissues' flags and count the rebuilds. Run by one block of the
// candidate search. (gate_compact cleared the "some tissue" word.)
__device__ __forceinline__ void gate_clear(const DevState& S, int32_t cnt) {
  for (int32_t k = threadIdx.x; k < cnt; k += blockDim.x) S.gate[1 + S.rl_list[k]] = 0;
  if (threadIdx.x == 0 && cnt) atomicAdd(S.rebuilds, (unsigned long long)cnt);
}

// index k of the last prefix entry <= g (pre[0] = 0, non-decreasing, n+1 entries)
__device__ __forceinline__ int32_t locate(const int32_t* pre, int32_t n, int32_t g) {
  int32_t lo = 0, hi = n;  // answer in [lo, hi)
  while (hi - lo > 1) {
    const int32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Gated particle g -> global particle index (and its tissue).
__device__ __forceinline__ int32_t gated_particle(const DevState& S, int32_t cnt, int32_t g,
                                                  int32_t* tissue) {
  const int32_t k = locate(S.rl_ppre, cnt, g);
  const int32_t t = S.rl_list[k];
  *tissue = t;
  return S.tissues[t].pbase + (g - S.rl_ppre[k]);
}

#define GATED_PARTICLES(g, cnt)                                                        \
  const int32_t cnt = S.rl_count[0];                                                   \
  if (cnt == 0) return;                                                                \
  const int32_t ngated_ = S.rl_ppre[cnt];                                              \
  for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngated_;                 \
       g += gridDim.x * blockDim.x)

// Binning on the reference's 2.0 grid (grid_init, cell_connection.cpp:38-62).
__device__ __forceinline__ void rebuild_bin(const DevState& S) {
  GATED_PARTICLES(g, cnt) {
    int32_t t;
    const int32_t i = gated_particle(S, cnt, g, &t);
    const TissueDev& T = S.tissues[t];
    const double4 p = S.pos_cur[i];
    if (!isfinite(p.x) || !isfinite(p.y) || !isfinite(p.z)) {
      raise_error(S.status, E_NONFINITE, i, -1, p.x);
      S.bin[i] = -1;
      continue;
    }
    const int32_t lb = ref_bin(T, p.x, p.y, p.z, attr_state(S.attr[i]) == ST_MEMB);
    if (lb < 0) {
      raise_error(S.status, E_BIN_RANGE, i, -1, p.z);
      S.bin[i] = -1;
      continue;
    }
    const int32_t b = T.binbase + lb;
    const int32_t rk = atomicAdd(&S.counts[b], 1);
    if (rk + 1 >= kBinCap) raise_error(S.status, E_BIN_OVERFLOW, i, b, (double)(rk + 1));
    S.bin[i] = b;
    S.rank[i] = rk;
  }
}

// Exclusive scan of the bin counts of every listed tissue into starts, offset
// by the tissue's first particle, so each tissue's sorted particles occupy
// its own slots [pbase, pbase + n). Each tissue's bins end with a sentinel
// entry that receives the end offset. A tissue's bins are cut into chunks
// (S.scan_chunks for the batch's largest tissue), a block each: it sums the
// counts before its chunk, then scans the chunk, NT threads 8 NT bins at a
// time. Cutting costs reads (of chunks before one's own) and saves the
// serial chain: 262,144 bins took one block 192 us, now 20.
template <int NT>
__device__ __forceinline__ void rebuild_scan(const DevState& S) {
  const int32_t cnt = S.rl_count[0];
  __shared__ int32_t s_sum[NT / 32];
  for (int32_t u = blockIdx.x; u < cnt * S.scan_chunks; u += gridDim.x) {
    const int32_t k = u / S.scan_chunks, c = u - k * S.scan_chunks;
    const TissueDev& T = S.tissues[S.rl_list[k]];
    const int32_t nb = T.anx * T.any * T.anz;
    const int32_t lo = c * S.scan_bins;
    if (lo >= nb) continue;
    const int32_t hi = lo + S.scan_bins < nb ? lo + S.scan_bins : nb;
    const int32_t* in = S.counts + T.binbase;
    int32_t* out = S.starts + T.binbase;
    // binbase and lo are multiples of four
    int32_t before = 0;
    for (int32_t b = 4 * (int32_t)threadIdx.x; b < lo; b += 4 * NT) {
      const int4 v = *reinterpret_cast<const int4*>(in + b);
      before += (v.x + v.y) + (v.z + v.w);
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = before;
    __syncthreads();
    int32_t carry = T.pbase;
    for (int w = 0; w < NT / 32; ++w) carry += s_sum[w];
    constexpr int32_t kTile = NT * kScanItems;
    for (int32_t base = lo; base < hi; base += kTile) {
      const int32_t b0 = base + threadIdx.x * kScanItems;
      int32_t v[kScanItems];
      int32_t sum = 0;
#pragma unroll
      for (int q = 0; q < kScanItems; ++q) {
        v[q] = b0 + q < hi ? in[b0 + q] : 0;
        sum += v[q];
      }
      int32_t tot;
      int32_t run = carry + block_excl_scan<NT>(sum, &tot);
#pragma unroll
      for (int q = 0; q < kScanItems; ++q) {
        if (b0 + q < hi) out[b0 + q] = run;
        run += v[q];
      }
      carry += tot;
    }
    if (hi == nb && threadIdx.x == 0) out[nb] = carry;
    __syncthreads();
  }
}

__device__ __forceinline__ void rebuild_scatter(const DevState& S) {
  GATED_PARTICLES(g, cnt) {
    int32_t t;
    const int32_t i = gated_particle(S, cnt, g, &t);
    const int32_t b = S.bin[i];
    if (b < 0) continue;
    const int32_t slot = S.starts[b] + S.rank[i];
    if (!EPI_CHECKED(slot >= S.tissues[t].pbase && slot < S.tissues[t].pbase + S.tissues[t].n,
                     S.status, i, slot))
      continue;
    S.skey[slot] = (uint32_t)i;
  }
}

// One sorted particle: its slot, the membrane tag and the FP32 copy of its
// position (x and y as grid_init bins them, in [0, L)).
__device__ __forceinline__ void place_particle(const DevState& S, const TissueDev& T, int32_t s,
                                               uint32_t gi) {
  if (!EPI_CHECKED(gi >= (uint32_t)T.pbase && gi < (uint32_t)(T.pbase + T.n), S.status,
                   (int32_t)gi, s))
    return;
  const bool memb = attr_state(S.attr[gi]) == ST_MEMB;
  S.skey[s] = gi | (memb ? 0x80000000u : 0u);
  S.rank[gi] = s;  // the particle's slot from here on (the search skips it)
  // x and y as grid_init bins them (ref_bin): in [0, L); w: LJ_THRESH *
  // radius, negative for a membrane particle (the search's reach and its
  // membrane test)
  const double4 pg = S.pos_cur[gi];
  const double xc = 0.5 * T.lx - pdiff(0.5 * T.lx, pg.x, T.lx);
  const double yc = 0.5 * T.ly - pdiff(0.5 * T.ly, pg.y, T.ly);
  const float lw = (float)(T.P.lj_thresh * pg.w);
  S.spos[s] = make_float4((float)xc, (float)yc, (float)pg.z, memb ? -lw : lw);
}

// Sorts every bin's particles by index -- the deterministic order the
// candidate search emits them in -- and writes the sorted FP32 copy the
// search streams through. Eight lanes per bin: a lane holds every eighth
// particle of it (a bin of 2.0 holds about six at unit density), finds its
// rank by counting smaller indices and places it; bins of more than 32 are
// sorted in place by one lane. 1.1M particles: 71 us with a thread per bin,
// now 45.
constexpr int kBinLanes = 8;
__device__ __forceinline__ void rebuild_sort(const DevState& S) {
  const int32_t cnt = S.rl_count[0];
  if (cnt == 0) return;
  const int32_t nbg = S.rl_bpre[cnt];
  const int sub = (int)threadIdx.x & (kBinLanes - 1), grp = ((int)threadIdx.x & 31) / kBinLanes;
  constexpr int kBins = 32 / kBinLanes;  // bins per warp, in step with each other
  const int32_t warps = (int32_t)((gridDim.x * blockDim.x) >> 5);
  for (int32_t w = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w * kBins < nbg;
       w += warps) {
    const int32_t g = w * kBins + grp;
    int32_t s0 = 0, m = 0;
    const TissueDev* T = S.tissues;
    if (g < nbg) {
      const int32_t k = locate(S.rl_bpre, cnt, g);
      T = S.tissues + S.rl_list[k];
      const int32_t b = T->binbase + (g - S.rl_bpre[k]);
      s0 = S.starts[b];
      m = S.starts[b + 1] - s0;
      if (m > 0 && sub == 0) S.counts[b] = 0;  // ready for the next binning
    }
    if (m > 4 * kBinLanes) {
      if (sub == 0) {
        for (int32_t s = s0 + 1; s < s0 + m; ++s) {
          const uint32_t v = S.skey[s];
          int32_t q = s - 1;
          while (q >= s0 && S.skey[q] > v) {
            S.skey[q + 1] = S.skey[q];
            --q;
          }
          S.skey[q + 1] = v;
        }
        for (int32_t s = s0; s < s0 + m; ++s) place_particle(S, *T, s, S.skey[s]);
      }
      m = 0;
    }
    __syncwarp();
    const int32_t most = __reduce_max_sync(0xffffffffu, m);
    uint32_t own[4];
    int32_t rank[4] = {0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int32_t e = u * kBinLanes + sub;
      own[u] = e < m ? S.skey[s0 + e] : 0xffffffffu;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u * kBinLanes >= most) break;
#pragma unroll
      for (int l = 0; l < kBinLanes; ++l) {
        const uint32_t o = __shfl_sync(0xffffffffu, own[u], l, kBinLanes);
#pragma unroll
        for (int v = 0; v < 4; ++v) rank[v] += o < own[v] ? 1 : 0;
      }
    }
    // (the shuffles keep every read of a key ahead of its replacement)
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u * kBinLanes + sub < m) place_particle(S, *T, s0 + rank[u], own[u]);
  }
}

// Bin ranges (inclusive) of the periodic window [x-R, x+R] along one axis:
// at most two ranges, because the window may wrap once. Bin k holds
// [k*AG, (k+1)*AG) of [0, L) (the last one is shortened; AG*AN > L).
// off[r]: the image of range r's particles nearest to x is their binned
// coordinate + off[r] (0, or +-L for the wrapped part of a split window).
__device__ __forceinline__ int window_ranges(double x, double R, double L, int32_t an,
                                             int32_t lo[2], int32_t hi[2], double off[2]) {
  off[0] = off[1] = 0.0;
  if (2.0 * R >= L) {
    lo[0] = 0;
    hi[0] = an - 1;
    return 1;
  }
  // floor(v / AG) through a multiply; the caller's window already carries a
  // margin far wider than the rounding difference.
  auto bin_of = [&](double v) {
    int32_t k = (int32_t)floor(v * (1.0 / kAreaGrid));
    return k < 0 ? 0 : (k > an - 1 ? an - 1 : k);
  };
  const double a = x - R, b = x + R;
  if (a < 0.0) {
    lo[0] = 0; hi[0] = bin_of(b);
    lo[1] = bin_of(a + L); hi[1] = an - 1;
    off[1] = -L;
    if (lo[1] <= hi[0]) { hi[0] = an - 1; return 1; }
    return 2;
  }
  if (b >= L) {
    lo[0] = bin_of(a); hi[0] = an - 1;
    lo[1] = 0; hi[1] = bin_of(b - L);
    off[1] = L;
    if (hi[1] >= lo[0]) { lo[0] = 0; return 1; }
    return 2;
  }
  lo[0] = bin_of(a);
  hi[0] = bin_of(b);
  return 1;
}

// Candidate search of a gated tissue: every partner within
// LJ_THRESH*(r_i+r_j) + skin (membrane pairs excluded: connect_proc only
// iterates non-membrane cells, cell_connection.cpp:93). The window covers
// every bin that can hold such a partner; the reference's fixed 5x5x5 window
// is a superset for every pair it can connect (reach <= 1.2 * 3.2 < 2 * 2.0).
// Candidates come out in column order (x ranges outer, y ranges inner), slot
// order within a column: deterministic after k_binsort.
// Slot positions are the grid's canonical [0, L) coordinates, so every
// particle of a window's x (or y) range has the same nearest image: the
// range's offset is folded into the particle's own coordinate (pxe, pye)
// and no per-slot wrap is needed. Boxes below 2 (R + AG) keep the per-slot
// minimum image (wrap_x, wrap_y): there an edge bin may hold the other image.
struct SearchWindow {
  int32_t xlo[2], xhi[2], ylo[2], yhi[2];
  int nxr, nyr;
  int32_t z0, z1;
  float pxe[2], pye[2], pz, flx, fly, fhx, fhy;
  float rw;        // LJ_THRESH * r_i + skin + margin: the reach less the partner's share
  float memb_lim;  // slots whose w lies below it are excluded (membrane pairs)
  int32_t s_self;  // the particle's own slot (-1: none)
  bool memb_i, wrap_x, wrap_y;

  __device__ __forceinline__ SearchWindow(const DevState& S, const TissueDev& T, int32_t i) {
    constexpr double kInvAG = 1.0 / kAreaGrid;
    memb_i = attr_state(S.attr[i]) == ST_MEMB;
    const double4 p = S.pos_cur[i];
    const double lt = T.P.lj_thresh;
    const double skin = S.skin;
    // Candidates are compared in float: the margin covers the rounding of
    // float coordinates up to the box size (and the window widens with it).
    const double margin = 1e-4 + 5e-7 * (T.lx > T.ly ? T.lx : T.ly) + 5e-7 * T.lz;
    const double R = lt * (p.w + (memb_i ? T.rmax_nm : T.rmax)) + skin + margin + 1e-6;
    double offx[2], offy[2];
    nxr = window_ranges(p.x, R, T.lx, T.anx, xlo, xhi, offx);
    nyr = window_ranges(p.y, R, T.ly, T.any, ylo, yhi, offy);
    wrap_x = !(T.lx > 2.0 * (R + kAreaGrid));
    wrap_y = !(T.ly > 2.0 * (R + kAreaGrid));
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      pxe[r] = (float)(wrap_x ? p.x : p.x - offx[r]);
      pye[r] = (float)(wrap_y ? p.y : p.y - offy[r]);
    }
    // z bins are floor(max(z, 0) / AG) (ref_bin); the margin in R covers the
    // multiply-for-divide rounding, so [z - R, z + R] needs no extra bins
    z0 = (int32_t)floor((p.z - R) * kInvAG);
    z1 = (int32_t)floor((p.z + R) * kInvAG);
    z0 = z0 < 0 ? 0 : (z0 > T.anz - 1 ? T.anz - 1 : z0);
    z1 = z1 < 0 ? 0 : (z1 > T.anz - 1 ? T.anz - 1 : z1);
    pz = (float)p.z;
    flx = (float)T.lx;
    fly = (float)T.ly;
    fhx = 0.5f * flx;
    fhy = 0.5f * fly;
    rw = (float)(lt * p.w + skin + margin);
    memb_lim = memb_i ? 0.f : -INFINITY;
    s_self = S.bin[i] < 0 ? -1 : S.rank[i];
  }
  // Is the particle in slot s (FP32 copy q) of a column of x range xr and y
  // range yr a candidate of i? (ex, ey: pxe[xr], pye[yr]) The reach
  // rw + |q.w| rounds differently from LJ_THRESH (r_i + r_j) + skin by a few
  // ulps, far inside the margin, so the candidates still hold every pair
  // that can be connected. kWrap = false: only for windows with neither
  // wrap_x nor wrap_y.
  template <bool kWrap>
  __device__ __forceinline__ bool hit(int32_t s, const float4& q, float ex, float ey) const {
    if (s == s_self || q.w < memb_lim) return false;
    float dx = ex - q.x, dy = ey - q.y;
    if (kWrap && wrap_x) dx = dx > fhx ? dx - flx : (dx <= -fhx ? dx + flx : dx);
    if (kWrap && wrap_y) dy = dy > fhy ? dy - fly : (dy <= -fhy ? dy + fly : dy);
    const float dz = pz - q.z;
    const float reach = rw + fabsf(q.w);
    return dx * dx + dy * dy + dz * dz <= reach * reach;
  }
};

__device__ __forceinline__ void finish_search(const DevState& S, int32_t i, int32_t count) {
  const int32_t cap = S.max_cand;
  if (count > cap) raise_error(S.status, E_LIST_OVERFLOW, i, -1, (double)count);
  cand_set(S, i, 0, (uint32_t)(count < cap ? count : cap));
  const double4 p = S.pos_cur[i];
  S.bpos[i] = make_float4((float)p.x, (float)p.y, (float)p.z, 0.f);
}

// Few gated particles (a tissue or two): G lanes per particle, so the GPU has
// work for all its warps. The group's lanes fetch the slot ranges of G bin
// columns at a time; a scan within the group lays the ranges end to end, the
// group sweeps the concatenation G slots at a time, and ballots keep the slot
// order. The groups of a warp run in step (to the longest of their loops):
// left to their own lengths they ran one after the other.
template <int G>
__device__ __forceinline__ void cand_search_groups(const DevState& S, int32_t cnt,
                                                   int32_t ngated) {
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "group of 4 to 32 lanes");
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1);          // lane within the group
  const int gbase = lane & ~(G - 1);      // the group's first lane
  const unsigned gmask = G == 32 ? kAll : (1u << G) - 1u;
  const unsigned lt_mask = (1u << gl) - 1u;
  const int32_t groups = (gridDim.x * blockDim.x) / G;
  const int32_t cap = S.max_cand;
  for (int32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / G; g - gbase / G < ngated;
       g += groups) {
    // a group past the end repeats the last particle and writes nothing
    const bool in = g < ngated;
    int32_t t;
    const int32_t i = gated_particle(S, cnt, in ? g : ngated - 1, &t);
    const TissueDev& T = S.tissues[t];
    const SearchWindow W(S, T, i);
    const int32_t nx0 = W.xhi[0] - W.xlo[0] + 1, ny0 = W.yhi[0] - W.ylo[0] + 1;
    const int32_t ncx = nx0 + (W.nxr > 1 ? W.xhi[1] - W.xlo[1] + 1 : 0);
    const int32_t ncy = ny0 + (W.nyr > 1 ? W.yhi[1] - W.ylo[1] + 1 : 0);
    const int32_t ncol = ncx * ncy;  // column c = cx * ncy + cy
    const int32_t most_col = G == 32 ? ncol : __reduce_max_sync(kAll, ncol);
    int32_t count = 0;
    for (int32_t c0 = 0; c0 < most_col; c0 += G) {
      const int32_t c = c0 + gl;
      int32_t lo = 0, len = 0;
      float cex = 0.f, cey = 0.f;
      if (c < ncol) {
        const int32_t cx = c / ncy, cy = c - cx * ncy;
        cex = cx < nx0 ? W.pxe[0] : W.pxe[1];
        cey = cy < ny0 ? W.pye[0] : W.pye[1];
        const int32_t bx = cx < nx0 ? W.xlo[0] + cx : W.xlo[1] + (cx - nx0);
        const int32_t by = cy < ny0 ? W.ylo[0] + cy : W.ylo[1] + (cy - ny0);
        const int32_t col = T.binbase + (bx * T.any + by) * T.anz;
        lo = S.starts[col + W.z0];
        len = S.starts[col + W.z1 + 1] - lo;
      }
      int32_t incl = len;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const int32_t v = __shfl_up_sync(kAll, incl, o, G);
        if (gl >= o) incl += v;
      }
      const int32_t excl = incl - len;
      const int32_t total = __shfl_sync(kAll, incl, G - 1, G);
      const int32_t most = G == 32 ? total : __reduce_max_sync(kAll, total);
      for (int32_t base = 0; base < most; base += G) {
        const int32_t f = base + gl;
        // the last column whose range starts at or before f (k + step <= G - 1)
        int32_t k = 0;
#pragma unroll
        for (int32_t step = G / 2; step > 0; step >>= 1) {
          const int32_t e = __shfl_sync(kAll, excl, k + step, G);
          if (e <= f) k += step;
        }
        const int32_t s = __shfl_sync(kAll, lo, k, G) + (f - __shfl_sync(kAll, excl, k, G));
        const float ex = __shfl_sync(kAll, cex, k, G), ey = __shfl_sync(kAll, cey, k, G);
        bool hit = false;
        uint32_t key = 0;
        if (f < total) {
          key = S.skey[s];
          hit = W.hit<true>(s, S.spos[s], ex, ey);
        }
        const unsigned m = (__ballot_sync(kAll, hit) >> gbase) & gmask;
        if (hit && in) {
          const int32_t kk = count + __popc(m & lt_mask);
          if (kk < cap) cand_set(S, i, kk + 1, (key & 0x7fffffffu) - (uint32_t)T.pbase);
        }
        count += __popc(m);
      }
    }
    if (gl == 0 && in) finish_search(S, i, count);
  }
}

// A thread's candidate row written a whole 16-byte chunk at a time: entries
// are shifted into a register chunk from the top (the oldest reaches slot 0
// after a chunk's worth of entries) and the chunk is stored when full or at
// the end. Chunk 0 starts with a zero in the count slot; the caller stores
// the count afterwards.
template <bool k16>
struct RowWriter {
  static constexpr int kPer = k16 ? 8 : 4;  // entries per chunk
  uint32_t w0 = 0, w1 = 0, w2 = 0, w3 = 0;
  int32_t e = 1;  // next entry (entry 0 is the count)
  __device__ __forceinline__ void shift_in(uint32_t v) {
    if (k16) {
      w0 = __funnelshift_r(w0, w1, 16);
      w1 = __funnelshift_r(w1, w2, 16);
      w2 = __funnelshift_r(w2, w3, 16);
      w3 = __funnelshift_r(w3, v, 16);
    } else {
      w0 = w1;
      w1 = w2;
      w2 = w3;
      w3 = v;
    }
  }
  __device__ __forceinline__ void put(const DevState& S, int64_t i, uint32_t v) {
    if (!EPI_CHECKED(!k16 || v < 65536u, S.status, (int32_t)i, e)) return;
    shift_in(v);
    ++e;
    if ((e & (kPer - 1)) == 0)
      S.cand[(int64_t)(e / kPer - 1) * S.n_total + i] = make_uint4(w0, w1, w2, w3);
  }
  __device__ __forceinline__ void close(const DevState& S, int64_t i) {
    const int n = e & (kPer - 1);
    if (n == 0) return;
    for (int k = n; k < kPer; ++k) shift_in(0u);
    S.cand[(int64_t)(e / kPer) * S.n_total + i] = make_uint4(w0, w1, w2, w3);
  }
};

// One particle's candidate search by one thread. The window's columns
// (x ranges outer, y ranges inner) are walked as one flat sequence of
// slots, two per iteration: a lane moves on to its next column whenever it
// has used up the current one, so the lanes of a warp stay in step however
// their columns' slot counts differ. Each column's slot range is fetched one
// column ahead, so opening a column waits on no load. kWrap: the box is too
// small for the folded images (per-slot minimum image).
template <bool k16, bool kWrap>
__device__ __forceinline__ void search_particle(const DevState& S, const TissueDev& T,
                                                const SearchWindow& W, int32_t i) {
  constexpr int kWide = 2;  // slots in flight (four: 0.076 against 0.065 ms per step)
  const int32_t cap = S.max_cand;
  const int32_t nx0 = W.xhi[0] - W.xlo[0] + 1, ny0 = W.yhi[0] - W.ylo[0] + 1;
  const int32_t ncx = nx0 + (W.nxr > 1 ? W.xhi[1] - W.xlo[1] + 1 : 0);
  const int32_t ncy = ny0 + (W.nyr > 1 ? W.yhi[1] - W.ylo[1] + 1 : 0);
  const int32_t any = T.any, anz = T.anz, binbase = T.binbase;
  const uint32_t pbase = (uint32_t)T.pbase;
  RowWriter<k16> row;
  int32_t count = 0;
  // the column after the current one: its slot range and folded coordinates
  int32_t cx = 0, cy = 0;  // the column to fetch next
  int32_t ns = 0, nhi = 0;
  float nex = 0.f, ney = 0.f;
  bool nvalid = false;
  auto fetch = [&]() {
    nvalid = cx < ncx;
    if (!nvalid) return;
    const int32_t bx = cx < nx0 ? W.xlo[0] + cx : W.xlo[1] + (cx - nx0);
    const int32_t by = cy < ny0 ? W.ylo[0] + cy : W.ylo[1] + (cy - ny0);
    nex = cx < nx0 ? W.pxe[0] : W.pxe[1];
    ney = cy < ny0 ? W.pye[0] : W.pye[1];
    const int32_t col = binbase + (bx * any + by) * anz;
    ns = S.starts[col + W.z0];
    nhi = S.starts[col + W.z1 + 1];
    if (++cy == ncy) {
      cy = 0;
      ++cx;
    }
  };
  fetch();
  int32_t s = 0, s_hi = 0;
  float ex = 0.f, ey = 0.f;
  for (;;) {
    bool live = true;
    while (s >= s_hi) {  // open the next column
      if (!nvalid) {
        live = false;
        break;
      }
      s = ns;
      s_hi = nhi;
      ex = nex;
      ey = ney;
      fetch();
    }
    if (!live) break;
    uint32_t key[kWide];
    float4 q[kWide];
#pragma unroll
    for (int u = 0; u < kWide; ++u) {
      key[u] = s + u < s_hi ? S.skey[s + u] : 0u;
      q[u] = s + u < s_hi ? S.spos[s + u] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kWide; ++u) {
      if (s + u < s_hi && W.template hit<kWrap>(s + u, q[u], ex, ey)) {
        if (count < cap) row.put(S, i, (key[u] & 0x7fffffffu) - pbase);
        ++count;
      }
    }
    s += kWide;
  }
  row.close(S, i);
  finish_search(S, i, count);
}

// Many gated particles: one thread per particle (about a hundred slots each:
// bins of 2.0 hold about six particles); a warp keeps 32 particles in flight
// and writes the column-major candidate rows coalesced.
template <bool k16>
__device__ __forceinline__ void cand_search_threads(const DevState& S, int32_t cnt,
                                                    int32_t ngated) {
  for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngated;
       g += gridDim.x * blockDim.x) {
    int32_t t;
    const int32_t i = gated_particle(S, cnt, g, &t);
    const TissueDev& T = S.tissues[t];
    const SearchWindow W(S, T, i);
    if (W.wrap_x || W.wrap_y) search_particle<k16, true>(S, T, W, i);
    else search_particle<k16, false>(S, T, W, i);
  }
}

// Below `thread_from` gated particles several lanes per particle search (which
// keeps the GPU busy with few particles): a warp, or as many lanes, at least
// four, as leave every particle a group of its own; from there on one thread
// per particle. All emit every row in the same order.
template <bool k16>
__device__ __forceinline__ void rebuild_search(const DevState& S, int32_t thread_from) {
  const int32_t cnt = S.rl_count[0];
  if (blockIdx.x == 0) gate_clear(S, cnt);
  if (cnt == 0) return;
  const int32_t ngated = S.rl_ppre[cnt];
  const int64_t threads = (int64_t)gridDim.x * blockDim.x;
  if (ngated >= thread_from) cand_search_threads<k16>(S, cnt, ngated);
  else if ((int64_t)ngated * 32 <= threads) cand_search_groups<32>(S, cnt, ngated);
  else if ((int64_t)ngated * 16 <= threads) cand_search_groups<16>(S, cnt, ngated);
  else if ((int64_t)ngated * 8 <= threads) cand_search_groups<8>(S, cnt, ngated);
  else cand_search_groups<4>(S, cnt, ngated);
}

}  // namespace
}  // namespace epi
