// The forces of one particle: membrane bending, lattice springs and wall
// (memb_force and its terms), and the pair laws with the commit (Particle).
// Shared by the kernels that give a particle a thread and by the resident
// kernel, which gives it several lanes; every operation's rounding is written
// out (xmul, xadd, xfma), so all of them get the same bits.
#pragma once
#include <type_traits>

#include "epi_device.cuh"

namespace epi {

#ifdef EPI_CHECK
constexpr bool kCheck = true;
#else
constexpr bool kCheck = false;
#endif

namespace {

// rintf(v) for |v| <= 2^22 on the FMA pipe: adding and subtracting
// 1.5 * 2^23 rounds v to the nearest integer (ties to even) exactly.
__device__ __forceinline__ float rint_fma(float v) {
  return __fsub_rn(__fadd_rn(v, 12582912.f), 12582912.f);
}

// Minimum image of the difference f as f - L rint(f / L) (il = 1 / L): four
// FMA-pipe instructions, no branch.
__device__ __forceinline__ float wrap_f(float f, float L, float il) {
  return xfma(-L, rint_fma(xmul(f, il)), f);
}

// Offsets of lattice neighbours from membrane particle i (minimum image): from
// the FP64 positions in the FP64 path, from the FP32 copies in the mixed path.
template <typename R>
struct SiteOffsets;
template <>
struct SiteOffsets<double> {
  using Pos = double4;
  const DevState& S;
  const double4 p;
  const TissueDev& T;
  __device__ __forceinline__ SiteOffsets(const DevState& S_, const double4& p_, const TissueDev& T_)
      : S(S_), p(p_), T(T_) {}
  static __device__ __forceinline__ double4 own(const DevState&, int32_t, const double4& p) {
    return p;
  }
  __device__ __forceinline__ double4 at(int32_t q) const { return S.pos_cur[q]; }
  __device__ __forceinline__ Vec3<double> from(const double4& o) const {
    return offset_of<double>(o, p, T);
  }
  __device__ __forceinline__ Vec3<double> operator()(int32_t q) const { return from(at(q)); }
};
template <>
struct SiteOffsets<float> {
  using Pos = float4;
  const DevState& S;
  const float4 p;
  const TissueDev& T;
  __device__ __forceinline__ SiteOffsets(const DevState& S_, const float4& p_, const TissueDev& T_)
      : S(S_), p(p_), T(T_) {}
  static __device__ __forceinline__ float4 own(const DevState& S, int32_t i, const double4&) {
    return S.posf_cur[i];
  }
  __device__ __forceinline__ float4 at(int32_t q) const { return S.posf_cur[q]; }
  // minimum image as d - L rint(d / L): lattice neighbours lie far closer
  // than L/2, where it equals the compare-and-shift form
  __device__ __forceinline__ Vec3<float> from(const float4& o) const {
    return Vec3<float>{wrap_f(xsub(o.x, p.x), T.lxf, T.ilxf),
                       wrap_f(xsub(o.y, p.y), T.lyf, T.ilyf), xsub(o.z, p.z)};
  }
  __device__ __forceinline__ Vec3<float> operator()(int32_t q) const { return from(at(q)); }
};

// _memb_bend_diff_factor with NEW_BEND_POT (cell_interaction.cpp:349-360)
template <typename R>
__device__ __forceinline__ R bend_factor(R c) {
  if (c >= R(0)) return xsub(R(1), c);
  const R e = xadd(R(1), c);
  return R(1) / xmul(e, e);
}

template <typename R>
__device__ __forceinline__ Vec3<R> v3_cross(const Vec3<R>& a, const Vec3<R>& b) {
  return Vec3<R>{xfma(a.y, b.z, -xmul(a.z, b.y)), xfma(a.z, b.x, -xmul(a.x, b.z)),
                 xfma(a.x, b.y, -xmul(a.y, b.x))};
}
template <typename R>
__device__ __forceinline__ Vec3<R> v3_sub(const Vec3<R>& a, const Vec3<R>& b) {
  return Vec3<R>{xsub(a.x, b.x), xsub(a.y, b.y), xsub(a.z, b.z)};
}
template <typename R>
__device__ __forceinline__ Vec3<R> v3_neg(const Vec3<R>& a) { return Vec3<R>{-a.x, -a.y, -a.z}; }
template <typename R>
__device__ __forceinline__ Vec3<R> v3_axpy(R s, const Vec3<R>& a, const Vec3<R>& b) {
  return Vec3<R>{xfma(s, a.x, b.x), xfma(s, a.y, b.y), xfma(s, a.z, b.z)};
}
template <typename R>
__device__ __forceinline__ R v3_dot(const Vec3<R>& a, const Vec3<R>& b) {
  return xdot(a.x, a.y, a.z, b.x, b.y, b.z);
}
template <typename R>
__device__ __forceinline__ Vec3<R> v3_scale(R s, const Vec3<R>& a) {
  return Vec3<R>{xmul(s, a.x), xmul(s, a.y), xmul(s, a.z)};
}
template <typename R>
__device__ __forceinline__ Vec3<R> v3_unit(const Vec3<R>& a) {
  return v3_scale(lrsqrt(v3_dot(a, a)), a);
}
// Unit vector of b - a with the inverse of its length: the nv / dn (or mv /
// dm) that _memb_bend_calc1 stores for a membrane particle
// (cell_interaction.cpp:296-309). (FP32: the inverse of the rounded length.)
template <typename R>
struct Unit {
  Vec3<R> v;
  R inv;
  Vec3<R> w;  // b - a
  R scale;    // v = scale w
};
template <typename R>
__device__ __forceinline__ Unit<R> unit_ab(const Vec3<R>& a, const Vec3<R>& b) {
  const Vec3<R> w = v3_sub(b, a);
  const R s = v3_dot(w, w);
  const R inv = lrsqrt(s);
  return Unit<R>{v3_scale(inv, w), sizeof(R) == 4 ? ldiv(R(1), xmul(s, inv)) : inv, w,
                 inv};
}

// The bending force of a membrane particle is a sum of terms g t, taken in a
// fixed order with one multiply-add each, so the terms may be evaluated one
// after the other by one thread or side by side by several lanes.
template <typename R>
struct BendTerm {
  Vec3<R> t;
  R g;
};
template <typename R>
__device__ __forceinline__ void bend_add(Vec3<R>& f, const BendTerm<R>& b) {
  f = v3_axpy(b.g, b.t, f);
}

// Square lattice (_memb_bend_calc1..3, :296-449). BCALC (:396-404) has three
// terms along the row and three along the column, each over two neighbouring
// links A, B of unit vectors a, b with cosine c (F the bend factor of c):
//   kind 0   F ((a - c b) / |B| - (b - c a) / |A|)      the links on either side
//   kind 1  -F (b - c a) / |A|                          the particle's own link, the next
//   kind 2   F (a - c b) / |B|                          the link before, the one before that
//   kind 3   the same, a formed within the difference
// taken in the order 0, 1, 2 of the row, then 1, 0, 3 of the column
// (square_kind). The roundings (kind 3's too, and the order of the cross
// products below) are those of the plain expressions as nvcc contracts them.
constexpr int kSquareTerms = 6;
__device__ __forceinline__ int square_kind(int e) { return e < 3 ? e : (e == 3 ? 1 : (e == 4 ? 0 : 3)); }
template <typename R>
__device__ __forceinline__ BendTerm<R> square_term(int kind, const Unit<R>& A, const Unit<R>& B,
                                                   R c) {
  const R F = bend_factor(c);
  const Vec3<R> P = v3_axpy(-c, B.v, A.v), Q = v3_axpy(-c, A.v, B.v);
  if (kind == 0) {
    const Vec3<R> q = v3_scale(A.inv, Q);
    return BendTerm<R>{v3_axpy(B.inv, P, v3_neg(q)), F};
  }
  if (kind == 1) return BendTerm<R>{v3_scale(-F, Q), A.inv};
  if (kind == 3) {
    const Vec3<R> cb = v3_scale(c, B.v);
    return BendTerm<R>{v3_scale(F, v3_axpy(A.scale, A.w, v3_neg(cb))), B.inv};
  }
  return BendTerm<R>{v3_scale(F, P), B.inv};
}

// Triangular lattice (tri_memb_bend, :451-508): the offsets n[i] of the six
// lattice neighbours memb[i], c[i] of the six second-ring sites
// memb[(i+1)%6]->memb[i]; the particle itself is the origin. The reference
// divides each term by the norm of a normal it has already normalised in
// place (vec3::normalize, vec3.h:40-44), i.e. by 1 up to rounding; that
// division is left out. Terms 0-5: tri_bend_1(r1 = self, a1 = n[i], b1 =
// n[i+1], c1 = c[i]); terms 6-11: tri_bend_2(r1 = self, a1 = n[i], b1 =
// n[i+1], c1 = n[i+2]).
constexpr int kTriTerms = 12;
template <typename R>
__device__ __forceinline__ BendTerm<R> tri_term1(const Vec3<R>& a, const Vec3<R>& b,
                                                 const Vec3<R>& c) {
  const Vec3<R> ab = v3_sub(a, b);
  const Vec3<R> n1 = v3_unit(v3_cross(ab, b));  // -b x ab
  const Vec3<R> n2 = v3_unit(v3_cross(ab, v3_sub(c, b)));
  const R d = v3_dot(n1, n2);
  return BendTerm<R>{v3_cross(ab, v3_axpy(-d, n1, n2)), bend_factor(d)};  // ab x tri_rho(n1, n2)
}
template <typename R>
__device__ __forceinline__ BendTerm<R> tri_term2(const Vec3<R>& a, const Vec3<R>& b,
                                                 const Vec3<R>& c) {
  const Vec3<R> bc = v3_sub(b, c), ab = v3_sub(a, b);
  const Vec3<R> n1 = v3_unit(v3_cross(bc, c));  // -c x bc
  const Vec3<R> n2 = v3_unit(v3_cross(ab, b));  // -b x ab
  const R d = v3_dot(n1, n2);
  const Vec3<R> t1 = v3_cross(bc, v3_axpy(-d, n1, n2));  // bc x tri_rho(n1, n2)
  const Vec3<R> t2 = v3_cross(ab, v3_axpy(-d, n2, n1));  // ab x tri_rho(n2, n1)
  return BendTerm<R>{Vec3<R>{xadd(t1.x, t2.x), xadd(t1.y, t2.y), xadd(t1.z, t2.z)},
                     bend_factor(d)};
}

// Lattice sites of a membrane particle at column jj, row kk of its tissue.
struct MembSites {
  int32_t pb, nmx, nmy, jj, kk, nmemb, self;
  __device__ __forceinline__ MembSites(const TissueDev& T, int32_t i)
      : MembSites(T, i, (i - T.pbase) % T.nmx, (i - T.pbase) / T.nmx) {}
  __device__ __forceinline__ MembSites(const TissueDev& T, int32_t i, int32_t jj_, int32_t kk_)
      : pb(T.pbase), nmx(T.nmx), nmy(T.nmy), jj(jj_), kk(kk_), nmemb(T.nmemb), self(i) {}
  __device__ __forceinline__ int32_t site(const DevState& S, int32_t col, int32_t row) const {
    const int32_t q = pb + row * nmx + col;
    return EPI_CHECKED(q >= pb && q < pb + nmemb, S.status, self, q) ? q : self;
  }
  // column jj+dj, row kk+dk with periodic wrap; the same wiring as _memb_init
  // (cellmanager.cpp:114-158)
  __device__ __forceinline__ int32_t square(const DevState& S, int dj, int dk) const {
    int32_t c = jj + dj, w = kk + dk;
    c += c < 0 ? nmx : 0;
    c -= c >= nmx ? nmx : 0;
    w += w < 0 ? nmy : 0;
    w -= w >= nmy ? nmy : 0;
    return site(S, c, w);
  }
  __device__ __forceinline__ int32_t tri(const DevState& S, int k) const {
    const TriSite a = tri_step(TriSite{jj, kk}, k, nmx, nmy);
    return site(S, a.col, a.row);
  }
  __device__ __forceinline__ int32_t tri_ring(const DevState& S, int k) const {
    const TriSite a =
        tri_step(tri_step(TriSite{jj, kk}, k == 5 ? 0 : k + 1, nmx, nmy), k, nmx, nmy);
    return site(S, a.col, a.row);
  }
  // lattice links in connected_cell's order (square: l, r, b, u)
  __device__ __forceinline__ int32_t link(const DevState& S, bool is_tri, int k) const {
    if (is_tri) return tri(S, k);
    return square(S, k == 0 ? -1 : (k == 1 ? 1 : 0), k == 2 ? -1 : (k == 3 ? 1 : 0));
  }
};

// The spring of membrane particle i's link to q at pq (_MEMB_interaction,
// :529-547, applied once by the higher index): DT coef separation, seen from
// i.
template <typename R>
__device__ __forceinline__ Vec3<R> link_term(const DevState& S, const SiteOffsets<R>& off,
                                             const TissueDev& T, const Laws<R>& L, R dt, int32_t i,
                                             int32_t q, const typename SiteOffsets<R>::Pos& pq) {
  const bool hi = i > q;
  const R rs = xadd(off.p.w, pq.w);
  R dx, dy, dz, d2;
  if constexpr (sizeof(R) == 4) {
    // mixed path: the FP32 copies, as for the bending stencil; the
    // minimum-image FP32 difference is antisymmetric, so both ends of a
    // link see opposite forces
    const Vec3<float> o = off.from(pq);
    dx = -o.x;
    dy = -o.y;
    dz = -o.z;
    d2 = xdot(dx, dy, dz, dx, dy, dz);
  } else {
    pair_sep(off.p, pq, hi, T, dx, dy, dz);
    d2 = dist_sq_exact(dx, dy, dz);
  }
  bool bad;
  const R c = L.memb_memb(d2, rs, &bad);
  if (bad) raise_error(S.status, E_MEMB_COEF_RANGE, hi ? i : q, hi ? q : i, double(c));
  const R sdt = xmul(dt, c);
  return Vec3<R>{xmul(sdt, dx), xmul(sdt, dy), xmul(sdt, dz)};
}

// Membrane particles: bending (square: the unit vectors of calc1 recomputed
// from the eleven lattice positions the stencil reaches instead of being
// stored), lattice springs and wall, summed for membrane particle i.
template <typename R>
__device__ __forceinline__ double3 memb_force(const DevState& S, int32_t i) {
  const TissueDev& T = S.tissues[attr_tissue(S.attr[i])];
  const Laws<R>& L = T.laws<R>();
  const R dt = R(T.P.dt);
  const MembSites M(T, i);
  const double4 p = S.pos_cur[i];
  const SiteOffsets<R> off(S, SiteOffsets<R>::own(S, i, p), T);
  const bool tri = T.lattice == kLatticeTriangular;
  Vec3<R> f{R(0), R(0), R(0)};
  if (tri) {
    Vec3<R> n[6], c[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) n[k] = off(M.tri(S, k));
#pragma unroll
    for (int k = 0; k < 6; ++k) c[k] = off(M.tri_ring(S, k));
#pragma unroll
    for (int k = 0; k < 6; ++k) bend_add(f, tri_term1(n[k], n[(k + 1) % 6], c[k]));
#pragma unroll
    for (int k = 0; k < 6; ++k) bend_add(f, tri_term2(n[k], n[(k + 1) % 6], n[(k + 2) % 6]));
  } else {
    const Vec3<R> o0{R(0), R(0), R(0)};
    {
      const Vec3<R> r = off(M.square(S, 1, 0)), rr = off(M.square(S, 2, 0));
      const Vec3<R> l = off(M.square(S, -1, 0)), ll = off(M.square(S, -2, 0));
      const Unit<R> nv = unit_ab(o0, r), nvr = unit_ab(r, rr);
      const Unit<R> nvl = unit_ab(l, o0), nvll = unit_ab(ll, l);
      bend_add(f, square_term(0, nv, nvl, v3_dot(nv.v, nvl.v)));
      bend_add(f, square_term(1, nv, nvr, v3_dot(nv.v, nvr.v)));
      bend_add(f, square_term(2, nvll, nvl, v3_dot(nvll.v, nvl.v)));
    }
    const Vec3<R> u = off(M.square(S, 0, 1)), uu = off(M.square(S, 0, 2));
    const Vec3<R> b = off(M.square(S, 0, -1)), bb = off(M.square(S, 0, -2));
    const Vec3<R> bbr = off(M.square(S, 1, -2)), bbrr = off(M.square(S, 2, -2));
    const Unit<R> mv = unit_ab(o0, u), mvu = unit_ab(u, uu);
    const Unit<R> mvb = unit_ab(b, o0), mvbb = unit_ab(bb, b);
    bend_add(f, square_term(1, mv, mvu, v3_dot(mv.v, mvu.v)));
    bend_add(f, square_term(0, mv, mvb, v3_dot(mv.v, mvb.v)));
    // the reference reads memb_bb's ipn (:380)
    const R c = v3_dot(unit_ab(bb, bbr).v, unit_ab(bbr, bbrr).v);
    bend_add(f, square_term(3, mvbb, mvb, c));
  }
  const R s = R(T.P.dt * T.P.kbend);
  double ax = double(xmul(s, f.x)), ay = double(xmul(s, f.y)), az = double(xmul(s, f.z));
  for (int k = 0; k < T.nadj; ++k) {
    const int32_t q = M.link(S, tri, k);
    const Vec3<R> w = link_term<R>(S, off, T, L, dt, i, q, off.at(q));
    ax = xadd(ax, double(w.x));
    ay = xadd(ay, double(w.y));
    az = xadd(az, double(w.z));
  }
  if (p.z < p.w) az = xadd(az, double(L.wall(dt, R(p.z), R(p.w))));
  return make_double3(ax, ay, az);
}

// The step proper. Per particle: connect_proc's exact predicate
// (cell_connection.cpp:115-119) on every candidate, the law(s) the reference
// applies to each connected pair, the particle's own terms, then pos_copy and
// the single wrap of cell_pos_periodic_fix.
//
// kSimple: every cell of the batch is ALIVE, DEAD or AIR (or a membrane
// particle) and none is paired; then each connected pair receives exactly
// one application of CI_al_air_de_to_al_air_de_fix_mu (:141-152): from the
// higher index when both cells are ALIVE/DEAD/AIR (:566-570), from the
// cell's side when the partner is a membrane particle (:573-575). kOld: some
// cell is older than THRESH_SP, so the adhesion constant depends on both
// cells' ages.
template <typename R, bool kSimple, bool kOld>
struct Particle {
  // The mixed path gathers candidates' FP32 copies and forms separations in
  // FP32; the FP64 path gathers the FP64 positions.
  static constexpr bool kFloatPos = sizeof(R) == 4;
  using Real = R;
  using Pos = typename std::conditional<kFloatPos, float4, double4>::type;
  const DevState& S;
  const int32_t i;
  const uint32_t a;
  const uint32_t t;
  const uint32_t st;
  const TissueDev& T;
  const Laws<R>& L;
  // FP64 path: the position; mixed path: its FP32 copy, as every writer of
  // posf forms it (the FP64 position is read again where it is needed, so it
  // holds no registers during the candidate loop)
  Pos p;
  const double lt2;  // LJ_THRESH * LJ_THRESH, folded as the reference does
  const R dt;
  R inv_ljt1sq;  // for aad_fused
  int32_t pair_i = -1, dermis_i = -1;
  double ax = 0.0, ay = 0.0, az = 0.0;
  // the first too-strong interaction of this particle (|coef| > 1000): kept
  // in registers and reported by finish(), so the candidate loop stores
  // nothing and the tissue's constants stay in registers across it. bad:
  // twice the partner's index, + 1 if it is the partner's law.
  uint32_t bad = 0xffffffffu;
  R bad_v = R(0);
  __device__ __forceinline__ void note_bad(R c, int32_t q, uint32_t theirs) {
    if (fabs(c) > R(1000) && bad == 0xffffffffu) {
      bad = 2u * (uint32_t)q + theirs;
      bad_v = c;
    }
  }
  static __device__ __forceinline__ Pos own(const double4& v) {
    if constexpr (kFloatPos) return make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    else return v;
  }

  // a_: the particle's attribute word, p_: its current position
  __device__ __forceinline__ Particle(const DevState& S_, int32_t i_, uint32_t a_,
                                     const double4& p_)
      : Particle(S_, i_, a_, own(p_), S_.tissues[attr_tissue(a_)]) {}
  // T_: the particle's tissue, wherever its constants are at hand
  __device__ __forceinline__ Particle(const DevState& S_, int32_t i_, uint32_t a_, const Pos& own_,
                                     const TissueDev& T_)
      : S(S_), i(i_), a(a_), t(attr_tissue(a)), st(attr_state(a)),
        T(T_), L(T.laws<R>()), p(own_),
        lt2(T.P.lj_thresh * T.P.lj_thresh), dt(R(T.P.dt)) {
    if constexpr (kFloatPos && kSimple) inv_ljt1sq = rcp_approx(L.ljt1sq);
    if (!kSimple && st != ST_MEMB) {
      pair_i = __ldg(&S.pair[i]);
      if (st == ST_FIX || st == ST_MUSUME) dermis_i = S.dermis[i];
      if (!EPI_CHECKED(pair_i < T.pbase + T.n && (pair_i >= T.pbase || pair_i == -1), S.status,
                       i, pair_i))
        pair_i = -1;
      if (!EPI_CHECKED(dermis_i < T.pbase + T.n && (dermis_i >= T.pbase || dermis_i == -1),
                       S.status, i, dermis_i))
        dermis_i = -1;
    }
  }

  // Connection test and separation of candidate q. FP64 path: the
  // reference's predicate (connect_proc :115-119) with its rounding. Mixed
  // path: the same test in FP32, decided by the FP64 predicate whenever the
  // FP32 d2 lies within T.ftol of the threshold, so the connection set is
  // the reference's in both.
  __device__ __forceinline__ bool connected(int32_t q, const double4& pq, R& dx, R& dy, R& dz,
                                            R& d2, R& rs) const {
    const double ddx = pdiff_h(p.x, pq.x, T.lx, T.hlx), ddy = pdiff_h(p.y, pq.y, T.ly, T.hly);
    const double ddz = p.z - pq.z;
    const double d2e = dist_sq_exact(ddx, ddy, ddz);
    const double rse = __dadd_rn(p.w, pq.w);
    if (!(d2e <= __dmul_rn(__dmul_rn(lt2, rse), rse))) return false;
    dx = R(ddx);
    dy = R(ddy);
    dz = R(ddz);
    d2 = R(d2e);
    rs = R(rse);
    return true;
  }
  // the reference's FP64 predicate of candidate q, from the FP64 positions
  __device__ __forceinline__ bool connected_fp64(int32_t q) const {
    const double4 pi = S.pos_cur[i], pq = S.pos_cur[q];
    const double d2e = dist_sq_exact(pdiff_h(pi.x, pq.x, T.lx, T.hlx),
                                     pdiff_h(pi.y, pq.y, T.ly, T.hly), pi.z - pq.z);
    const double rse = __dadd_rn(pi.w, pq.w);
    return d2e <= __dmul_rn(__dmul_rn(lt2, rse), rse);
  }
  // FP32 separation from the candidate's side (q - i; the minimum image is
  // antisymmetric), squared distance, radius sum and the squared distance
  // beyond the threshold. Minimum image as f - L rint(f / L) (positions lie
  // in [0, L], so |f| <= L): the compare-and-shift of p_diff_x for every |f|
  // away from L/2 by more than the rounding of f / L, i.e. for every pair
  // within reach of a connection (LJ_THRESH (r_i + r_j) + skin is far below
  // L/2); a pair near L/2 apart is rejected under either image. The packed
  // operations take x with y (four instructions) and z with the radius (one).
  struct Sep {
    F2 xy;
    float z, d2, rs, over;
  };
  __device__ __forceinline__ Sep separation(const float4& q) const {
    constexpr float kRound = 12582912.f;  // 1.5 * 2^23, see rint_fma
    Sep s;
    const F2 d = xadd(f2(q.x, q.y), f2(-p.x, -p.y));
    const F2 k = xadd(xfma(d, f2(T.ilxf, T.ilyf), f2(kRound, kRound)), f2(-kRound, -kRound));
    s.xy = xfma(k, f2(-T.lxf, -T.lyf), d);
    f2_out(xadd(f2(q.z, q.w), f2(-p.z, p.w)), s.z, s.rs);
    float x, y;
    f2_out(s.xy, x, y);
    s.d2 = xdot(x, y, s.z, x, y, s.z);
    s.over = xfma(-xmul(T.lt2f, s.rs), s.rs, s.d2);
    return s;
  }
  __device__ __forceinline__ bool connected(int32_t q, const float4& qf, R& dx, R& dy, R& dz,
                                            R& d2, R& rs) const {
    const Sep s = separation(qf);
    if (s.over > T.ftol) return false;
    // too close to the threshold for FP32: the reference's FP64 predicate
    if (s.over >= -T.ftol && !connected_fp64(q)) return false;
    f2_out(s.xy, dx, dy);
    dx = -dx;
    dy = -dy;
    dz = -s.z;
    d2 = s.d2;
    rs = s.rs;
    return true;
  }

  // Mixed path, simple states: the same test and law as connected() and
  // term(), with the law evaluated for every candidate and masked by the
  // test, so the lanes of a warp do not diverge on it; only the rare FP64
  // decision near the threshold branches. A candidate that is not connected
  // adds +0 or -0 to the sums, which leaves them unchanged: they start at +0
  // and, rounding to nearest, never become -0.
  __device__ __forceinline__ Vec3<R> term_simple(int32_t q, const float4& qf) {
    const Sep s = separation(qf);
    bool conn = !(s.over > T.ftol);
    if (conn && s.over >= -T.ftol) conn = connected_fp64(q);
    const bool both_old = kOld && attr_old(a) && attr_old(__ldg(&S.attr[q]));
    float coef = L.aad_fused(s.d2, s.rs, both_old, inv_ljt1sq);
    coef = conn ? coef : 0.f;
    note_bad(coef, q, 0);
    const float sdt = xmul(-dt, coef);
    Vec3<R> v;
    f2_out(xmul(s.xy, f2(sdt, sdt)), v.x, v.y);
    v.z = xmul(sdt, s.z);
    return v;
  }

  // DT * coef * separation of candidate q (cell_interaction_apply, :56-58);
  // zero when it is not connected.
  __device__ __forceinline__ Vec3<R> term(int32_t q, const Pos& pq) {
    if constexpr (kFloatPos && kSimple) {
      return term_simple(q, pq);
    } else {
      R dx, dy, dz, d2, rs;
      if (!connected(q, pq, dx, dy, dz, d2, rs)) return Vec3<R>{R(0), R(0), R(0)};
      R coef;
      if (kSimple) {
        const bool both_old = kOld && attr_old(a) && attr_old(__ldg(&S.attr[q]));
        coef = L.aad(d2, rs, both_old);
        note_bad(coef, q, 0);
      } else {
        const uint32_t aq = __ldg(&S.attr[q]);
        const uint32_t sq = attr_state(aq);
        const bool both_old = attr_old(a) && attr_old(aq);
        coef = R(0);
        // the law i applies while iterating q (if i is not a membrane particle)
        if (st != ST_MEMB) {
          const int law = law_of(st, i, pair_i, dermis_i, sq, q);
          if (law != L_NONE) {
            const R c = eval_law<R>(law, L, d2, rs, both_old, attr_sfm(a));
            note_bad(c, q, 0);
            coef = c;
          }
        }
        // ... and the law q applies while iterating i (if q is not)
        if (sq != ST_MEMB) {
          int32_t pair_q = -1, dermis_q = -1;
          if (sq == ST_FIX || sq == ST_MUSUME) {
            pair_q = __ldg(&S.pair[q]);
            dermis_q = S.dermis[q];
          }
          const int law = law_of(sq, q, pair_q, dermis_q, st, i);
          if (law != L_NONE) {
            const R c = eval_law<R>(law, L, d2, rs, both_old, attr_sfm(aq));
            note_bad(c, q, 1);
            coef = xadd(coef, c);
          }
        }
      }
      const R sdt = xmul(dt, coef);
      return Vec3<R>{xmul(sdt, dx), xmul(sdt, dy), xmul(sdt, dz)};
    }
  }

  // summed in FP64, in the row's order
  __device__ __forceinline__ void candidate(int32_t q, const Pos& pq) {
    const Vec3<R> v = term(q, pq);
    ax = xadd(ax, double(v.x));
    ay = xadd(ay, double(v.y));
    az = xadd(az, double(v.z));
  }

  __device__ __forceinline__ void report_bad() const {
    if (bad == 0xffffffffu) return;
    const int32_t q = (int32_t)(bad >> 1);
    const bool theirs = bad & 1u;
    raise_error(S.status, E_COEF_RANGE, theirs ? q : i, theirs ? i : q, double(bad_v));
  }

  // p: the position; b: that of the tissue's last candidate rebuild; f: the
  // membrane sums (membrane particles only). Returns the new position.
  __device__ __forceinline__ double4 finish(const double4& p, const float4& b, const double4& f) {
    report_bad();
    if (st == ST_MEMB) {
      ax += f.x;
      ay += f.y;
      az += f.z;
    } else if (!kSimple) {
      // wall_interaction (:287-294) for DER below its radius
      if (st == ST_DER && p.z < p.w) az += double(L.wall(dt, R(p.z), R(p.w)));
      // _pair_interaction (:637-641), applied by the higher index of the pair
      if (pair_i >= 0) {
        const double4 pq = S.pos_cur[pair_i];
        const bool hi = i > pair_i;
        double dx, dy, dz;
        pair_sep(p, pq, hi, T, dx, dy, dz);
        const R d2 = R(dist_sq_exact(dx, dy, dz));
        const R c = L.pair(d2, R(hi ? S.spr[i] : S.spr[pair_i]));
        if (fabs(c) > R(1000)) raise_error(S.status, E_COEF_RANGE, i, pair_i, double(c));
        const R sdt = xmul(dt, c);
        ax += double(xmul(sdt, R(dx)));
        ay += double(xmul(sdt, R(dy)));
        az += double(xmul(sdt, R(dz)));
      }
    }
    // pos_copy + the single wrap of cell_pos_periodic_fix
    const double lx = T.lx, ly = T.ly;
    double nx = p.x + ax, ny = p.y + ay;
    const double nz = p.z + az;
    if (nx > lx) nx -= lx;
    else if (nx < 0) nx += lx;
    if (ny > ly) ny -= ly;
    else if (ny < 0) ny += ly;
    if (!isfinite(nx) || !isfinite(ny) || !isfinite(nz)) {
      raise_error(S.status, E_NONFINITE, i, -1, nz);
    } else if (!range_ok(T, nx, ny, nz, st == ST_MEMB)) {
      raise_error(S.status, E_BIN_RANGE, i, -1, nz);
    }
    S.pos_nxt[i] = make_double4(nx, ny, nz, p.w);
    if (kFloatPos) S.posf_nxt[i] = make_float4((float)nx, (float)ny, (float)nz, (float)p.w);
    // Candidate validity: rebuild the tissue once a particle moved skin/2.
    if (moved_too_far(S.skin, T, nx, ny, nz, b)) {
      S.gate[1 + t] = 1;
      *S.flag = 1;
    }
    return make_double4(nx, ny, nz, p.w);
  }
};

// find_dermis (cell_connection.cpp:158-172) of FIX / MUSUME cell i by one
// warp: the nearest connected membrane particle, strict <, starting from
// LX*LX; on exact ties the lowest index wins (the reference: first in list
// order). The cell's row holds a hundred or more candidates, which one thread
// walked one after the other.
__device__ __forceinline__ void dermis_cell(const DevState& S, int32_t i, int lane) {
  const TissueDev& T = S.tissues[attr_tissue(S.attr[i])];
  const double4 p = S.pos_cur[i];
  const int32_t nc = cand_count(S, i);
  const double lt = T.P.lj_thresh;
  int32_t best = -1;
  double bestd = T.lx * T.lx;
  for (int32_t k = lane; k < nc; k += 32) {
    const int32_t q = T.pbase + (int32_t)cand_entry(S, i, k + 1);
    if (!EPI_CHECKED(q < T.pbase + T.n, S.status, i, q)) continue;
    if (attr_state(S.attr[q]) != ST_MEMB) continue;
    const double4 pq = S.pos_cur[q];
    const double d2 = dist_sq_exact(pdiff(p.x, pq.x, T.lx), pdiff(p.y, pq.y, T.ly), p.z - pq.z);
    if (!connected_pred(d2, lt, p.w, pq.w)) continue;
    if (d2 < bestd || (d2 == bestd && q < best)) {
      bestd = d2;
      best = q;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double od = __shfl_xor_sync(0xffffffffu, bestd, o);
    const int32_t ob = __shfl_xor_sync(0xffffffffu, best, o);
    if (od < bestd || (od == bestd && ob < best)) {
      bestd = od;
      best = ob;
    }
  }
  if (lane == 0) S.dermis[i] = best;
}

}  // namespace
}  // namespace epi
