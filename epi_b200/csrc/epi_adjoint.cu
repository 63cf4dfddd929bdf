// Reverse-mode adjoint of the mechanics step, FP64.
//
// The step maps positions X_t to X_{t+1} = wrap(X_t + D(X_t; s)), where D is
// the displacement cell_interaction accumulates (epi5_MT/cell_interaction.cpp
// :648-685) and s = (s_spring, s_eps, s_bend) multiplies every spring
// constant, eps_m and KBEND. The wrap is a translation by a box length, so
// its derivative is the identity. Given lambda = dL/dX_{t+1}, one backward
// step returns
//   dL/dX_t = lambda + (dD/dX_t)^T lambda     and adds   (dD/ds)^T lambda
// to the parameter gradient. The connection set of step t is the exact
// predicate of connect_proc at X_t (piecewise constant in X), evaluated on
// the Verlet candidates like the forward step.
//
// Terms of D, for every cell state of the path:
//   pairs     D_i += DT c(r2) d_ij, c the sum of the laws the reference
//             applies to the pair from either side (law_of: ljmain, adhesion,
//             CI_der_to_der, the FIX / MUSUME dermis springs, :103-183,
//             549-634); J = c I + 2 c'(r2) d d^T and D_j gets -DT c d_ij, so
//             (dD/dX)^T lambda at i is DT sum_j J (lambda_i - lambda_j): a
//             gather over the same lists. The pair springs of dividing cells
//             (CI_pair, :281-285, 637-641) add the same form for the partner.
//   lattice   the four lattice springs of _MEMB_interaction (CI_memb_to_memb,
//             :185-234), the same gather over fixed partners.
//   wall      z += DT W(z) for z < r, membrane and DER (:287-294, 549-561).
//   bending   D_k += DT KBEND B_k(stencil sites): square, eleven lattice
//             sites (_memb_bend_calc1..3, :296-449); triangular, the six
//             neighbours and six second-ring sites of the twelve dihedral
//             terms of tri_memb_bend (:451-508). Their vector-Jacobian
//             products are derived by hand below; each membrane particle
//             writes the products for the sites of its stencil and every
//             site gathers the entries that name it, so no atomics are
//             needed and results are deterministic.
#include "epi_kernels.h"
#include "epi_device.cuh"

namespace epi {
namespace {

struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 d3(double x, double y, double z) { return D3{x, y, z}; }
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return D3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return D3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 operator*(double s, D3 a) { return D3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ D3& operator+=(D3& a, D3 b) { return a = a + b; }
__device__ __forceinline__ D3& operator-=(D3& a, D3 b) { return a = a - b; }
__device__ __forceinline__ double dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 xyz(double4 v) { return D3{v.x, v.y, v.z}; }
__device__ __forceinline__ D3 cross(D3 a, D3 b) {
  return D3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// A pair coefficient with its derivatives: c, dc/d(r2), and the parts of c
// that scale with s_spring and with s_eps (each law is linear in them).
struct LawD {
  double c, dc_dr2, c_spring, c_eps;
};
__device__ __forceinline__ LawD operator+(const LawD& a, const LawD& b) {
  return LawD{a.c + b.c, a.dc_dr2 + b.dc_dr2, a.c_spring + b.c_spring, a.c_eps + b.c_eps};
}

// A pair's distance with its reciprocals, from one corrected rsqrt: the laws
// and their derivatives divide by r and r2 up to six times, and an FP64
// division is a chain of a dozen operations.
struct Dist {
  double r2, r, i, i2;  // r2, r, 1 / r, 1 / r2
};
__device__ __forceinline__ Dist dist_d(double r2) {
  const double i = rsqrt(r2);
  return Dist{r2, dist_of(r2, i), i, inv_sq(r2, i)};
}

// ljmain (:103-111): c = eps4 u (u - 1) / r2 with u = rs^6 / r2^3.
__device__ __forceinline__ LawD ljmain_d(const Laws<double>& L, const Dist& d, double rs2) {
  const double q = rs2 * d.i2;
  const double u = q * q * q;
  const double c = L.eps4 * u * (u - 1.0) * d.i2;
  const double dc = -L.eps4 * u * (7.0 * u - 4.0) * (d.i2 * d.i2);
  return LawD{c, dc, 0.0, c};
}

// adhesion (:113-124) with spring constant k.
__device__ __forceinline__ LawD adhesion_d(const Laws<double>& L, const Dist& d, double rs,
                                           double k) {
  const double irs = 1.0 / rs;
  const double y = d.r * irs - 1.0;
  if (y + 1.0 > L.lj_thresh) return LawD{0.0, 0.0, 0.0, 0.0};
  const double w = y * y * L.inv_ljt1sq;
  const double h = 1.0 - w;
  const double c = -(k * d.i) * y * h;
  // dc/dr = k y h / r^2 - (k / r) (1 - 3 y^2 / a^2) / rs
  const double dcdr = k * y * h * d.i2 - (k * d.i) * (1.0 - 3.0 * w) * irs;
  return LawD{c, 0.5 * dcdr * d.i, c, 0.0};
}

// CI_al_air_de_to_al_air_de_fix_mu (:141-152).
__device__ __forceinline__ LawD aad_d(const Laws<double>& L, const Dist& d, double rs,
                                      bool both_old) {
  if (d.r2 < rs * rs) return ljmain_d(L, d, rs * rs);
  return adhesion_d(L, d, rs, both_old ? L.k_total : L.k_desmosome);
}

// CI_fix_mu_to_fix_mu (:154-162).
__device__ __forceinline__ LawD fixmu_d(const Laws<double>& L, const Dist& d, double rs) {
  if (d.r2 < rs * rs) return ljmain_d(L, d, rs * rs);
  return adhesion_d(L, d, rs, L.k_desmosome);
}

// CI_mu_to_memb (:164-172) with the MUSUME's spring_force_to_memb.
__device__ __forceinline__ LawD mu_memb_d(const Laws<double>& L, const Dist& d, double rs,
                                          uint32_t sfm) {
  if (d.r2 < rs * rs) return ljmain_d(L, d, rs * rs);
  return adhesion_d(L, d, rs, sfm_value(sfm, L));
}

// A spring c = -(k / r) (r / a - 1) = k (1/r - 1/a).
__device__ __forceinline__ LawD spring_d(const Dist& d, double a, double k) {
  const double c = -(k * d.i) * (d.r / a - 1.0);
  return LawD{c, -0.5 * k * d.i * d.i2, c, 0.0};
}

// CI_fix_to_memb (:174-183).
__device__ __forceinline__ LawD fix_memb_d(const Laws<double>& L, const Dist& d, double rs) {
  if (d.r2 < rs * rs) return ljmain_d(L, d, rs * rs);
  return spring_d(d, rs, L.kspring);
}

// CI_der_to_der (:129-139), dd = r + delta_R, u = (rs / dd)^6, h = u (u - 1):
// eps4 h / (r dd) + para_ljp2 while dd < rs, para_ljp2 inside the radius
// sum, eps4 h / r^2 + para_ljp2 beyond; dh/dr = -6 u (2 u - 1) / dd.
__device__ __forceinline__ LawD der_der_d(const Laws<double>& L, const Dist& d, double rs) {
  const double dd = d.r + L.delta_r;
  if (!(dd < rs) && d.r2 < rs * rs) return LawD{L.para_ljp2, 0.0, 0.0, 0.0};
  const double rs2 = rs * rs, idd = 1.0 / dd;
  const double v = rs2 * (idd * idd);
  const double u = v * v * v;
  const double h = u * (u - 1.0);
  const double dh = -6.0 * u * (2.0 * u - 1.0) * idd;
  double ce, dce;
  if (dd < rs) {
    const double iq = d.i * idd;
    ce = L.eps4 * h * iq;
    dce = L.eps4 * (dh * iq - h * (dd + d.r) * (iq * iq));
  } else {
    ce = L.eps4 * h * d.i2;
    dce = L.eps4 * (dh * d.i2 - 2.0 * h * (d.i2 * d.i));
  }
  return LawD{ce + L.para_ljp2, 0.5 * dce * d.i, 0.0, ce};
}

// CI_pair (:281-285): c = -Kdiv (r - rest) / r, rest the higher index's
// spr_nat_len.
__device__ __forceinline__ LawD pair_d(const Laws<double>& L, const Dist& d, double rest) {
  const double c = -(L.kspring_division * (d.r - rest)) * d.i;
  return LawD{c, -0.5 * L.kspring_division * rest * (d.i2 * d.i), c, 0.0};
}

// The law `law` (law_of) as a LawD.
__device__ __forceinline__ LawD law_d(int law, const Laws<double>& L, const Dist& d, double rs,
                                      bool both_old, uint32_t sfm) {
  switch (law) {
    case L_OTHER: return ljmain_d(L, d, rs * rs);
    case L_DER_DER: return der_der_d(L, d, rs);
    case L_AAD: return aad_d(L, d, rs, both_old);
    case L_FIXMU: return fixmu_d(L, d, rs);
    case L_FIX_MEMB: return fix_memb_d(L, d, rs);
    case L_MU_MEMB: return mu_memb_d(L, d, rs, sfm);
    default: return LawD{0.0, 0.0, 0.0, 0.0};
  }
}

// wall_interaction (:287-294): dz = dt eps4 u (u - 1) / (2 z), u = (r / z)^6;
// adds its adjoint to mu.z and its eps part to g_eps.
__device__ __forceinline__ void wall_back(const Laws<double>& L, double dt, double z, double rad,
                                          double lz, D3& mu, double& g_eps) {
  const double rz = rad / z;
  const double rz2 = rz * rz;
  const double u = rz2 * rz2 * rz2;
  const double W = dt * L.eps4 * u * (u - 1.0) / (2.0 * z);
  const double dW = -dt * L.eps4 * u * (13.0 * u - 7.0) / (2.0 * z * z);
  mu.z += dW * lz;
  g_eps += W * lz;
}

// CI_memb_to_memb (:185-234), three branches.
__device__ __forceinline__ LawD memb_memb_d(const Laws<double>& L, double r2, double rs) {
  const double P = L.p_memb;
  const double rs2 = rs * rs;
  const double cr2 = rs2 * P * P;
  const Dist d = dist_d(r2);
  if (r2 < cr2) return ljmain_d(L, d, cr2);
  if (r2 < rs2) return spring_d(d, rs * P, L.der_der_const);
  const double lam = (1.0 + P) * rs;
  const double v = lam - d.r;
  const double cr = rs * P;
  const double iv = 1.0 / v;
  const double cr2v = cr * iv * (cr * iv);
  const double u = cr2v * cr2v * cr2v;
  const double c_spring = -L.memb_far / rs;
  const double ivr = iv * d.i;
  const double c_eps = -L.eps4 * u * (u - 1.0) * ivr;
  // d/dr of u (u - 1) / (v r), with du/dr = 6 u / v and d(v r)/dr = v - r
  const double dh =
      6.0 * u * (2.0 * u - 1.0) * (iv * ivr) - u * (u - 1.0) * (v - d.r) * (ivr * ivr);
  return LawD{c_spring + c_eps, -0.5 * L.eps4 * dh * d.i, c_spring, c_eps};
}

// _memb_bend_diff_factor (:349-360) and its derivative.
__device__ __forceinline__ double bf(double c) {
  return c >= 0.0 ? 1.0 - c : 1.0 / ((1.0 + c) * (1.0 + c));
}
__device__ __forceinline__ double bf_d(double c) {
  if (c >= 0.0) return -1.0;
  const double e = 1.0 + c;
  return -2.0 / (e * e * e);
}

// Unit vector of b - a with the inverse of its length.
struct U3 {
  D3 v;
  double inv;
};
__device__ __forceinline__ U3 unit3(D3 a, D3 b) {
  const D3 w = b - a;
  const double inv = rsqrt(dot(w, w));
  return U3{inv * w, inv};
}
// Adjoint of w = b - a from the adjoints of the unit vector (ub) and of the
// length (lb): w_bar = (ub - (ub . u) u) / len + lb u; b += w_bar, a -= w_bar.
__device__ __forceinline__ void unit3_back(const U3& u, D3 ub, double lb, D3& abar, D3& bbar) {
  const D3 w = u.inv * (ub - dot(ub, u.v) * u.v) + lb * u.v;
  bbar += w;
  abar -= w;
}

// Stencil slots of the bending term of particle k, as lattice offsets:
// k, r, rr, l, ll, u, uu, b, bb, r of bb, rr of bb.
constexpr int kSlots = 11;
// The row half of BCALC names k, r, rr, l, ll (slots 0-4), the column half
// the rest and k again (slot kSelf2): a thread each.
constexpr int kSelf2 = 11;
// Triangular lattice: k, its neighbour in direction i (slot 1 + i), and the
// second-ring site c_i = memb[(i+1)%6]->memb[i] (slot 7 + i).
constexpr int kTriSlots = 13;
// Entries per membrane particle in the bending-product buffer.
constexpr int kBendStride = 13;
__constant__ int kSlotDj[kSlots] = {0, 1, 2, -1, -2, 0, 0, 0, 0, 1, 2};
__constant__ int kSlotDk[kSlots] = {0, 0, 0, 0, 0, 1, 2, -1, -2, -2, -2};

// One half of BCALC (:396-404) and its adjoint. With n, a (the right /
// upper neighbour's vector), l, m (the left / lower ones), the lengths D, E
// and the cosines p = n.a, q = l.n, w:
//   T = -g(p) (a - p n) / D + g(q) ((n - q l) / E - (l - q n) / D)
//       + g(w) (m - w l) / E.
// Given ybar, returns y . T and accumulates the adjoints of n, a, l, m, D, E
// and w (w's inputs differ between the two halves).
struct HalfBar {
  D3 n, a, l, m;
  double D, E, w;
};
// iD, iE: 1 / D, 1 / E.
__device__ __forceinline__ double half_back(D3 yb, D3 n, D3 a, D3 l, D3 m, double iD, double iE,
                                            double w, HalfBar& hb) {
  const double p = dot(n, a), q = dot(l, n);
  const double gp = bf(p), gq = bf(q), gw = bf(w);
  const double yn = dot(yb, n), ya = dot(yb, a), yl = dot(yb, l), ym = dot(yb, m);
  const double val = -gp * (ya - p * yn) * iD + gq * ((yn - q * yl) * iE - (yl - q * yn) * iD) +
                     gw * (ym - w * yl) * iE;
  const double pb = (-bf_d(p) * (ya - p * yn) + gp * yn) * iD;
  const double qb = bf_d(q) * ((yn - q * yl) * iE - (yl - q * yn) * iD) + gq * (yn * iD - yl * iE);
  hb.w = bf_d(w) * (ym - w * yl) * iE - gw * yl * iE;
  hb.a = (-gp * iD) * yb + pb * n;
  hb.n = (gp * p * iD + gq * iE + gq * q * iD) * yb + pb * a + qb * l;
  hb.l = (-gq * q * iE - gq * iD - gw * w * iE) * yb + qb * n;
  hb.m = (gw * iE) * yb;
  hb.D = (gp * (ya - p * yn) + gq * (yl - q * yn)) * iD * iD;
  hb.E = -(gq * (yn - q * yl) + gw * (ym - w * yl)) * iE * iE;
  return val;
}

// tri_bend_1 (:475-481) of particle k with offsets a = n_i, b = n_{i+1},
// c = c_i (k at the origin): term = g(d) ab x (n2 - d n1), n1 = unit(rb x
// ab), n2 = unit(ab x cb), d = n1 . n2, rb = -b, ab = a - b, cb = c - b (the
// reference's division by the norm of an already normalised normal is 1 up
// to rounding and is left out, as in the forward step). Returns y . term and
// accumulates the adjoints of a, b, c. For p x q the adjoints are q x ybar
// and ybar x p; for n = N / |N|, Nbar = (nbar - (nbar . n) n) / |N|.
__device__ __forceinline__ double tri1_back(D3 y, D3 a, D3 b, D3 c, D3& abar, D3& bbar,
                                            D3& cbar) {
  const D3 rb = d3(-b.x, -b.y, -b.z), ab = a - b, cb = c - b;
  const D3 N1 = cross(rb, ab), N2 = cross(ab, cb);
  const double i1 = rsqrt(dot(N1, N1)), i2 = rsqrt(dot(N2, N2));
  const D3 n1 = i1 * N1, n2 = i2 * N2;
  const double d = dot(n1, n2);
  const D3 v = n2 - d * n1;
  const D3 t = cross(ab, v);
  const double g = bf(d), yt = dot(y, t);
  double dbar = bf_d(d) * yt;
  const D3 tbar = g * y;
  D3 abbar = cross(v, tbar);
  const D3 vbar = cross(tbar, ab);
  D3 n2bar = vbar, n1bar = (-d) * vbar;
  dbar -= dot(vbar, n1);
  n1bar += dbar * n2;
  n2bar += dbar * n1;
  const D3 N1bar = i1 * (n1bar - dot(n1bar, n1) * n1);
  const D3 N2bar = i2 * (n2bar - dot(n2bar, n2) * n2);
  const D3 rbbar = cross(ab, N1bar);
  abbar += cross(N1bar, rb);
  abbar += cross(cb, N2bar);
  const D3 cbbar = cross(N2bar, ab);
  abar += abbar;
  bbar -= abbar;
  bbar -= rbbar;
  bbar -= cbbar;
  cbar += cbbar;
  return g * yt;
}

// tri_bend_2 (:483-495) with a = n_i, b = n_{i+1}, cc = n_{i+2}: term =
// g(d) [bc x (n2 - d n1) + ab x (n1 - d n2)], n1 = unit(rc x bc), n2 =
// unit(rb x ab), rc = -cc, rb = -b, bc = b - cc, ab = a - b.
__device__ __forceinline__ double tri2_back(D3 y, D3 a, D3 b, D3 cc, D3& abar, D3& bbar,
                                            D3& ccbar) {
  const D3 rc = d3(-cc.x, -cc.y, -cc.z), rb = d3(-b.x, -b.y, -b.z);
  const D3 bc = b - cc, ab = a - b;
  const D3 N1 = cross(rc, bc), N2 = cross(rb, ab);
  const double i1 = rsqrt(dot(N1, N1)), i2 = rsqrt(dot(N2, N2));
  const D3 n1 = i1 * N1, n2 = i2 * N2;
  const double d = dot(n1, n2);
  const D3 v1 = n2 - d * n1, v2 = n1 - d * n2;
  const D3 t = cross(bc, v1) + cross(ab, v2);
  const double g = bf(d), yt = dot(y, t);
  double dbar = bf_d(d) * yt;
  const D3 tbar = g * y;
  D3 bcbar = cross(v1, tbar);
  const D3 v1bar = cross(tbar, bc);
  D3 abbar = cross(v2, tbar);
  const D3 v2bar = cross(tbar, ab);
  D3 n2bar = v1bar - d * v2bar, n1bar = v2bar - d * v1bar;
  dbar -= dot(v1bar, n1) + dot(v2bar, n2);
  n1bar += dbar * n2;
  n2bar += dbar * n1;
  const D3 N1bar = i1 * (n1bar - dot(n1bar, n1) * n1);
  const D3 N2bar = i2 * (n2bar - dot(n2bar, n2) * n2);
  const D3 rcbar = cross(bc, N1bar);
  bcbar += cross(N1bar, rc);
  const D3 rbbar = cross(ab, N2bar);
  abbar += cross(N2bar, rb);
  ccbar -= rcbar;
  ccbar -= bcbar;
  bbar -= rbbar;
  bbar += bcbar;
  bbar -= abbar;
  abar += abbar;
  return g * yt;
}

// The bending adjoint of every membrane particle: its products for the sites
// of its stencil to bend[e * kBendStride + slot], its parameter partial in the
// .w of slot 0 (and kSelf2). kLanes threads per particle. Square: the row
// half of BCALC by the first, the column half by the second. Triangular
// (kLanes = 8): terms k of both kinds by lane k < 6; a neighbour's products
// come from the lanes whose terms name it. Bound by the latency of one
// thread's chain, which is why it is cut: one thread per particle took 21 us
// on 4,096 membrane particles, on 16 of the SMs.
template <int kLanes>
__global__ void __launch_bounds__(64) k_adj_bend(DevState S, const double4* lam,
                                                 double4* bend) {
  pdl_entry();
  const int sub = (int)threadIdx.x & (kLanes - 1);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x / kLanes;
  for (int64_t e0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
       e0 - (threadIdx.x & 31) / kLanes < S.nprep_memb; e0 += stride) {
    // the lanes of a warp run in step; those past the end write nothing
    const bool in = e0 < S.nprep_memb;
    const int64_t e = in ? e0 : S.nprep_memb - 1;
    const int32_t i = S.prep[e];
    const TissueDev& T = S.tissues[attr_tissue(S.attr[i])];
    const int32_t pb = T.pbase, NMX = T.nmx, NMY = T.nmy;
    const int32_t j = i - pb, jj = j % NMX, kk = j / NMX;
    const double4 p = S.pos_cur[i];
    const D3 yb = (T.P.dt * T.P.kbend) * xyz(lam[i]);
    double4* out = bend + e * kBendStride;
    auto put = [&](int slot, D3 v, double w) {
      if (in) out[slot] = make_double4(v.x, v.y, v.z, w);
    };
    auto offset = [&](int32_t q) {
      const Vec3<double> v = offset_of<double>(S.pos_cur[q], p, T);
      return d3(v.x, v.y, v.z);
    };
    const bool tri = T.lattice == kLatticeTriangular;
    if constexpr (kLanes == 8) {
      // every lane takes part in the exchange
      D3 ob[4] = {};  // of this lane's terms: a, b, c of kind 2, ring
      double g = 0.0;
      if (tri && sub < 6) {
        auto site = [&](TriSite t) { return offset(pb + t.row * NMX + t.col); };
        auto turn = [](int k) { return k >= 6 ? k - 6 : k; };
        const TriSite s0{jj, kk};
        const D3 a = site(tri_step(s0, sub, NMX, NMY));
        const TriSite sb = tri_step(s0, turn(sub + 1), NMX, NMY);
        const D3 b = site(sb), c = site(tri_step(s0, turn(sub + 2), NMX, NMY));
        const D3 r = site(tri_step(sb, sub, NMX, NMY));
        g = tri1_back(yb, a, b, r, ob[0], ob[1], ob[3]);
        g += tri2_back(yb, a, b, c, ob[0], ob[1], ob[2]);
      }
      // neighbour k: a of term k, b of term k - 1, c of term k - 2
      auto from = [&](D3 v, int k) {
        const int l = sub >= k ? sub - k : sub - k + 6;
        return d3(__shfl_sync(0xffffffffu, v.x, l, 8), __shfl_sync(0xffffffffu, v.y, l, 8),
                  __shfl_sync(0xffffffffu, v.z, l, 8));
      };
      const D3 nb = ob[0] + from(ob[1], 1) + from(ob[2], 2);
      D3 self = sub < 6 ? nb + ob[3] : d3(0.0, 0.0, 0.0);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        self += d3(__shfl_xor_sync(0xffffffffu, self.x, o, 8),
                   __shfl_xor_sync(0xffffffffu, self.y, o, 8),
                   __shfl_xor_sync(0xffffffffu, self.z, o, 8));
        g += __shfl_xor_sync(0xffffffffu, g, o, 8);
      }
      if (tri) {
        if (sub < 6) {
          put(1 + sub, nb, 0.0);
          put(7 + sub, ob[3], 0.0);
        }
        if (sub == 0) put(0, d3(-self.x, -self.y, -self.z), g);
        continue;
      }
    }
    if (sub > 1) continue;
    auto at = [&](int dj, int dk) {
      int32_t c = jj + dj, w = kk + dk;
      c += c < 0 ? NMX : 0;
      c -= c >= NMX ? NMX : 0;
      w += w < 0 ? NMY : 0;
      w -= w >= NMY ? NMY : 0;
      return offset(pb + w * NMX + c);
    };
    // the half's line of sites: next, after next, previous, before previous;
    // the column half also the row two below
    const bool col = sub == 1;
    D3 o1 = at(col ? 0 : 1, col ? 1 : 0), o2 = at(col ? 0 : 2, col ? 2 : 0);
    D3 o3 = at(col ? 0 : -1, col ? -1 : 0), o4 = at(col ? 0 : -2, col ? -2 : 0);
    const D3 o0 = d3(0.0, 0.0, 0.0);
    const U3 nv = unit3(o0, o1), nvr = unit3(o1, o2), nvl = unit3(o3, o0), nvll = unit3(o4, o3);
    D3 b0 = o0, b1 = o0, b2 = o0, b3 = o0, b4 = o0, b9 = o0, b10 = o0;
    HalfBar h;
    double g;
    if (!col) {
      g = half_back(yb, nv.v, nvr.v, nvl.v, nvll.v, nv.inv, nvl.inv, dot(nvll.v, nvl.v), h);
      h.m += h.w * nvl.v;  // w = nvll . nvl
      h.l += h.w * nvll.v;
    } else {
      const D3 o9 = at(1, -2), o10 = at(2, -2);
      const U3 nvbb = unit3(o4, o9), nvbbr = unit3(o9, o10);
      // w is memb_bb's ipn (:380)
      g = half_back(yb, nv.v, nvr.v, nvl.v, nvll.v, nv.inv, nvl.inv, dot(nvbb.v, nvbbr.v), h);
      unit3_back(nvbb, h.w * nvbbr.v, 0.0, b4, b9);
      unit3_back(nvbbr, h.w * nvbb.v, 0.0, b9, b10);
    }
    unit3_back(nv, h.n, h.D, b0, b1);
    unit3_back(nvr, h.a, 0.0, b1, b2);
    unit3_back(nvl, h.l, h.E, b3, b0);
    unit3_back(nvll, h.m, 0.0, b4, b3);
    // offsets are x_site - x_k: the particle itself receives minus every
    // offset's adjoint (o0 is the constant zero)
    const D3 self = b1 + b2 + b3 + b4 + b9 + b10;
    put(col ? kSelf2 : 0, d3(-self.x, -self.y, -self.z), g);
    put(col ? 5 : 1, b1, 0.0);
    put(col ? 6 : 2, b2, 0.0);
    put(col ? 7 : 3, b3, 0.0);
    put(col ? 8 : 4, b4, 0.0);
    if (col) {
      put(9, b9, 0.0);
      put(10, b10, 0.0);
    }
  }
}

// Every particle: the pair adjoint over the exact connections at X_t, and for
// membrane particles the lattice springs, the wall and the bending products
// that name them, into lam_out; its parameter partials are added to gpart
// (summed per tissue once, after the last step). kLanes lanes per particle
// share candidates, springs and products and add up in a fixed tree, so a row
// costs one or two evaluations in a row instead of ten: 36,864 particles 54 us
// with one thread per particle, 23 with eight lanes. (What the previous kernel
// of the chain wrote is read with ordinary loads, not through restricted
// pointers: the two kernels' lifetimes overlap.)
template <int kLanes>
__global__ void __launch_bounds__(128) k_adj_pairs(DevState S, const double4* lam,
                                                   double4* lam_out,
                                                   const double4* bend,
                                                   double4* gpart) {
  pdl_entry();
  const int64_t N = S.n_total;
  const int sub = (int)threadIdx.x & (kLanes - 1);
  const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  const int64_t i = i0 < N ? i0 : N - 1;
  const uint32_t a = S.attr[i];
  const TissueDev& T = S.tissues[attr_tissue(a)];
  const Laws<double>& L = T.lawd;
  const double dt = T.P.dt;
  const double lt2 = T.P.lj_thresh * T.P.lj_thresh;
  const double4 p = S.pos_cur[i];
  const D3 li = xyz(lam[i]);
  D3 mu = d3(0.0, 0.0, 0.0);
  double g_spring = 0.0, g_eps = 0.0, g_bend = 0.0;
  const uint32_t st = attr_state(a);
  int32_t pair_i = -1, dermis_i = -1;
  if (st != ST_MEMB) {
    pair_i = S.pair[i];
    if (st == ST_FIX || st == ST_MUSUME) dermis_i = S.dermis[i];
  }
  auto add = [&](const LawD& w, const D3& d, int32_t q) {
    const D3 dl = li - xyz(lam[q]);
    mu += dt * (w.c * dl + (2.0 * w.dc_dr2 * dot(d, dl)) * d);
    const double ld = dot(li, d);
    g_spring += dt * w.c_spring * ld;
    g_eps += dt * w.c_eps * ld;
  };
  const int32_t nc = cand_count(S, i);
  for (int32_t k = sub; k < nc; k += kLanes) {
    const int32_t q = T.pbase + (int32_t)cand_entry(S, i, k + 1);
    const double4 pq = S.pos_cur[q];
    const double dx = pdiff_h(p.x, pq.x, T.lx, T.hlx), dy = pdiff_h(p.y, pq.y, T.ly, T.hly);
    const double dz = p.z - pq.z;
    const double r2 = dist_sq_exact(dx, dy, dz);
    const double rs = __dadd_rn(p.w, pq.w);
    if (!(r2 <= __dmul_rn(__dmul_rn(lt2, rs), rs))) continue;  // connect_proc :115-119
    const uint32_t aq = S.attr[q];
    const uint32_t sq = attr_state(aq);
    const bool both_old = attr_old(a) && attr_old(aq);
    const Dist dd = dist_d(r2);
    // the laws i applies while iterating q and q applies while iterating i
    LawD w{0.0, 0.0, 0.0, 0.0};
    if (st != ST_MEMB) {
      const int law = law_of(st, (int32_t)i, pair_i, dermis_i, sq, q);
      if (law != L_NONE) w = w + law_d(law, L, dd, rs, both_old, attr_sfm(a));
    }
    if (sq != ST_MEMB) {
      int32_t pair_q = -1, dermis_q = -1;
      if (sq == ST_FIX || sq == ST_MUSUME) {
        pair_q = S.pair[q];
        dermis_q = S.dermis[q];
      }
      const int law = law_of(sq, q, pair_q, dermis_q, st, (int32_t)i);
      if (law != L_NONE) w = w + law_d(law, L, dd, rs, both_old, attr_sfm(aq));
    }
    add(w, d3(dx, dy, dz), q);
  }
  // _pair_interaction (:637-641): the spring to the partner, from the
  // higher index's rest length, in the separation of pair_sep
  if (pair_i >= 0 && sub == 0) {
    const int32_t q = pair_i;
    const double4 pq = S.pos_cur[q];
    double dx, dy, dz;
    pair_sep(p, pq, i > q, T, dx, dy, dz);
    add(pair_d(L, dist_d(dist_sq_exact(dx, dy, dz)), S.spr[i > q ? i : q]), d3(dx, dy, dz), q);
  }
  if ((st == ST_DER || st == ST_MEMB) && p.z < p.w && sub == kLanes - 1)
    wall_back(L, dt, p.z, p.w, li.z, mu, g_eps);
  if (st == ST_MEMB) {
    const int32_t j = (int32_t)i - T.pbase;
    const int32_t NMX = T.nmx, NMY = T.nmy, jj = j % NMX, kk = j / NMX;
    const bool tri = T.lattice == kLatticeTriangular;
    // lattice springs (each pair from both sides: gather)
    for (int k = sub; k < T.nadj; k += kLanes) {
      const int32_t q = T.pbase + lattice_link(T, j, k);
      const double4 pq = S.pos_cur[q];
      double dx, dy, dz;
      pair_sep(p, pq, i > q, T, dx, dy, dz);
      add(memb_memb_d(L, dist_sq_exact(dx, dy, dz), p.w + pq.w), d3(dx, dy, dz), q);
    }
    // bending products naming this site. Square: slot s of the particle at
    // (jj - dj_s, kk - dk_s), and the second self slot. Triangular: slot 1 + d
    // names this site for its neighbour in the opposite direction (d + 3) %
    // 6; slot 7 + k (the site two links away, along (k + 1) % 6 then k) for
    // the particle reached back along the opposite directions, (k + 3) % 6
    // then (k + 4) % 6.
    const int ns = tri ? kTriSlots : kSlots + 1;
    for (int s = sub; s < ns; s += kLanes) {
      int32_t src = j;
      if (tri) {
        const TriSite s0{jj, kk};
        if (s > 0) {
          const TriSite t =
              s < 7 ? tri_step(s0, (s + 2) % 6, NMX, NMY)
                    : tri_step(tri_step(s0, (s - 4) % 6, NMX, NMY), (s - 3) % 6, NMX, NMY);
          src = t.row * NMX + t.col;
        }
      } else if (s < kSlots) {
        int32_t c = jj - kSlotDj[s], w = kk - kSlotDk[s];
        c += c < 0 ? NMX : 0;
        c -= c >= NMX ? NMX : 0;
        w += w < 0 ? NMY : 0;
        w -= w >= NMY ? NMY : 0;
        src = w * NMX + c;
      }
      const double4 b = bend[(int64_t)(T.mbase + src) * kBendStride + s];
      mu += xyz(b);
      if (src == j && (s == 0 || s == kSelf2)) g_bend += b.w;
    }
  }
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) {
    mu += d3(__shfl_xor_sync(0xffffffffu, mu.x, o), __shfl_xor_sync(0xffffffffu, mu.y, o),
             __shfl_xor_sync(0xffffffffu, mu.z, o));
    g_spring += __shfl_xor_sync(0xffffffffu, g_spring, o);
    g_eps += __shfl_xor_sync(0xffffffffu, g_eps, o);
    g_bend += __shfl_xor_sync(0xffffffffu, g_bend, o);
  }
  if (sub != 0 || i0 >= N) return;
  lam_out[i] = make_double4(li.x + mu.x, li.y + mu.y, li.z + mu.z, 0.0);
  double4 g = gpart[i];
  g.x += g_spring;
  g.y += g_eps;
  g.z += g_bend;
  gpart[i] = g;
}

// lambda at the last step: dL/dX_T of L_t = inv_cnt[t] sum |X_T - X*|^2 over
// the loss set (minimum image in x and y); the loss terms go to gpart.w.
__global__ void k_adj_seed(DevState S, const double* __restrict__ target, int32_t cells_only,
                           const double* __restrict__ inv_cnt, double4* __restrict__ lam,
                           double4* __restrict__ gpart) {
  const int64_t N = S.n_total;
  GRID_STRIDE(i, 0, N) {
    const uint32_t a = S.attr[i];
    const uint32_t t = attr_tissue(a);
    const TissueDev& T = S.tissues[t];
    const double4 p = S.pos_cur[i];
    const bool in = !(cells_only && attr_state(a) == ST_MEMB);
    const double w = in ? inv_cnt[t] : 0.0;
    const double dx = pdiff(p.x, target[i], T.lx);
    const double dy = pdiff(p.y, target[N + i], T.ly);
    const double dz = p.z - target[2 * N + i];
    lam[i] = make_double4(2.0 * w * dx, 2.0 * w * dy, 2.0 * w * dz, 0.0);
    gpart[i] = make_double4(0.0, 0.0, 0.0, w * (dx * dx + dy * dy + dz * dz));
  }
}

// Per tissue, in a fixed order: acc[4 t + c] += sum over its particles of
// gpart[i].{x, y, z, w}.
__global__ void __launch_bounds__(256) k_tissue_sum(DevState S, const double4* __restrict__ gpart,
                                                    double* __restrict__ acc) {
  __shared__ double4 sh[256];
  for (int32_t t = blockIdx.x; t < S.ntissues; t += gridDim.x) {
    const TissueDev& T = S.tissues[t];
    double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
    for (int32_t k = threadIdx.x; k < T.n; k += blockDim.x) {
      const double4 g = gpart[T.pbase + k];
      s.x += g.x;
      s.y += g.y;
      s.z += g.z;
      s.w += g.w;
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
      if ((int)threadIdx.x < h) {
        const double4 o = sh[threadIdx.x + h];
        sh[threadIdx.x].x += o.x;
        sh[threadIdx.x].y += o.y;
        sh[threadIdx.x].z += o.z;
        sh[threadIdx.x].w += o.w;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      acc[4 * t + 0] += sh[0].x;
      acc[4 * t + 1] += sh[0].y;
      acc[4 * t + 2] += sh[0].z;
      acc[4 * t + 3] += sh[0].w;
    }
    __syncthreads();
  }
}

// Flags the tissues whose particles moved more than skin/2 from the
// positions of their last candidate rebuild (the forward step's test, for
// positions loaded from a checkpoint or a stored step).
__global__ void k_gate_check(DevState S) {
  GRID_STRIDE(i, 0, S.n_total) {
    const uint32_t t = attr_tissue(S.attr[i]);
    const TissueDev& T = S.tissues[t];
    const double4 p = S.pos_cur[i];
    const float4 b = S.bpos[i];
    if (moved_too_far(S.skin, T, p.x, p.y, p.z, b)) {
      S.gate[1 + t] = 1;
      S.gate[0] = 1;
    }
  }
}

// k_gate_check over the m position sets in hist. With moved, *moved = 1 stands
// for the flags.
__global__ void k_hist_check(DevState S, const double4* __restrict__ hist, int64_t m,
                             int32_t* moved) {
  GRID_STRIDE(e, 0, m * S.n_total) {
    const int64_t i = e % S.n_total;
    const uint32_t t = attr_tissue(S.attr[i]);
    const double4 p = hist[e];
    if (!moved_too_far(S.skin, S.tissues[t], p.x, p.y, p.z, S.bpos[i])) continue;
    if (moved) {
      *moved = 1;
    } else {
      S.gate[1 + t] = 1;
      S.gate[0] = 1;
    }
  }
}

}  // namespace

void launch_hist_check(const DevState& S, const double4* hist, int32_t m, int32_t* moved,
                       const LaunchCfg& lc, cudaStream_t s) {
  if (S.n_total > 0 && m > 0)
    k_hist_check<<<stride_blocks(S.n_total * m, lc.block, lc), lc.block, 0, s>>>(S, hist, m, moved);
}

void launch_gate_check(const DevState& S, const LaunchCfg& lc, cudaStream_t s) {
  if (S.n_total > 0)
    k_gate_check<<<stride_blocks(S.n_total, lc.block, lc), lc.block, 0, s>>>(S);
}

void launch_adjoint_seed(const DevState& S, const double* target, int32_t cells_only,
                         const double* inv_cnt, double4* lam, double4* gpart,
                         const LaunchCfg& lc, cudaStream_t s) {
  if (S.n_total > 0)
    k_adj_seed<<<stride_blocks(S.n_total, lc.block, lc), lc.block, 0, s>>>(
        S, target, cells_only, inv_cnt, lam, gpart);
}

// Lanes per particle in k_adj_pairs: as many as keep a batch within a wave or
// two of the blocks the GPU holds (36,864 particles, whole 200-step gradient:
// 10.5 ms with four lanes, 11.3 with eight; 11,040 particles 8.9 and 8.6).
constexpr int64_t kEightLanes = 16384, kFourLanes = 262144;

template <int kLanes>
void launch_adj_pairs(const DevState& S, const AdjointBuffers& B, cudaStream_t s) {
  launch_pdl(k_adj_pairs<kLanes>, blocks_for(S.n_total * kLanes, 128), 128, s, S, B.lam_in,
             B.lam_out, B.bend, B.gpart);
}

void launch_adjoint_step(const DevState& S, const AdjointBuffers& B, bool tri, const LaunchCfg& lc,
                         cudaStream_t s) {
  const int64_t nm = S.nprep_memb;
  if (nm > 0 && tri)
    launch_pdl(k_adj_bend<8>, stride_blocks(nm * 8, 64, lc), 64, s, S, B.lam_in, B.bend);
  else if (nm > 0)
    launch_pdl(k_adj_bend<2>, stride_blocks(nm * 2, 64, lc), 64, s, S, B.lam_in, B.bend);
  if (S.n_total <= 0) return;
  if (S.n_total <= kEightLanes) launch_adj_pairs<8>(S, B, s);
  else if (S.n_total <= kFourLanes) launch_adj_pairs<4>(S, B, s);
  else launch_adj_pairs<2>(S, B, s);
}

void launch_tissue_sum(const DevState& S, const double4* gpart, double* acc, const LaunchCfg& lc,
                       cudaStream_t s) {
  const int grid = S.ntissues < lc.num_sms * 8 ? S.ntissues : lc.num_sms * 8;
  if (grid > 0) k_tissue_sum<<<grid, 256, 0, s>>>(S, gpart, acc);
}

}  // namespace epi
