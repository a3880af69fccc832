// Reverse mode of the FP64 sweeps, one direction at a time.
//
// Every sweep of the dynamical core is a flux along x plus a flux along y of
// quantities that need only a point's neighbours in the other direction.  The
// adjoint of the step's update needs the new fields (which the forward
// stored), not the other direction's fluxes, so each sweep is reversed by two
// kernels that meet in global memory:
//  * x kernels: a warp walks a strip of rows upward, a lane a column.  The
//    lines along x (XLineAdj) are evaluated and reversed within the row, their
//    neighbours by warp shuffles; 26 of the 32 columns carry the adjoints of
//    the strip's outputs and the halo lanes receive what these pass on.
//  * y kernels: the same march, with the line along y of each lane's column in
//    registers (YLineAdj): its forward windows, and five rows behind them the
//    reverse ones.  28 to 30 of the 32 columns are the strip's own.
// Each lane sums what its column of a row receives in registers; a finished
// row is added to the global adjoint once (a reduction without return value),
// as neighbouring strips add to the same halo points.
//
// The forward values are recomputed with the forward's operations
// (atm_march.cuh), hence the same limiter and upwind branches.  Derivatives
// follow the branch the forward took; conventions at kinks (shared with the
// oracle's tangent-linear model): d|x|/dx = 0 at x = 0; d copysign(a, b)/da =
// sgn(a) * (sign of b); min/max pass the derivative of the argument they
// return.  A strip whose output adjoints are all zero returns at once (a loss
// over a sub-domain reaches only its domain of dependence).
//
// Bound by the latency of the FP64 chains at the three blocks an SM that the
// registers leave, once the loads run ahead (RowRing).  Measured on B200 at
// 512x512x32 (ms a launch; first: one or two kernels on 32 x 4-8 tiles that
// kept every intermediate and its adjoint in shared memory, with shared-memory
// atomics and block barriers between about ten stages, ~6000 instructions a
// cell; then this march with its loads at their use, then with the rings and
// with the strips of atm_strips.h, every output with an adjoint):
// C mass 3.37, 0.58 + 0.87, 0.36 + 0.45; C momentum 3.27, 1.05, 0.79; D mass
// 3.53, 0.63 + 1.02, 0.47 + 0.63; D momentum 4.16, 0.59 + 0.57, 0.40 + 0.38.
// With the rings, rows unrolled 2 or 3 times gain up to 4% in the momentum x
// kernels and lose 10-25% in the y kernels; four blocks an SM lose 50% there.
#pragma once

#include "atm_march.cuh"

namespace atm {

constexpr double THIRD = 1.0 / 3.0;
constexpr int PGF_CHUNK = 8;  // levels a thread of k_pgf_adj_corners walks

// slope_d and which of |dqi| (0), dm (1), dp (2) it returns: where it is not
// zero the slope is that difference itself, so its adjoint goes there whole
// (3: the slope is zero and passes nothing).
__device__ __forceinline__ double slope_sel(double dm, double dp, double dqi, int& sel) {
  double m = fabs(dqi);
  const double b = xsign(dm, dqi), c = xsign(dp, dqi);
  sel = 0;
  if (b < m) { m = b; sel = 1; }
  if (c < m) { m = c; sel = 2; }
  if (!(m > 0.)) { m = 0.; sel = 3; }
  return copysign(m, dqi);
}

// Reverse of limit_con: the adjoints lL, lR of a cell's limited edges become
// those of its raw edges; ldq gains that of dqi (a limited edge is -+2 dqi).
__device__ __forceinline__ void limit_con_adj(double dqi, double eL, double eR, double& lL, double& lR, double& ldq) {
  const double lim = 2. * fabs(dqi);
  const bool rawL = fabs(eL) < lim, rawR = fabs(eR) < lim;
  if (lim > 0.) ldq += 2. * ((rawR ? 0. : lR) - (rawL ? 0. : lL));
  lL = rawL && eL != 0. ? xsign(xsign(-lL, dqi), eL) : 0.;
  lR = rawR && eR != 0. ? xsign(xsign(lR, dqi), eR) : 0.;
}

// Reverse of limit_nn; lq gains the adjoint of the cell's value (the floors).
__device__ __forceinline__ void limit_nn_adj(double q0, double dqi, double eL, double eR, double& lL, double& lR,
                                             double& ldq, double& lq) {
  if (!(q0 > 6. * fabs(dqi))) {
    double eL1 = eL, eR1 = eR;
    limit_con(dqi, eL1, eR1);
    const bool floorL = eL1 < -q0, floorR = eR1 < -q0;
    const double eL2 = mx(eL1, -q0), eR2 = mx(eR1, -q0);
    const double a = eR2 - eL2, b = -3. * (eR2 + eL2);
    if ((fabs(a) < -b) && (q0 + a * a / (4. * b) + div_const<12>(b) < 0.)) {
      if (eL2 * eR2 > 0.) {  // both edges zero
        lL = 0.;
        lR = 0.;
      } else if (eL2 > eR2) {  // eL = 2 |eR|
        lR += 2. * (eR2 > 0. ? 1. : (eR2 < 0. ? -1. : 0.)) * lL;
        lL = 0.;
      } else {  // eR = 2 |eL|
        lL += 2. * (eL2 > 0. ? 1. : (eL2 < 0. ? -1. : 0.)) * lR;
        lR = 0.;
      }
    }
    if (floorL) { lq -= lL; lL = 0.; }
    if (floorR) { lq -= lR; lR = 0.; }
  }
  limit_con_adj(dqi, eL, eR, lL, lR, ldq);
}

// Reverse of flux_e / flux_con_e with respect to the edges and c: the adjoint
// of the upwind cell's edge at the interface (near) and of its far edge.
__device__ __forceinline__ void flux_e_adj(double c, double eLm, double eRm, double eL0, double eR0, bool flat,
                                           double lamF, double& near, double& far, double& lamc) {
  const bool pos = c > 0.;
  const double sa = fabs(c), lf = flat ? 0. : lamF;
  near = fmx(-2., sa, 1.) * (1. - sa) * lf;
  far = sa * (sa - 1.) * lf;
  const double g = (fmx(4., sa, -3.) * (pos ? eRm : eL0) + fmx(2., sa, -1.) * (pos ? eLm : eR0)) * lf;
  if (c != 0.) lamc += xsign(g, c);
}

// t = inner_e(q, f0, f1, den, rA) reversed: the adjoints of the lower, own and
// upper value of q (f0 is the lower one where p0, f1 the upper where !p1), and
// of den.
__device__ __forceinline__ void inner_e_adj(double q, double f0, double f1, bool p0, bool p1, double den, double rA,
                                            double lam, double& am, double& a0, double& ap, double& lden) {
  const double lf = .5 * den * rA * lam;
  am = p0 ? lf : 0.;
  ap = p1 ? 0. : -lf;
  a0 = .5 * (1. + den) * lam + ((p0 ? 0. : lf) - (p1 ? lf : 0.));
  lden += .5 * (q - rA * (f1 - f0)) * lam;
}

// A line along x, one cell a lane, and its reverse.  forward() gives the flux
// at the interface below the lane's cell (xline_flux); reverse() takes that
// flux's adjoint and gives the adjoint of the lane's value, adding that of c.
// Adjoints given at lanes 3..29 stay within the warp.
template <int V>
struct XLineAdj {
  double q, dqi, eLr, eRr, eL, eR, eLm, eRm, c, F;
  int sel;
  bool flat;
  __device__ __forceinline__ double forward(double q_, double c_) {
    q = q_;
    c = c_;
    const double qL = shfl_up(q, 1), qR = shfl_dn(q, 1);
    const double dm = q - qL;
    dqi = (qR - qL) * 0.25;
    const double m = slope_sel(dm, qR - q, dqi, sel);
    const double h = third(shfl_up(m, 1) - m);
    const double rI = fmx(.5, dm, h);
    eLr = fmx(-.5, dm, h);
    eRr = shfl_dn(rI, 1);
    eL = eLr;
    eR = eRr;
    flat = false;
    if (V == PPM_UNC) {
      eLm = shfl_up(eL, 1);
      eRm = rI;
      F = flux_e(c, qL, eLm, eRm, q, eL, eR);
    } else {
      if (V == PPM_NN) limit_nn(q, dqi, eL, eR);
      else limit_con(dqi, eL, eR);
      eLm = shfl_up(eL, 1);
      eRm = shfl_up(eR, 1);
      if (V == PPM_CON) {
        const unsigned fl = __ballot_sync(0xffffffffu, flat_e(eL, eR));
        const int lane = threadIdx.x & (MW - 1);
        flat = lane > 0 && ((fl >> (lane - 1)) & 3u) == 3u;
        F = flux_con_e(c, qL, eLm, eRm, q, eL, eR, flat);
      } else {
        F = flux_e(c, qL, eLm, eRm, q, eL, eR);
      }
    }
    return F;
  }
  __device__ __forceinline__ double reverse(double lamF, double& lamc) const {
    const int lane = threadIdx.x & (MW - 1);
    const bool pos = c > 0.;
    double near, far;
    flux_e_adj(c, eLm, eRm, eL, eR, flat, lamF, near, far, lamc);
    double lam = (pos ? 0. : lamF) + shfl_dn(pos ? lamF : 0., 1);       // of q, from the upwind value
    double lR = (pos ? near : 0.) + shfl_up(pos ? 0. : far, 1);         // of the upper edge of the cell below
    double lL = (pos ? 0. : near) + shfl_dn(pos ? far : 0., 1);         // of the cell's lower edge
    double ldq = 0.;
    if (V != PPM_UNC) {
      double lRc = shfl_dn(lR, 1);  // of the cell's upper edge
      if (V == PPM_NN) limit_nn_adj(q, dqi, eLr, eRr, lL, lRc, ldq, lam);
      else limit_con_adj(dqi, eLr, eRr, lL, lRc, ldq);
      lR = shfl_up(lRc, 1);
      if (lane == 0) lR = 0.;
    }
    const double lh = lR + lL;
    const double lm = (shfl_dn(lh, 1) - lh) * THIRD;
    if (sel == 0) ldq += lm;
    double ldif = .5 * (lR - lL) + (sel == 1 ? lm : 0.) + shfl_up(sel == 2 ? lm : 0., 1);
    double up = shfl_dn(ldif, 1);
    if (lane == MW - 1) up = 0.;
    lam += (ldif - up) + .25 * (shfl_up(ldq, 1) - shfl_dn(ldq, 1));
    return lam;
  }
};

// A line along y (YLine) and its reverse, five rows behind: after push() of
// row r, flux() is the flux at the interface between cells r-3 and r-2, and
// reverse() of that flux's adjoint gives the adjoint of the value of row r-5.
template <int V>
struct YLineAdj {
  double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  double dif = 0, mono = 0, dqi = 0, rawL = 0;
  double L2 = 0, R2 = 0, L3 = 0, R3 = 0;                            // edges of cells r-2, r-3
  double rL2 = 0, rR2 = 0, rL3 = 0, rR3 = 0, dq2 = 0, dq3 = 0;      // raw edges and dqi of the same (limited lines)
  bool fl2 = false, fl3 = false;
  unsigned sel = 0xff;                                              // slope_sel of cells r-1 (low bits) .. r-4
  double nN = 0, fN = 0, qN = 0;   // what interface r-3 passed to cell r-3: its near and far edge, its value
  double lRp = 0, lh = 0;          // adjoints of the raw upper edge of cell r-4, of h between r-5 and r-4
  double ld4 = 0, ld5 = 0;         // of the differences below cells r-4 (open) and r-5
  double ldq4 = 0, ldq5 = 0, ldq6 = 0;  // of dqi of cells r-4 (open), r-5, r-6
  double ft4 = 0, ft5 = 0;         // of the values of cells r-4, r-5, from the fluxes
  __device__ __forceinline__ void push(double v) {
    const double dn = v - q0;
    const double dq = (v - q1) * 0.25;
    int s;
    const double m = slope_sel(dif, dn, dq, s);
    sel = (sel << 2) | (unsigned)s;
    const double h = third(mono - m);
    L3 = L2;
    R3 = R2;
    L2 = rawL;
    R2 = fmx(.5, dif, h);
    rawL = fmx(-.5, dif, h);
    if (V != PPM_UNC) {
      rL3 = rL2; rR3 = rR2; dq3 = dq2;
      rL2 = L2; rR2 = R2; dq2 = dqi;
      if (V == PPM_NN) {
        limit_nn(q1, dqi, L2, R2);
      } else {
        limit_con(dqi, L2, R2);
        fl3 = fl2;
        fl2 = flat_e(L2, R2);
      }
    }
    q3 = q2; q2 = q1; q1 = q0; q0 = v;
    dif = dn;
    mono = m;
    dqi = dq;
  }
  __device__ __forceinline__ double flux(double c) const {
    if (V == PPM_CON) return flux_con_e(c, q3, L3, R3, q2, L2, R2, fl2 && fl3);
    return flux_e(c, q3, L3, R3, q2, L2, R2);
  }
  __device__ __forceinline__ double reverse(double c, double lamF, double& lamc) {
    const bool pos = c > 0.;
    double near, far;
    flux_e_adj(c, L3, R3, L2, R2, V == PPM_CON && fl2 && fl3, lamF, near, far, lamc);
    double lL = nN + (pos ? far : 0.), lR = fN + (pos ? near : 0.), ft = qN + (pos ? lamF : 0.);  // cell r-3
    nN = pos ? 0. : near;
    fN = pos ? 0. : far;
    qN = pos ? 0. : lamF;
    double ldq = 0.;
    if (V == PPM_NN) limit_nn_adj(q3, dq3, rL3, rR3, lL, lR, ldq, ft);
    if (V == PPM_CON) limit_con_adj(dq3, rL3, rR3, lL, lR, ldq);
    const double lh3 = lRp + lL;  // interface r-3
    double ld3 = .5 * (lRp - lL);
    lRp = lR;
    const double lm = (lh3 - lh) * THIRD;  // slope of cell r-4
    lh = lh3;
    const unsigned s4 = (sel >> 6) & 3u;
    const double q4 = ldq4 + (s4 == 0u ? lm : 0.), d4 = ld4 + (s4 == 1u ? lm : 0.);
    if (s4 == 2u) ld3 += lm;
    const double lam = ft5 + (ld5 - d4) + .25 * (ldq6 - q4);
    ft5 = ft4; ft4 = ft;
    ld5 = d4; ld4 = ld3;
    ldq6 = ldq5; ldq5 = q4; ldq4 = ldq;
    return lam;
  }
};

// The rows a strip is about to need, brought into shared memory by asynchronous
// copies two iterations ahead: NF values a lane and iteration, each lane its own
// (no barrier), DEPTH iterations kept.  Loaded at their use, or a row ahead into
// registers, these left the reverse mass kernels waiting for 3 of 6 cycles an
// issued instruction; the gradient at 512x512x32 went from 52.0 to 45.4 ms.
template <int NF, int DEPTH>
struct RowRing {
  static constexpr int bytes = NF * DEPTH * MW * 8;  // of a warp
  double* p;
  unsigned s;
  __device__ __forceinline__ explicit RowRing(double* sm) {
    p = sm + (threadIdx.x >> 5) * (bytes / 8) + (threadIdx.x & (MW - 1));
    s = (unsigned)__cvta_generic_to_shared(p);
  }
  __device__ __forceinline__ static int slot(int r, int f) { return ((r & (DEPTH - 1)) * NF + f) * MW; }
  __device__ __forceinline__ void copy(int r, int f, const double* g) const {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s + slot(r, f) * 8), "l"(g) : "memory");
  }
  __device__ __forceinline__ static void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  // every group but the newest two has arrived
  __device__ __forceinline__ static void wait() { asm volatile("cp.async.wait_group 2;" ::: "memory"); }
  __device__ __forceinline__ double get(int r, int f) const { return p[slot(r, f)]; }
};

// add v to a global adjoint (ok: the point is stored)
__device__ __forceinline__ void radd(double* f, unsigned i, double v, bool ok) {
  if (ok && v != 0.) atomicAdd(f + i, v);
}

// shuffles that give zero past the warp's ends
__device__ __forceinline__ double up0(double v) {
  const double r = shfl_up(v, 1);
  return (threadIdx.x & (MW - 1)) == 0 ? 0. : r;
}
__device__ __forceinline__ double dn0(double v) {
  const double r = shfl_dn(v, 1);
  return (threadIdx.x & (MW - 1)) == MW - 1 ? 0. : r;
}

// whether any lane's column of rows [y0, y1) of a or b holds a nonzero (own: the lane looks)
__device__ __forceinline__ bool strip_active(const double* a, const double* b, const Geom& g, int y0, int y1,
                                             unsigned xi, bool own) {
  bool any = false;
  if (own)
    for (int y = y0; y < y1; ++y) {
      const unsigned i = row_of(g, y) + xi;
      any = any || a[i] != 0. || b[i] != 0.;
    }
  return __any_sync(0xffffffffu, any);
}

// ======================================================== mass adjoint ====
// Reverse of the C-grid (dpc, ptc from dp, pt, ud, vd) and D-grid (dp, pt from
// dp, pt, uc, vc) mass sweeps, src/mod_sw_dyn.f90:94-270 and 439-600 (heating
// off).  The new pt is q / v with v the new dp; with lv, lq the adjoints of v
// and q, the flux of q at a face is H = (fp + vd (lap pt)') fd.
struct MassAdjArgs {
  const double *dp, *pt, *u, *v, *dpo, *pto, *lam_dpo, *lam_pto;
  double *lam_dp, *lam_pt, *lam_u, *lam_v;
};

// lv, lq of an output point with new fields d, t and their adjoints ld, lt
__device__ __forceinline__ void mass_out_adj(double ld, double lt, double d, double t, double& lv, double& lq) {
  lq = lt / d;
  lv = ld - t * lq;
}

// The x branch: the outer x fluxes, the inner y sweeps, the direct dependence
// of the new fields on the old, and the whole damping of dp.
template <bool CGRID>
__global__ void __launch_bounds__(MW * MWARPS, 3) k_mass_adj_x(Geom g, Consts c, MassAdjArgs a, int lo, int hi, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  constexpr int V = CGRID ? PPM_UNC : PPM_NN;
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int xhi = g.nx - 1 + hi, yhi = g.ny - 1 + hi;
  const int ox = lo + strip_x() * MOUT, oy = lo + (int)blockIdx.y * tys;
  if (ox > xhi) return;
  const int x = ox - MXH + lane, yend = min(oy + tys, yhi + 1);
  const bool own = lane >= MXH && lane < MXH + MOUT && x <= xhi, in = x < g.nx + H;
  const long long kS = (long long)k * g.S;
  const unsigned xi = col_of(g, x), xr = col_of(g, x + 1);
  if (!strip_active(a.lam_dpo + kS, a.lam_pto + kS, g, oy, yend, xi, own)) return;
  const double dtdx = c.dtdx, dtdy = c.dtdy, rA = c.rA;
  const double rdx2 = c.rdx2, rdy2 = c.rdy2, m2rdxy = -2. * c.rdx2rdy2;
  const double dxv = dtdx * c.vdx, dyv = dtdy * c.vdy, vdx = c.vdx;
  const double *dp = a.dp + kS, *pt = a.pt + kS, *u = a.u + kS, *v = a.v + kS;
  double *lam_dp = a.lam_dp + kS, *lam_pt = a.lam_pt + kS, *lam_u = a.lam_u + kS, *lam_v = a.lam_v + kS;

  // iteration r brings rows r+1 of dp, pt, v and u (D grid: row r of u), and
  // row r of the outputs and their adjoints
  enum { F_DP, F_PT, F_U, F_V, F_LD, F_LP, F_DO, F_PO, F_VR };
  const RowRing<CGRID ? 9 : 8, 4> ring(adj_sm);
  auto issue = [&](int r) {
    if (r < yend + 4) {
      const unsigned i1 = row_of(g, r + 1), i0 = row_of(g, r) + xi;
      ring.copy(r, F_DP, dp + (i1 + xi));
      ring.copy(r, F_PT, pt + (i1 + xi));
      ring.copy(r, F_U, u + (CGRID ? i1 + xi : i0));
      ring.copy(r, F_V, v + (i1 + xi));
      if (CGRID) ring.copy(r, F_VR, v + (i1 + xr));
      if (r < yend) {
        ring.copy(r, F_LD, a.lam_dpo + (kS + i0));
        ring.copy(r, F_LP, a.lam_pto + (kS + i0));
        ring.copy(r, F_DO, a.dpo + (kS + i0));
        ring.copy(r, F_PO, a.pto + (kS + i0));
      }
    }
    ring.commit();
  };
  issue(oy);
  issue(oy + 1);
  const unsigned rm = row_of(g, oy - 1), r0 = row_of(g, oy);
  double dm = dp[rm + xi], d0 = dp[r0 + xi], pm = pt[rm + xi], p0 = pt[r0 + xi];
  // C grid: sums of the D-grid winds that the C-grid winds average
  double us = 0., vc0 = v[r0 + xi], vo = 0., vor_ = 0.;
  if constexpr (CGRID) {
    const double ur = u[r0 + xi];
    us = ur + shfl_up(ur, 1);
    vo = vc0;
    vor_ = v[r0 + xr];
    vc0 = .25 * ((vo + v[rm + xi]) + (vor_ + v[rm + xr]));
  }
  double aD2 = 0, aD1 = 0, aD0 = 0, aP2 = 0, aP1 = 0, aP0 = 0;  // adjoints of dp, pt of rows r-2, r-1, r
  double lv1 = 0, lv2 = 0, x1 = 0, alp1 = 0;                    // lv of rows r-1, r-2; x damping term, pt Laplacian's adjoint of r-1
  double lwp = 0, Up = 0, Wp = 0;
#pragma unroll 1
  for (int r = oy; r < yend + 4; ++r) {
    issue(r + 2);
    ring.wait();
    const unsigned ri = row_of(g, r) + xi;
    const double d1 = ring.get(r, F_DP), p1 = ring.get(r, F_PT), ur = ring.get(r, F_U), vn = ring.get(r, F_V);
    double lv = 0., lq = 0.;
    const bool live = r < yend;
    if (live && own) mass_out_adj(ring.get(r, F_LD), ring.get(r, F_LP), ring.get(r, F_DO), ring.get(r, F_PO), lv, lq);
    double uc = ur, vc1 = vn;
    if constexpr (CGRID) {
      const double vnr = ring.get(r, F_VR), su = ur + shfl_up(ur, 1);
      uc = .25 * (us + su);
      us = su;
      vc1 = .25 * ((vn + vo) + (vnr + vor_));
      vo = vn;
      vor_ = vnr;
    }
    double luc = 0., lw = 0., alp = 0., aD = 0., aP = 0., X = 0.;
    const double lvL = up0(lv), lvR = dn0(lv);
    if (live && __any_sync(0xffffffffu, lv != 0. || lq != 0.)) {
      X = dxv * (2. * lv - lvL - lvR);
      const bool c0 = dtdx * vc0 > 0., c1 = dtdx * vc1 > 0.;
      const double den = 1. / (1. - dtdy * (vc1 - vc0));
      const double fd0 = c0 ? dm : d0, fd1 = c1 ? d0 : d1, fp0 = c0 ? pm : p0, fp1 = c1 ? p0 : p1;
      const double cx = dtdx * uc;
      XLineAdj<V> xd, xp;
      const double Fd = xd.forward(inner_e(d0, fd0, fd1, den, rA), cx);
      const double Fp = xp.forward(inner_e(p0, fp0, fp1, den, rA), cx);
      const double fd = Fd * cx;
      const double dLv = lv - lvL, dLq = lq - up0(lq);
      const double lp = (p1 + pm) * rdy2 + ((shfl_dn(p0, 1) + shfl_up(p0, 1)) * rdx2 + p0 * m2rdxy);
      const double lfd = dLv + (Fp + vdx * (lp - shfl_up(lp, 1))) * dLq;
      const double G = fd * dLq;  // the adjoint of fp
      double lc = lfd * Fd;
      const double lamd = xd.reverse(lfd * cx, lc);
      const double lamp = xp.reverse(G, lc);
      luc = dtdx * lc;
      alp = vdx * (G - dn0(G));
      double am, a0, ap, lden = 0.;
      inner_e_adj(d0, fd0, fd1, c0, c1, den, rA, lamd, am, a0, ap, lden);
      aD1 += am;
      aD0 += a0 + lv + p0 * lq;
      aD = ap;
      inner_e_adj(p0, fp0, fp1, c0, c1, den, rA, lamp, am, a0, ap, lden);
      aP1 += am;
      aP0 += a0 + d0 * lq;
      aP = ap;
      lw = dtdy * den * den * lden;
    }
    {  // the damping: al = adjoint of the Laplacians at row r-1, spread over rows r-2 .. r
      const double al = x1 + dyv * (2. * lv1 - lv2 - lv);
      aD2 += rdy2 * al;
      aD1 += m2rdxy * al + rdx2 * (up0(al) + dn0(al));
      aD0 += rdy2 * al;
      aP2 += rdy2 * alp1;
      aP1 += m2rdxy * alp1 + rdx2 * (up0(alp1) + dn0(alp1));
      aP0 += rdy2 * alp1;
    }
    const unsigned e2 = row_of(g, r - 2) + xi;
    radd(lam_dp, e2, aD2, in);
    radd(lam_pt, e2, aP2, in);
    aD2 = aD1; aD1 = aD0; aD0 = aD;
    aP2 = aP1; aP1 = aP0; aP0 = aP;
    lv2 = lv1; lv1 = lv;
    x1 = X;
    alp1 = alp;
    const double W = lwp - lw;  // of the C-grid v of row r
    lwp = lw;
    if constexpr (CGRID) {
      // uc averages u(x), u(x-1) of rows r, r+1; vc averages v(x), v(x+1) of rows r, r-1
      const double U = luc + dn0(luc);
      radd(lam_u, ri, .25 * (U + Up), in);
      Up = U;
      const unsigned e1 = row_of(g, r - 1);
      const double Ws = W + Wp;
      radd(lam_v, e1 + xi, .25 * (Ws + up0(Ws)), in);
      if (lane == MW - 1) radd(lam_v, e1 + xr, .25 * Ws, x + 1 < g.nx + H);
      Wp = W;
    } else {
      radd(lam_u, ri, luc, in);
      radd(lam_v, ri, W, in);
    }
    dm = d0; d0 = d1;
    pm = p0; p0 = p1;
    vc0 = vc1;
  }
}

// The y branch: the outer y fluxes, the inner x sweeps, the y part of the
// damping of pt.  Own columns: lanes 1 to 30.
constexpr int YOUT_MASS = 30;
constexpr int mass_adj_smem(bool cgrid, bool xb) {  // of a warp
  return (!xb ? RowRing<8, 8>::bytes : cgrid ? RowRing<9, 4>::bytes : RowRing<8, 4>::bytes);
}
template <bool CGRID>
__global__ void __launch_bounds__(MW * MWARPS, 3) k_mass_adj_y(Geom g, Consts c, MassAdjArgs a, int lo, int hi, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  constexpr int V = CGRID ? PPM_UNC : PPM_NN;
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int xhi = g.nx - 1 + hi, yhi = g.ny - 1 + hi;
  const int ox = lo + strip_x() * YOUT_MASS, oy = lo + (int)blockIdx.y * tys;
  if (ox > xhi) return;
  const int x = ox - 1 + lane, yend = min(oy + tys, yhi + 1);
  const bool own = lane >= 1 && lane <= YOUT_MASS && x <= xhi, in = x < g.nx + H;
  const long long kS = (long long)k * g.S;
  const unsigned xi = col_of(g, x);
  if (!strip_active(a.lam_dpo + kS, a.lam_pto + kS, g, oy, yend, xi, own)) return;
  const double dtdx = c.dtdx, rA = c.rA;
  const double rdx2 = c.rdx2, rdy2 = c.rdy2, m2rdxy = -2. * c.rdx2rdy2, vdy = c.vdy;
  const double *dp = a.dp + kS, *pt = a.pt + kS, *u = a.u + kS, *v = a.v + kS;
  double *lam_dp = a.lam_dp + kS, *lam_pt = a.lam_pt + kS, *lam_u = a.lam_u + kS, *lam_v = a.lam_v + kS;

  // iteration r brings row r of dp, pt and u (C grid: row r+1 of u), kept until
  // the reverse of the inner sweep at row s = r-5 reads them again, and row i =
  // r-2 of v, the outputs and their adjoints
  enum { F_DP, F_PT, F_U, F_V, F_LD, F_LP, F_DO, F_PO };
  const RowRing<8, 8> ring(adj_sm);
  const int rend = yend + 8 + (CGRID ? 1 : 0);
  auto issue = [&](int r) {
    if (r < rend) {
      const unsigned i0 = row_of(g, r) + xi, ii = row_of(g, r - 2) + xi;
      ring.copy(r, F_DP, dp + i0);
      ring.copy(r, F_PT, pt + i0);
      ring.copy(r, F_U, u + (CGRID ? row_of(g, r + 1) + xi : i0));
      ring.copy(r, F_V, v + ii);
      if (r - 2 >= oy && r - 2 < yend) {
        ring.copy(r, F_LD, a.lam_dpo + (kS + ii));
        ring.copy(r, F_LP, a.lam_pto + (kS + ii));
        ring.copy(r, F_DO, a.dpo + (kS + ii));
        ring.copy(r, F_PO, a.pto + (kS + ii));
      }
    }
    ring.commit();
  };
  issue(oy - 3);
  issue(oy - 2);
  YLineAdj<V> yd, yp;
  double p1 = 0, p2 = 0, ps1 = 0;                   // pt of rows r-1, r-2; pt(x+1) + pt(x-1) of row r-1
  double lp1 = 0, lp2 = 0, lp3 = 0;                 // Laplacian of pt of rows r-1 .. r-3
  double lv3 = 0, lq3 = 0;                          // lv, lq of row r-3
  double Gp = 0, al4 = 0, al5 = 0, al6 = 0;         // adjoint of fp at interface r-3; of pt's Laplacian, rows r-4 .. r-6
  double us = 0, vo = 0, uss = 0, Sp = 0, Up = 0;   // C grid: sums of the winds; row sums of their adjoints
  if constexpr (CGRID) {
    const double ur = u[row_of(g, oy - 3) + xi];
    us = ur + shfl_up(ur, 1);
    uss = us;
    vo = v[row_of(g, oy - 6) + xi];
  }
#pragma unroll 1
  for (int r = oy - 3; r < rend; ++r) {
    issue(r + 2);
    ring.wait();
    const int i = r - 2, s = r - 5;
    const unsigned si = row_of(g, s) + xi, ii = row_of(g, i) + xi;
    double lv = 0., lq = 0.;
    if (i >= oy && i < yend && own)
      mass_out_adj(ring.get(r, F_LD), ring.get(r, F_LP), ring.get(r, F_DO), ring.get(r, F_PO), lv, lq);
    // ---- forward: row r
    const double d = ring.get(r, F_DP), p = ring.get(r, F_PT), ur = ring.get(r, F_U), vr = ring.get(r, F_V);
    double uc = ur, vc = vr;
    if constexpr (CGRID) {
      const double su = ur + shfl_up(ur, 1), sv = vr + vo;
      uc = .25 * (us + su);
      us = su;
      vc = .25 * (sv + shfl_dn(sv, 1));
      vo = vr;
    }
    const double pL = shfl_up(p, 1), pR = shfl_dn(p, 1);
    {
      const double dL = shfl_up(d, 1), dR = shfl_dn(d, 1), ucR = shfl_dn(uc, 1);
      const bool c0 = dtdx * uc > 0., c1 = dtdx * ucR > 0.;
      const double den = 1. / (1. - dtdx * (ucR - uc));
      yd.push(inner_e(d, c0 ? dL : d, c1 ? d : dR, den, rA));
      yp.push(inner_e(p, c0 ? pL : p, c1 ? p : pR, den, rA));
    }
    lp3 = lp2; lp2 = lp1;
    lp1 = (p + p2) * rdy2 + (ps1 * rdx2 + p1 * m2rdxy);
    p2 = p1; p1 = p;
    ps1 = pR + pL;
    // ---- interface i: the fluxes and their adjoints
    const double cy = dtdx * vc;
    const double Fd = yd.flux(cy), Fp = yp.flux(cy);
    const double dLq = lq - lq3;
    const double lfd = (lv - lv3) + (Fp + vdy * (lp2 - lp3)) * dLq;
    const double G = Fd * cy * dLq;
    lv3 = lv;
    lq3 = lq;
    double lc = lfd * Fd;
    const double lamd = yd.reverse(cy, lfd * cy, lc);
    const double lamp = yp.reverse(cy, G, lc);
    const double W = dtdx * lc;
    const double al3 = vdy * (Gp - G);
    Gp = G;
    // ---- row s: the inner x sweep
    double lu = 0.;
    if (s >= oy - 3) {
      const double ds = ring.get(s, F_DP), ps = ring.get(s, F_PT), usr = ring.get(s, F_U);
      double ucs = usr;
      if constexpr (CGRID) {
        const double su = usr + shfl_up(usr, 1);
        ucs = .25 * (uss + su);
        uss = su;
      }
      const double ucR = shfl_dn(ucs, 1);
      const double dL = shfl_up(ds, 1), dR = shfl_dn(ds, 1), qL = shfl_up(ps, 1), qR = shfl_dn(ps, 1);
      const bool c0 = dtdx * ucs > 0., c1 = dtdx * ucR > 0.;
      const double den = 1. / (1. - dtdx * (ucR - ucs));
      double am, a0, ap, lden = 0.;
      inner_e_adj(ds, c0 ? dL : ds, c1 ? ds : dR, c0, c1, den, rA, lamd, am, a0, ap, lden);
      radd(lam_dp, si, a0 + dn0(am) + up0(ap), in);
      inner_e_adj(ps, c0 ? qL : ps, c1 ? ps : qR, c0, c1, den, rA, lamp, am, a0, ap, lden);
      radd(lam_pt, si, a0 + dn0(am) + up0(ap) + rdy2 * (al6 + al4) + (m2rdxy * al5 + rdx2 * (up0(al5) + dn0(al5))),
           in);
      const double lw = dtdx * den * den * lden;
      lu = up0(lw) - lw;
    }
    al6 = al5; al5 = al4; al4 = al3;
    if constexpr (CGRID) {
      const double U = lu + dn0(lu);
      radd(lam_u, si, .25 * (U + Up), in);
      Up = U;
      const double S = W + up0(W);
      radd(lam_v, row_of(g, i - 1) + xi, .25 * (S + Sp), in);
      Sp = S;
    } else {
      radd(lam_u, si, lu, in);
      radd(lam_v, ii, W, in);
    }
  }
}

// ================================================== C-momentum adjoint ====
// Reverse of the C-grid momentum sweep, src/mod_sw_dyn.f90:294-414: uc, vc of
// layer k from ud, vd of layers k and nlay and pkap, gz of levels k, k+1.  The
// two branches leave the adjoints of the vorticity (lam_w), of the C-grid winds
// as advected quantities (lam_uc1, lam_vc1) and, summed over the layers, of
// the layer-nlay A-grid winds (lam_ua, lam_va, one level each) in scratch
// fields, which k_c_mom_adj_fin turns into those of ud, vd; the
// pressure-gradient force is reversed with the columns (k_column_adj<true>).
struct CMomAdjArgs {
  const double *ud, *vd, *lam_uc, *lam_vc;
  double *lam_ud, *lam_vd, *lam_w, *lam_uc1, *lam_vc1, *lam_ua, *lam_va;
};

// The x branch: the x fluxes of the vorticity and of the kinetic energy, the
// damping.
static __global__ void __launch_bounds__(MW * MWARPS, 3) k_c_mom_adj_x(Geom g, Consts c, CMomAdjArgs a, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int ox = strip_x() * MOUT, oy = (int)blockIdx.y * tys;
  if (ox >= g.nx) return;
  const int x = ox - MXH + lane, yend = min(oy + tys, g.ny);
  const bool own = lane >= MXH && lane < MXH + MOUT && x < g.nx, in = x < g.nx + H;
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const unsigned xi = col_of(g, x), xl = col_of(g, x - 1), xr = col_of(g, x + 1);
  const double *lam_uc = a.lam_uc + kS, *lam_vc = a.lam_vc + kS;
  if (!strip_active(lam_uc, lam_vc, g, oy, yend, xi, own)) return;
  const double dt = c.dt, dtdx = c.dtdx, dtdy = c.dtdy, rA = c.rA, rdx = c.rdx, rdy = c.rdy, f = c.coriolis;
  const double rdx2 = c.rdx2, rdy2 = c.rdy2, m2rdxy = -2. * c.rdx2rdy2, vdx = c.vdx, vdy = c.vdy;
  const double *ud = a.ud + kS, *vd = a.vd + kS, *uL = a.ud + LS;
  double *lam_ud = a.lam_ud + kS, *lam_vd = a.lam_vd + kS, *lam_w = a.lam_w + kS, *lam_uc1 = a.lam_uc1 + kS;

  // iteration r brings rows r+2 of ud, r+1 of vd and of layer-nlay ud, r of lam_uc, lam_vc
  enum { F_U, F_UL, F_V, F_VR, F_UN, F_LU, F_LV };
  const RowRing<7, 4> ring(adj_sm);
  auto issue = [&](int r) {
    if (r < yend + 3) {
      const unsigned r0 = row_of(g, r) + xi, r1 = row_of(g, r + 1), r2 = row_of(g, r + 2);
      ring.copy(r, F_U, ud + (r2 + xi));
      ring.copy(r, F_UL, ud + (r2 + xl));
      ring.copy(r, F_V, vd + (r1 + xi));
      ring.copy(r, F_VR, vd + (r1 + xr));
      ring.copy(r, F_UN, uL + (r1 + xi));
      if (r < yend) {
        ring.copy(r, F_LU, lam_uc + r0);
        ring.copy(r, F_LV, lam_vc + r0);
      }
    }
    ring.commit();
  };
  issue(oy);
  issue(oy + 1);
  // rows of the layer's C-grid winds and vorticity: a0 = uc1(r), aN = uc1(r+1), w = vor(r-1, r, r+1)
  auto uavg = [&](unsigned ra, unsigned rb) { return .25 * ((ud[ra + xi] + ud[ra + xl]) + (ud[rb + xi] + ud[rb + xl])); };
  auto vavg = [&](unsigned ra, unsigned rb) { return .25 * ((vd[rb + xi] + vd[ra + xi]) + (vd[rb + xr] + vd[ra + xr])); };
  unsigned q2 = row_of(g, oy - 2), q1 = row_of(g, oy - 1), q0 = row_of(g, oy), p1 = row_of(g, oy + 1);
  double uc_m = uavg(q2, q1), uc_0 = uavg(q1, q0), uc_1 = uavg(q0, p1);  // uc1 of rows oy-2, oy-1, oy
  double vc_0 = vavg(q2, q1), vc_1 = vavg(q1, q0);                       // vc1 of rows oy-1, oy
  double wm = f - (uc_0 - uc_m) * rdy + (vc_0 - shfl_up(vc_0, 1)) * rdx;
  double w0 = f - (uc_1 - uc_0) * rdy + (vc_1 - shfl_up(vc_1, 1)) * rdx;
  double ucr = uc_1, ucm = uc_0;                 // uc1 of rows r, r-1
  double v_m = vd[q1 + xi], v_0 = vd[q0 + xi];   // vd(x) of rows r-1, r
  double vR0 = vd[q0 + xr];                      // vd(x+1) of row r
  double u0 = ud[q0 + xi], u1 = ud[p1 + xi];     // ud(x) of rows r, r+1
  double su1 = u1 + ud[p1 + xl];                 // ud(x) + ud(x-1) of row r+1
  double uLm = uL[q1 + xi], uL0 = uL[q0 + xi];   // layer-nlay ud of rows r-1, r
  double lu1 = 0, lv1 = 0, lwd1 = 0;             // lam_uc, lam_vc, den's adjoint of row r-1
  double aW1 = 0, aW0 = 0;                       // adjoints of the vorticity of rows r-1, r
#pragma unroll 1
  for (int r = oy; r < yend + 3; ++r) {
    issue(r + 2);
    ring.wait();
    const unsigned rr = row_of(g, r);
    const bool live = r < yend;
    double lu = 0., lv = 0.;
    if (live && own) {
      lu = ring.get(r, F_LU);
      lv = ring.get(r, F_LV);
    }
    const double u2 = ring.get(r, F_U), su2 = u2 + ring.get(r, F_UL);
    const double v_n = ring.get(r, F_V), vR_n = ring.get(r, F_VR), uL1 = ring.get(r, F_UN);
    const double uc_n = .25 * (su1 + su2), vc_n = .25 * ((v_n + v_0) + (vR_n + vR0));
    const double wp = f - (uc_n - ucr) * rdy + (vc_n - shfl_up(vc_n, 1)) * rdx;
    double lwd = 0., aW = 0.;
    if (live && __any_sync(0xffffffffu, lv != 0.)) {
      // v = vc1 - dt (ud fx + ...): the flux above the cell, reversed as the one below the next lane's
      const bool c0 = dtdx * v_m > 0., c1 = dtdx * v_0 > 0.;
      const double den = 1. / (1. - dtdy * (v_0 - v_m));
      const double f0 = c0 ? wm : w0, f1 = c1 ? w0 : wp;
      XLineAdj<PPM_UNC> ln;
      const double F = shfl_dn(ln.forward(inner_e(w0, f0, f1, den, rA), shfl_up(dtdx * u0, 1)), 1);
      double lcb = 0.;
      const double lt = ln.reverse(up0(-dt * u0 * lv), lcb);
      const double lc = dn0(lcb);
      radd(lam_ud, rr + xi, own ? -dt * F * lv + dtdx * lc : 0., in);
      double am, a0, ap, lden = 0.;
      inner_e_adj(w0, f0, f1, c0, c1, den, rA, lt, am, a0, ap, lden);
      lwd = dtdy * den * den * lden;
      aW1 += am;
      aW0 += a0;
      aW = ap;
    }
    // kinetic energy of row r-1 (:299-317) with the layer-nlay A-grid winds
    const double lke = -dtdx * (lu1 - dn0(lu1)) - dtdy * (lv1 - lv);
    if (r <= yend && __any_sync(0xffffffffu, lke != 0.)) {
      const double ub = .5 * (uLm + shfl_up(uLm, 1));
      const double ucl = .5 * (ub + .5 * (uL0 + shfl_up(uL0, 1)));
      const double ua = .5 * (ucl + .25 * (shfl_dn(uLm, 1) + uLm + shfl_dn(uL0, 1) + uL0));
      XLineAdj<PPM_UNC> ln;
      const double F = shfl_dn(ln.forward(ucm, shfl_up(dtdx * ua, 1)), 1);
      double lcb = 0.;
      const double l1 = ln.reverse(up0(.5 * ua * lke), lcb);
      const double lua = .5 * F * lke + dtdx * dn0(lcb);
      const unsigned rm = row_of(g, r - 1) + xi;
      radd(lam_uc1, rm, l1, in);
      radd(a.lam_ua, rm, lke != 0. ? lua : 0., in);
    }
    // the damping: the adjoint of the vorticity's Laplacian at row r
    const double al = dt * vdy * (lu1 - lu) + dt * vdx * (lv - up0(lv));
    aW1 += rdy2 * al;
    aW0 += m2rdxy * al + rdx2 * (up0(al) + dn0(al));
    aW += rdy2 * al;
    const unsigned rm = row_of(g, r - 1) + xi;
    radd(lam_w, rm, aW1, in);
    radd(lam_vd, rm, lwd1 - lwd, in);
    aW1 = aW0;
    aW0 = aW;
    lu1 = lu;
    lv1 = lv;
    lwd1 = lwd;
    ucm = ucr;
    ucr = uc_n;
    wm = w0;
    w0 = wp;
    v_m = v_0;
    v_0 = v_n;
    vR0 = vR_n;
    u0 = u1;
    u1 = u2;
    su1 = su2;
    uLm = uL0;
    uL0 = uL1;
  }
}

// The y branch: the y fluxes of the vorticity and of the kinetic energy.  Own
// columns: lanes 2 to 29, over [-1, n-1] (the kinetic energy's range).
constexpr int YOUT_CMOM = 28;
static __global__ void __launch_bounds__(MW * MWARPS, 3) k_c_mom_adj_y(Geom g, Consts c, CMomAdjArgs a, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int ox = -1 + strip_x() * YOUT_CMOM, oy = -1 + (int)blockIdx.y * tys;
  if (ox >= g.nx) return;
  const int x = ox - 2 + lane, yend = min(oy + tys, g.ny);
  const bool own = lane >= 2 && lane < 2 + YOUT_CMOM && x < g.nx, in = x < g.nx + H;
  const bool dom = x >= 0 && x < g.nx;
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const unsigned xi = col_of(g, x);
  const double *lam_uc = a.lam_uc + kS, *lam_vc = a.lam_vc + kS;
  if (!strip_active(lam_uc, lam_vc, g, max(oy, 0), min(yend + 1, g.ny), xi, dom)) return;
  const double dt = c.dt, dtdx = c.dtdx, dtdy = c.dtdy, rA = c.rA, rdx = c.rdx, rdy = c.rdy, f = c.coriolis;
  const double *ud = a.ud + kS, *vd = a.vd + kS, *vL = a.vd + LS;
  double *lam_ud = a.lam_ud + kS, *lam_vd = a.lam_vd + kS, *lam_w = a.lam_w + kS, *lam_vc1 = a.lam_vc1 + kS;

  // iteration r brings rows r+1 of ud and r of vd and, with y = r-3, rows y of
  // lam_uc, y+1 of lam_vc, y of vd, r-5 of ud and y+1 of layer-nlay vd
  enum { F_U, F_V, F_LU, F_LV, F_VY, F_US, F_VN };
  const RowRing<7, 4> ring(adj_sm);
  auto issue = [&](int r) {
    if (r < yend + 8) {
      const int y = r - 3;
      const unsigned y0 = row_of(g, y) + xi, y1 = row_of(g, y + 1) + xi;
      ring.copy(r, F_U, ud + (row_of(g, r + 1) + xi));
      ring.copy(r, F_V, vd + (row_of(g, r) + xi));
      if (y >= 0 && y < g.ny) ring.copy(r, F_LU, lam_uc + y0);
      if (y >= -1 && y < g.ny - 1) ring.copy(r, F_LV, lam_vc + y1);
      ring.copy(r, F_VY, vd + y0);
      ring.copy(r, F_US, ud + (row_of(g, r - 5) + xi));
      ring.copy(r, F_VN, vL + y1);
    }
    ring.commit();
  };
  issue(oy - 2);
  issue(oy - 1);
  YLineAdj<PPM_UNC> lt, lb;  // the inner x sweep of the vorticity, the layer's C-grid v, along y
  double w0 = 0, w1 = 0, w2 = 0, w3 = 0, w4 = 0, w5 = 0;  // vorticity of rows r .. r-5
  int r = oy - 2;
  unsigned rm = row_of(g, r - 1), r0 = row_of(g, r);
  double u0 = ud[r0 + xi];                                  // ud of row r
  double us = u0 + shfl_up(u0, 1);                          // u(x) + u(x-1) of row r
  double ucp = ud[rm + xi];                                 // uc1 of row r-1
  ucp = .25 * ((ucp + shfl_up(ucp, 1)) + us);
  double vo = vd[rm + xi];                                  // vd of row r-1
  // layer-nlay vd of rows y-1, y with y = r-3
  double vL2 = vL[row_of(g, r - 4) + xi], vL1 = vL[row_of(g, r - 3) + xi];
  double lv3 = 0;                                           // lam_vc of row y
#pragma unroll 1
  for (; r < yend + 8; ++r) {
    issue(r + 2);
    ring.wait();
    const int y = r - 3, s = r - 5;
    const unsigned yi = row_of(g, y) + xi, si = row_of(g, s) + xi;
    const bool ownr = own && y >= oy && y < yend;
    double lu = 0., lvn = 0.;  // lam_uc of row y, lam_vc of row y+1, over the domain
    if (dom && y >= 0 && y < g.ny) lu = ring.get(r, F_LU);
    if (dom && y >= -1 && y < g.ny - 1) lvn = ring.get(r, F_LV);
    const double vy = ring.get(r, F_VY), uxs = ring.get(r, F_US), vL0 = ring.get(r, F_VN);
    // ---- forward: row r
    const double u1 = ring.get(r, F_U), v = ring.get(r, F_V);
    const double su = u1 + shfl_up(u1, 1), sv = v + vo;
    const double uc = .25 * (us + su), vc = .25 * (sv + shfl_dn(sv, 1));
    const double w = f - (uc - ucp) * rdy + (vc - shfl_up(vc, 1)) * rdx;
    w5 = w4; w4 = w3; w3 = w2; w2 = w1; w1 = w0; w0 = w;
    {
      const double wl = shfl_up(w, 1), wr = shfl_dn(w, 1), um = shfl_up(u0, 1);
      const double den = 1. / (1. - dtdx * (u0 - um));
      lt.push(inner_e(w, dtdx * um > 0. ? wl : w, dtdx * u0 > 0. ? w : wr, den, rA));
    }
    lb.push(vc);
    us = su;
    u0 = u1;
    ucp = uc;
    vo = v;
    // ---- the fluxes above row y (interface r-2) and their adjoints
    {
      const double cy = dtdx * vy, luo = ownr ? lu : 0.;
      const double F = lt.flux(cy);
      double lc = 0.;
      const double lamt = lt.reverse(cy, dt * vy * luo, lc);
      radd(lam_vd, yi, ownr ? dt * F * luo + dtdx * lc : 0., in);
      // row s: the inner x sweep
      const double wl = shfl_up(w5, 1), wr = shfl_dn(w5, 1), um = shfl_up(uxs, 1);
      const bool c0 = dtdx * um > 0., c1 = dtdx * uxs > 0.;
      const double den = 1. / (1. - dtdx * (uxs - um));
      double am, a0, ap, lden = 0.;
      inner_e_adj(w5, c0 ? wl : w5, c1 ? w5 : wr, c0, c1, den, rA, lamt, am, a0, ap, lden);
      radd(lam_w, si, a0 + dn0(am) + up0(ap), in);
      const double lw = dtdx * den * den * lden;
      radd(lam_ud, si, lw - dn0(lw), in);
    }
    {
      // kinetic energy of row y (:299-317) with the layer-nlay A-grid winds
      const double lur = shfl_dn(lu, 1);
      const double lke = ownr ? -dtdx * (lu - lur) - dtdy * (lv3 - lvn) : 0.;
      const double vb = .5 * (vL1 + vL2);
      const double vL1r = shfl_dn(vL1, 1);
      const double vcl = .5 * (vb + .5 * (vL1r + shfl_dn(vL2, 1)));
      const double va = .5 * (vcl + .25 * (vL0 + vL1 + shfl_dn(vL0, 1) + vL1r));
      const double cy = dtdy * va, F = lb.flux(cy);
      double lc = 0.;
      const double lamb = lb.reverse(cy, .5 * va * lke, lc);
      radd(a.lam_va, yi, ownr ? .5 * F * lke + dtdy * lc : 0., in);
      radd(lam_vc1, si, lamb, in);
    }
    lv3 = lvn;
    vL2 = vL1;
    vL1 = vL0;
  }
}

// lam_ud, lam_vd += the adjoints of the layer's C-grid winds (their direct
// terms lam_uc, lam_vc, their part in the vorticity and as advected
// quantities) through the averages that form them (:110-117), and, in layer
// nlay, of the A-grid winds of the kinetic energy.  A thread a column of
// [-4, n+3]^2, blockIdx.y its first row and gridDim.y the step to the next (a
// grid holds 65535 rows of blocks, a domain may have more), blockIdx.z the layer.
static __global__ void __launch_bounds__(128) k_c_mom_adj_fin(Geom g, Consts c, CMomAdjArgs a) {
  stream_order();
  const int x = -4 + (int)(blockIdx.x * blockDim.x + threadIdx.x), k = blockIdx.z;
  if (x >= g.nx + 4) return;
  const int P = g.P;
  auto inx = [&](int q) { return q >= 0 && q < g.nx; };
  auto iny = [&](int q) { return q >= 0 && q < g.ny; };
  for (int y = -4 + (int)blockIdx.y; y < g.ny + 4; y += gridDim.y) {
    const long long o = g.at(x, y, k);
    const double* w = a.lam_w + o;
    const double *s2 = a.lam_uc1 + o, *s3 = a.lam_vc1 + o, *lu = a.lam_uc + o, *lv = a.lam_vc + o;
    const double wy = (w[-P] - w[P]) + (w[1 - P] - w[1 + P]);
    const double wx = (w[-1] - w[1]) + (w[P - 1] - w[P + 1]);
    double su = (s2[0] + s2[1]) + (s2[-P] + s2[1 - P]);
    double sv = (s3[0] + s3[P]) + (s3[-1] + s3[P - 1]);
    if (iny(y)) su += (inx(x) ? lu[0] : 0.) + (inx(x + 1) ? lu[1] : 0.);
    if (iny(y - 1)) su += (inx(x) ? lu[-P] : 0.) + (inx(x + 1) ? lu[1 - P] : 0.);
    if (iny(y)) sv += (inx(x) ? lv[0] : 0.) + (inx(x - 1) ? lv[-1] : 0.);
    if (iny(y + 1)) sv += (inx(x) ? lv[P] : 0.) + (inx(x - 1) ? lv[P - 1] : 0.);
    double du = .25 * (su - c.rdy * wy), dv = .25 * (sv + c.rdx * wx);
    if (k == g.L - 1) {
      const double *A = a.lam_ua + g.at(x, y), *B = a.lam_va + g.at(x, y);
      du += .25 * (A[0] + A[-P]) + .125 * ((A[1] + A[-1]) + (A[1 - P] + A[-1 - P]));
      dv += .25 * (B[0] + B[-1]) + .125 * ((B[P] + B[-P]) + (B[P - 1] + B[-P - 1]));
    }
    if (du != 0.) a.lam_ud[o] += du;
    if (dv != 0.) a.lam_vd[o] += dv;
  }
}

// The four-point pressure-gradient term between two neighbours a (lower index)
// and b, src/mod_sw_dyn.f90:325-339 and 665-679:
//   pg = ((pb0 - pa1)(za0 - zb1) + (pa0 - pb1)(za1 - zb0)) / (pb0 - pa1 + pa0 - pb1)
// with 0, 1 the levels below and above the layer.  Adds lam times its
// derivatives with respect to one side's pressures and geopotentials.
struct PgfPoint {
  double p0, p1, z0, z1;
};
__device__ __forceinline__ void pgf_adj_a(const PgfPoint& A, const PgfPoint& B, double lam, PgfPoint& l) {
  const double a = B.p0 - A.p1, b = A.z0 - B.z1, cc = A.p0 - B.p1, d = A.z1 - B.z0;
  const double rD = 1. / (a + cc);
  const double pg = (a * b + cc * d) * rD, q = lam * rD;
  l.p1 -= (b - pg) * q;
  l.p0 += (d - pg) * q;
  l.z0 += a * q;
  l.z1 += cc * q;
}
__device__ __forceinline__ void pgf_adj_b(const PgfPoint& A, const PgfPoint& B, double lam, PgfPoint& l) {
  const double a = B.p0 - A.p1, b = A.z0 - B.z1, cc = A.p0 - B.p1, d = A.z1 - B.z0;
  const double rD = 1. / (a + cc);
  const double pg = (a * b + cc * d) * rD, q = lam * rD;
  l.p0 += (b - pg) * q;
  l.p1 -= (d - pg) * q;
  l.z1 -= a * q;
  l.z0 -= cc * q;
}

// What a layer's wind adjoints pass to the pressures and geopotentials of one
// column through the pressure-gradient force: lu, lv at the column's own
// lower faces and at its upper ones, times dtdx, dtdy.  CGRID: the force at
// (x, y) is between (x-1, y), (x, y) and (x, y-1), (x, y); D grid: between
// (x, y), (x+1, y) and (x, y), (x, y+1).
template <bool CGRID>
struct PgfColumn {
  const double *pk, *gz, *lam_u, *lam_v;
  Geom g;
  int x, y;
  long long o;
  double fx, fy;
  bool ul, uh, vl, vh;  // which of the four faces lie in the domain
  __device__ __forceinline__ PgfColumn(const Geom& g_, const Consts& c, const double* pk_, const double* gz_,
                                       const double* lu, const double* lv, int x_, int y_)
      : pk(pk_), gz(gz_), lam_u(lu), lam_v(lv), g(g_), x(x_), y(y_), o(g_.at(x_, y_)), fx(c.dtdx), fy(c.dtdy) {
    const int xl = CGRID ? x : x - 1, yl = CGRID ? y : y - 1;  // the faces' indices
    const bool xin = x >= 0 && x < g.nx, yin = y >= 0 && y < g.ny;
    ul = yin && xl >= 0 && xl < g.nx;
    uh = yin && xl + 1 >= 0 && xl + 1 < g.nx;
    vl = xin && yl >= 0 && yl < g.ny;
    vh = xin && yl + 1 >= 0 && yl + 1 < g.ny;
  }
  __device__ __forceinline__ PgfPoint point(long long q) const {
    return PgfPoint{pk[q], pk[q + g.S], gz[q], gz[q + g.S]};
  }
  // adjoints of this column's pkap, gz at levels k (p0, z0) and k+1 (p1, z1)
  __device__ __forceinline__ PgfPoint layer(int k) const {
    PgfPoint l{0., 0., 0., 0.};
    const long long q = o + (long long)k * g.S;
    const int dx = CGRID ? 0 : -1, dy = CGRID ? 0 : -g.P;
    const double a = ul ? lam_u[q + dx] : 0., b = uh ? lam_u[q + dx + 1] : 0.;
    const double d = vl ? lam_v[q + dy] : 0., e = vh ? lam_v[q + dy + g.P] : 0.;
    if (a == 0. && b == 0. && d == 0. && e == 0.) return l;
    const PgfPoint own = point(q);
    if (a != 0.) pgf_adj_b(point(q - 1), own, fx * a, l);
    if (b != 0.) pgf_adj_a(own, point(q + 1), fx * b, l);
    if (d != 0.) pgf_adj_b(point(q - g.P), own, fy * d, l);
    if (e != 0.) pgf_adj_a(own, point(q + g.P), fy * e, l);
    return l;
  }
};

// Reverse of the C grid's columns (k_column: plev = ptop + suffix sums of dp,
// pkap = plev**kappa, gz(k+1) = gz(k) + cp pt(k) (pkap(k) - pkap(k+1)) from the
// fixed surface gz, src/mod_sw_dyn.f90:276-292) and of the pressure-gradient
// force of the momentum sweep that reads them, over [-2, n+1]^2.  D grid
// (:606-626): lam_u, lam_v are the adjoints of pkap and gz that the corners gave.
// A block owns 32 columns (lane = column), its warps share the layers, whose
// terms are independent but for three running sums of 32 columns each, which one
// warp forms; the sums and the terms lie in shared memory (four arrays).
// Measured on B200 (ms, C grid's / D grid's; before: a thread a column, its layers
// one after the other): 64x64x20 0.059 / 0.055 -> 0.020 / 0.029, 301x203x40 0.160 /
// 0.113 -> 0.116 / 0.084; 4 or 16 warps a block: 10 to 20% slower there.
constexpr int CADJ_WARPS = 8;
inline size_t column_adj_smem(int L) { return (size_t)4 * L * 32 * sizeof(double); }
// columns up to which this is the faster form
inline long long column_adj_few(int L) {
  const long long blocks = (long long)(228 * 1024 / (column_adj_smem(L) + 1024)), most = blocks > 2 ? 640 : 170 * blocks;
  return 148 * (45 * L < most ? 45 * L : most);
}
template <bool CGRID>
__global__ void __launch_bounds__(32 * CADJ_WARPS) k_column_adj(Geom g, Consts c, const double* dpl,
                                                                const double* ptl,
                                                                const double* pkap,
                                                                const double* gz,
                                                                const double* lam_u,
                                                                const double* lam_v, double* lam_dp,
                                                                double* lam_pt) {
  stream_order();
  extern __shared__ double adj_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w = g.nx + 4, L = g.L;
  const int col = blockIdx.x * 32 + lane;
  const bool in = col < w * (g.ny + 4);
  const int x = in ? -2 + col % w : 0, y = in ? -2 + col / w : 0;
  const long long o = g.at(x, y), S = g.S;
  // Q: adjoint of pkap(k), then of plev(k); Z: of gz(k+1), then what the layer
  // takes from pkap(k+1); PL, PK: plev, pkap (before: what layer k gives to
  // pkap(k+1) and to gz(k))
  double *Q = adj_sm + lane, *Z = Q + 32 * L, *PL = Z + 32 * L, *PK = PL + 32 * L;
  if constexpr (CGRID) {
    const PgfColumn<true> pgf(g, c, pkap, gz, lam_u, lam_v, x, y);
    for (int k = warp; k < L; k += CADJ_WARPS) {
      const PgfPoint l = pgf.layer(k);
      Q[32 * k] = l.p0;
      PL[32 * k] = l.p1;
      Z[32 * k] = l.z1;
      PK[32 * k] = l.z0;
    }
    __syncthreads();
    for (int k = warp; k < L; k += CADJ_WARPS) {
      if (k > 0) Q[32 * k] += PL[32 * (k - 1)];
      if (k + 1 < L) Z[32 * k] += PK[32 * (k + 1)];
    }
  } else {
    for (int k = warp; k < L; k += CADJ_WARPS) {
      const long long ok = o + (long long)k * S;
      Q[32 * k] = lam_u[ok];
      Z[32 * k] = lam_v[ok + S];
    }
  }
  __syncthreads();
  if (warp == 0) {
    double lz = 0.;
#pragma unroll 4
    for (int k = L - 1; k >= 0; --k) {
      lz += Z[32 * k];
      Z[32 * k] = lz;
    }
  } else if (warp == 1) {
    double pl = c.ptop;
#pragma unroll 8
    for (int k = L - 1; k >= 0; --k) {
      pl = pl + dpl[o + (long long)k * S];
      PL[32 * k] = pl;
    }
  }
  if constexpr (!CGRID) __syncthreads();
  for (int k = warp; k < L; k += CADJ_WARPS) PK[32 * k] = CGRID ? pkap[o + (long long)k * S] : atm_pow(PL[32 * k], KAPPA);
  __syncthreads();
  for (int k = warp; k < L; k += CADJ_WARPS) {
    const long long ok = o + (long long)k * S;
    const double lz = Z[32 * k], cpz = CP_DRY * ptl[ok] * lz;
    if (in) lam_pt[ok] += CP_DRY * (PK[32 * k] - (k + 1 < L ? PK[32 * (k + 1)] : c.pk_top)) * lz;
    Z[32 * k] = cpz;
  }
  __syncthreads();
  for (int k = warp; k < L; k += CADJ_WARPS)
    Q[32 * k] = (Q[32 * k] + Z[32 * k] - (k > 0 ? Z[32 * (k - 1)] : 0.)) * KAPPA * PK[32 * k] / PL[32 * k];
  __syncthreads();
  if (warp == 0) {
    double acc = 0.;
#pragma unroll 4
    for (int k = 0; k < L; ++k) {
      acc += Q[32 * k];
      Q[32 * k] = acc;
    }
  }
  __syncthreads();
  if (!in) return;
  for (int k = warp; k < L; k += CADJ_WARPS) lam_dp[o + (long long)k * S] += Q[32 * k];
}

// The same with a thread a column, its layers in turn; the terms of a layer that its
// neighbours complete wait a turn.  For domains of more columns than column_adj_few:
// the warps of a block that wait for the sums are hidden by other blocks only while an
// SM holds several, and few layers leave them idle.  Measured on B200 (us, C grid's
// column stage, D grid's with the corners; shared levels / a thread a column; columns
// in thousands): 3 layers 31 25/23 26/24, 1049 433/150 337/141; 12 layers 66 82/77 65/67,
// 262 239/152 222/159; 20 layers 66 113/115 91/103, 96 148/122 132/118; 40 layers 96 228/230 223/234,
// 262 523/521 534/489; 64 layers 66 289/326 272/311, 262 963/826 952/765; 100 layers (two blocks an SM)
// 31 318/430 270/374, 66 627/511 520/413; 128 (one) 16 356/529 262/425, 31 619/570 456/472, 160 2729/1217 2160/904.
template <int LM, bool CGRID>
__global__ void __launch_bounds__(128) k_column_adj_columns(Geom g, Consts c, const double* dpl,
                                                            const double* ptl,
                                                            const double* pkap,
                                                            const double* gz,
                                                            const double* lam_u,
                                                            const double* lam_v, double* lam_dp,
                                                            double* lam_pt) {
  stream_order();
  const int w = g.nx + 4, L = g.L, col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= w * (g.ny + 4)) return;
  const int x = -2 + col % w, y = -2 + col / w;
  const long long o = g.at(x, y), S = g.S;
  const PgfColumn<true> pgf(g, c, pkap, gz, lam_u, lam_v, x, y);
  double q[LM];  // adjoint of plev(k)
  double pl = c.ptop, lz = 0.;
  double pl1 = 1., pk1 = c.pk_top, q1 = 0., cpz1 = 0., z1 = 0.;  // of layer k+1; z1: what it gives to gz(k+1)
  for (int k = L - 1; k >= 0; --k) {
    const long long ok = o + (long long)k * S;
    PgfPoint l{0., 0., 0., 0.};
    if constexpr (CGRID) {
      l = pgf.layer(k);
    } else {
      l.p0 = lam_u[ok];
      l.z1 = lam_v[ok + S];
    }
    pl = pl + dpl[ok];
    const double pk = CGRID ? pkap[ok] : atm_pow(pl, KAPPA);
    lz += k + 1 < L ? l.z1 + z1 : l.z1;
    const double cpz = CP_DRY * ptl[ok] * lz;
    lam_pt[ok] += CP_DRY * (pk - pk1) * lz;
    if (k + 1 < L) q[k + 1] = ((CGRID ? q1 + l.p1 : q1) + cpz1 - cpz) * KAPPA * pk1 / pl1;
    q1 = l.p0;
    z1 = l.z0;
    cpz1 = cpz;
    pk1 = pk;
    pl1 = pl;
  }
  q[0] = (q1 + cpz1) * KAPPA * pk1 / pl1;
  double acc = 0.;
  for (int k = 0; k < L; ++k) {
    acc += q[k];
    lam_dp[o + (long long)k * S] += acc;
  }
}

// What the D grid's pressure-gradient force passes to pkapb (levels 1..nlay)
// and gzb (levels 2..nlay+1) of the corners [0, n]^2: a thread a corner.
static __global__ void __launch_bounds__(128) k_pgf_adj_corners(Geom g, Consts c, const double* pkb,
                                                                const double* gzb,
                                                                const double* lam_u,
                                                                const double* lam_v,
                                                                double* lam_pkb,
                                                                double* lam_gzb) {
  stream_order();
  const int w = g.nx + 1;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= w * (g.ny + 1)) return;
  const PgfColumn<false> pgf(g, c, pkb, gzb, lam_u, lam_v, idx % w, idx / w);
  // blockIdx.y: a chunk of levels; its lowest level also needs the layer below
  const int k1 = min(g.L, ((int)blockIdx.y + 1) * PGF_CHUNK), k0 = (int)blockIdx.y * PGF_CHUNK;
  PgfPoint lo = k0 > 0 ? pgf.layer(k0 - 1) : PgfPoint{0., 0., 0., 0.};
  for (int k = k0; k < k1; ++k) {
    const PgfPoint l = pgf.layer(k);
    const long long q = pgf.o + (long long)k * g.S;
    lam_pkb[q] = l.p0 + lo.p1;
    lam_gzb[q] = l.z0 + lo.z1;
    lo = l;
  }
  if (k1 == g.L) lam_gzb[pgf.o + (long long)g.L * g.S] = lo.z1;
}

// ==================================================== corners adjoint ====
// Adjoint of interpolate_to_corners (src/mod_sw_dyn.f90:921-956): the 4x4-point
// corner value has weights a(dx) b(dy) + b(dx) a(dy) with a = (-1/12, 7/12, 7/12,
// -1/12) and b = (-1/32, 9/32, 9/32, -1/32) over dx, dy = -2..1.  Gathered over the
// corners [0, nx] x [0, ny] that each point of [-2, nx+1]^2 feeds: pkapb(l) ->
// pkap(l) and gzb(l+1) -> gz(l+1), l < nlay; the results are stored, not added.
// Strips as the forward's (k_corners_m): the two sums along x of a row are formed
// once and kept for four rows; 29 of the 32 columns are outputs.  A thread a point
// gathered 32 values: 0.16 ms at 512x512x32 -> 0.07.
struct CornerAdjLine {
  double a3 = 0, a2 = 0, a1 = 0, a0 = 0, b3 = 0, b2 = 0, b1 = 0, b0 = 0;  // sums along x with a, b, rows j-3 .. j
  __device__ __forceinline__ double push(double q) {  // the gather of row j-2
    a3 = a2; a2 = a1; a1 = a0;
    b3 = b2; b2 = b1; b1 = b0;
    const double n = q + shfl_dn(q, 1), f = shfl_dn(q, 2) + shfl_up(q, 1);
    a0 = C7_12 * n - C1_12 * f;
    b0 = C9_32 * n - C1_32 * f;
    return (C9_32 * (a2 + a1) - C1_32 * (a0 + a3)) + (C7_12 * (b2 + b1) - C1_12 * (b0 + b3));
  }
};
static __global__ void __launch_bounds__(MW * MWARPS, CORN_WARPS_SM / MWARPS) k_corners_adj(
    Geom g, const double* lam_pkb, const double* lam_gzb, double* lam_pk,
    double* lam_gz, int tys) {
  stream_order();
  extern __shared__ __align__(16) char feed_sm[];
  const int lane = threadIdx.x & (MW - 1);
  const int ox = -2 + strip_x() * COUT, oy = -2 + (int)blockIdx.y * tys;
  if (ox > g.nx + 1) return;
  const int x = ox - 1 + lane, yend = min(oy + tys, g.ny + 2);
  const bool out = lane >= 1 && lane < 1 + COUT && x <= g.nx + 1, inx = x >= 0 && x <= g.nx;
  const long long kS = (long long)blockIdx.z * g.S, zS = kS + g.S;
  const unsigned xi = col_of(g, x);
  enum { F_GZ, F_PK };
  FeedRing<2, 0> feed(feed_sm);
  auto copy = [&](int j) {
    const unsigned r = row_of(g, j) + xi;
    feed.early(j, F_GZ, lam_gzb + (zS + r));
    feed.early(j, F_PK, lam_pkb + (kS + r));
  };
  auto none = [](int) {};
  feed.start(copy, none, oy - 1);
  CornerAdjLine lz, lp;
#pragma unroll 4
  for (int j = oy - 1; j < yend + 2; ++j) {
    feed.next(copy, none, j, yend + 2);
    const bool ok = inx && j >= 0 && j <= g.ny;  // a corner
    const double z = lz.push(ok ? feed.get<double>(j, F_GZ) : 0.), p = lp.push(ok ? feed.get<double>(j, F_PK) : 0.);
    if (j >= oy + 2 && out) {
      const unsigned r = row_of(g, j - 2) + xi;
      lam_gz[zS + r] = z;
      lam_pk[kS + r] = p;
    }
  }
}

// ================================================== D-momentum adjoint ====
// Reverse of the D-grid momentum sweep, src/mod_sw_dyn.f90:634-771: ud, vd of
// layer k from the old ud, vd, uc, vc of layers k and nlay (the pressure-
// gradient force apart: k_pgf_adj_corners).
struct DMomAdjArgs {
  const double *ud, *vd, *uc, *vc, *lam_udo, *lam_vdo;
  double *lam_ud, *lam_vd, *lam_uc, *lam_vc;
};

// The x branch: the x fluxes of the vorticity and of the kinetic energy, the
// direct terms and both dampings.
static __global__ void __launch_bounds__(MW * MWARPS, 3) k_d_mom_adj_x(Geom g, Consts c, DMomAdjArgs a, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int ox = strip_x() * MOUT, oy = (int)blockIdx.y * tys;
  if (ox >= g.nx) return;
  const int x = ox - MXH + lane, yend = min(oy + tys, g.ny);
  const bool own = lane >= MXH && lane < MXH + MOUT && x < g.nx, in = x < g.nx + H;
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const unsigned xi = col_of(g, x);
  const double *lam_udo = a.lam_udo + kS, *lam_vdo = a.lam_vdo + kS;
  if (!strip_active(lam_udo, lam_vdo, g, oy, yend, xi, own)) return;
  const double dt = c.dt, dtdx = c.dtdx, dtdy = c.dtdy, rA = c.rA, rdx = c.rdx, rdy = c.rdy, f = c.coriolis;
  const double rdx2 = c.rdx2, rdy2 = c.rdy2, m2rdxy = -2. * c.rdx2rdy2, vdx = c.vdx, vdy = c.vdy;
  const double *ud = a.ud + kS, *vd = a.vd + kS, *uck = a.uc + kS, *uL = a.uc + LS, *vL = a.vc + LS;
  double *lam_ud = a.lam_ud + kS, *lam_vd = a.lam_vd + kS, *lam_uc = a.lam_uc + kS;
  double *lam_uL = a.lam_uc + LS, *lam_vL = a.lam_vc + LS;

  // iteration r brings rows r+2 of ud, r+1 of vd, r of uc and of layer-nlay uc,
  // r+1 of layer-nlay vc, r of lam_udo, lam_vdo
  enum { F_U, F_V, F_UC, F_UN, F_VN, F_LU, F_LV };
  const RowRing<7, 4> ring(adj_sm);
  auto issue = [&](int r) {
    if (r < yend + 6) {
      const unsigned r0 = row_of(g, r) + xi, r1 = row_of(g, r + 1) + xi;
      ring.copy(r, F_U, ud + (row_of(g, r + 2) + xi));
      ring.copy(r, F_V, vd + r1);
      ring.copy(r, F_UN, uL + r0);
      ring.copy(r, F_VN, vL + r1);
      if (r < yend) {
        ring.copy(r, F_UC, uck + r0);
        ring.copy(r, F_LU, lam_udo + r0);
        ring.copy(r, F_LV, lam_vdo + r0);
      }
    }
    ring.commit();
  };
  issue(oy);
  issue(oy + 1);
  auto row = [&](const double* q, int y) { return q[row_of(g, y) + xi]; };
  double um = row(ud, oy - 1), u0 = row(ud, oy), u1 = row(ud, oy + 1);  // rows r-1, r, r+1
  auto vort = [&](double ub, double ut, double v) { return f - (ut - ub) * rdy + (shfl_dn(v, 1) - v) * rdx; };
  double wm = vort(um, u0, row(vd, oy - 1)), w0 = vort(u0, u1, row(vd, oy));  // vorticity of rows r-1, r
  double cum = row(uL, oy - 1), cv0 = row(vL, oy);
  double lu1 = 0, lv1 = 0, lwp = 0, lubp = 0, e1 = 0;       // of row r-1: lam_udo, lam_vdo, den's, half ubL's, ud line's
  double e2 = 0, dir2 = 0, dirv2 = 0, dirv3 = 0;            // ud line's adjoint of row r-2, lam_udo of r-2, lam_vdo of r-2, r-3
  double aW2 = 0, aW1 = 0, aW0 = 0, W3 = 0;                 // adjoints of the vorticity of rows r-2 .. r, and (complete) r-3
  double vw3 = 0;                                           // the vorticity's part of lam_vd of row r-3
  double k1 = 0, k2 = 0;                                    // lke of rows r-1, r-2
  double b1 = 0, b2 = 0;                                    // adjoint of the divergence's Laplacian, rows r-2, r-3
  double g3 = 0;                                            // adjoint of the divergence, row r-3
#pragma unroll 1
  for (int r = oy; r < yend + 6; ++r) {
    issue(r + 2);
    ring.wait();
    const unsigned rr = row_of(g, r) + xi;
    const bool live = r < yend;
    double lu = 0., lv = 0.;
    if (live && own) {
      lu = ring.get(r, F_LU);
      lv = ring.get(r, F_LV);
    }
    const double un = ring.get(r, F_U), cu0 = ring.get(r, F_UN), cv1 = ring.get(r, F_VN);
    const double w1 = vort(u1, un, ring.get(r, F_V));
    double lwv = 0., lcu = 0., aW = 0.;
    if (live && __any_sync(0xffffffffu, lv != 0.)) {
      // v = vd - dt (uc fx + ...), the flux below the cell with the layer-nlay Courant number
      const double uc = ring.get(r, F_UC);
      const bool c0 = dtdx * cv0 > 0., c1 = dtdx * cv1 > 0.;
      const double den = 1. / (1. - dtdy * (cv1 - cv0));
      const double f0 = c0 ? wm : w0, f1 = c1 ? w0 : w1;
      XLineAdj<PPM_CON> ln;
      const double F = ln.forward(inner_e(w0, f0, f1, den, rA), dtdx * cu0);
      double lc = 0.;
      const double lt = ln.reverse(-dt * uc * lv, lc);
      radd(lam_uc, rr, -dt * F * lv, in);
      lcu = dtdx * lc;
      double am, a0, ap, lden = 0.;
      inner_e_adj(w0, f0, f1, c0, c1, den, rA, lt, am, a0, ap, lden);
      lwv = dtdy * den * den * lden;
      aW1 += am;
      aW0 += a0;
      aW = ap;
    }
    // kinetic energy of row r (:639-657) with the layer-nlay B-grid winds (:441-444)
    const double lke = r <= yend ? -dtdx * (up0(lu) - lu) - dtdy * (lv1 - lv) : 0.;
    double e0 = 0., lub = 0.;
    if (r <= yend && __any_sync(0xffffffffu, lke != 0.)) {
      const double ubL = .5 * (cu0 + cum);
      XLineAdj<PPM_CON> ln;
      const double F = ln.forward(u0, dtdx * ubL);
      double lc = 0.;
      e0 = ln.reverse(.5 * ubL * lke, lc);
      lub = .5 * (.5 * F * lke + dtdx * lc);
    }
    radd(lam_uL, row_of(g, r - 1) + xi, lubp + lub, in);  // row r-1: half of ubL of rows r-1 and r
    radd(lam_uL, rr, lcu, in);
    radd(lam_vL, rr, lwp - lwv, in);
    lwp = lwv;
    lubp = lub;
    // damping of the vorticity: adjoint of its Laplacian at row r-1
    {
      const double al = dt * vdy * (lu1 - lu) - dt * vdx * (lv1 - dn0(lv1));
      aW2 += rdy2 * al;
      aW1 += m2rdxy * al + rdx2 * (up0(al) + dn0(al));
      aW0 += rdy2 * al;
    }
    // the vorticity of row r-2 (complete): ud of rows r-2, r-1, vd of row r-2
    const double vw2 = rdx * (up0(aW2) - aW2);
    double su = dir2 + e2 + rdy * (aW2 - W3);
    // damping of the divergence (:682-702): del^4's adjoint is -lke; of del^2 at row r-1, of the divergence at row r-2
    const double b0 = -c.divdamp * (rdy2 * (lke + k2) + (m2rdxy * k1 + rdx2 * (up0(k1) + dn0(k1))));  // row r-1
    const double g2 = rdy2 * (b0 + b2) + (m2rdxy * b1 + rdx2 * (up0(b1) + dn0(b1)));                  // row r-2
    su += rdx * (g2 - dn0(g2));
    radd(lam_ud, row_of(g, r - 2) + xi, su, in);
    radd(lam_vd, row_of(g, r - 3) + xi, dirv3 + vw3 + rdy * (g3 - g2), in);
    k2 = k1; k1 = lke;
    b2 = b1; b1 = b0;
    g3 = g2;
    W3 = aW2;
    vw3 = vw2;
    aW2 = aW1; aW1 = aW0; aW0 = aW;
    e2 = e1; e1 = e0;
    dir2 = lu1;
    dirv3 = dirv2; dirv2 = lv1;
    lu1 = lu;
    lv1 = lv;
    u0 = u1;
    u1 = un;
    wm = w0;
    w0 = w1;
    cum = cu0;
    cv0 = cv1;
  }
}

// The y branch: the y fluxes of the vorticity and of the kinetic energy.  Own
// columns: lanes 1 to 29, over [0, n]^2 (the kinetic energy's range).
constexpr int YOUT_DMOM = 29;
static __global__ void __launch_bounds__(MW * MWARPS, 3) k_d_mom_adj_y(Geom g, Consts c, DMomAdjArgs a, int tys) {
  stream_order();
  extern __shared__ double adj_sm[];
  const int lane = threadIdx.x & (MW - 1), k = blockIdx.z;
  const int ox = strip_x() * YOUT_DMOM, oy = (int)blockIdx.y * tys;
  if (ox > g.nx) return;
  const int x = ox - 1 + lane, yend = min(oy + tys, g.ny + 1);
  const bool own = lane >= 1 && lane <= YOUT_DMOM && x <= g.nx, in = x < g.nx + H;
  const bool dom = x >= 0 && x < g.nx;
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const unsigned xi = col_of(g, x);
  const double *lam_udo = a.lam_udo + kS, *lam_vdo = a.lam_vdo + kS;
  if (!strip_active(lam_udo, lam_vdo, g, max(oy - 1, 0), min(yend, g.ny), xi, dom)) return;
  const double dt = c.dt, dtdx = c.dtdx, dtdy = c.dtdy, rA = c.rA, rdx = c.rdx, rdy = c.rdy, f = c.coriolis;
  const double *ud = a.ud + kS, *vd = a.vd + kS, *vck = a.vc + kS, *uL = a.uc + LS, *vL = a.vc + LS;
  double *lam_ud = a.lam_ud + kS, *lam_vd = a.lam_vd + kS, *lam_vc = a.lam_vc + kS;
  double *lam_uL = a.lam_uc + LS, *lam_vL = a.lam_vc + LS;

  // iteration r brings rows r+1 of ud, r of vd and of layer-nlay uc and, with
  // i = r-2, rows i of lam_udo, lam_vdo, vc and layer-nlay vc, r-5 of layer-nlay uc
  enum { F_U, F_V, F_C, F_LU, F_LV, F_VC, F_CV, F_CS };
  const RowRing<8, 4> ring(adj_sm);
  auto issue = [&](int r) {
    if (r < yend + 8) {
      const int i = r - 2;
      const unsigned r0 = row_of(g, r) + xi, i0 = row_of(g, i) + xi;
      ring.copy(r, F_U, ud + (row_of(g, r + 1) + xi));
      ring.copy(r, F_V, vd + r0);
      ring.copy(r, F_C, uL + r0);
      if (i >= 0 && i < g.ny) {
        ring.copy(r, F_LU, lam_udo + i0);
        ring.copy(r, F_LV, lam_vdo + i0);
      }
      ring.copy(r, F_VC, vck + i0);
      ring.copy(r, F_CV, vL + i0);
      ring.copy(r, F_CS, uL + (row_of(g, r - 5) + xi));
    }
    ring.commit();
  };
  issue(oy - 3);
  issue(oy - 2);
  YLineAdj<PPM_CON> lt, lv_;  // the inner x sweep of the vorticity, vd, along y
  double w1 = 0, w2 = 0, w3 = 0, w4 = 0, w5 = 0;  // vorticity of rows r-1 .. r-5
  double u0 = ud[row_of(g, oy - 3) + xi];
  double lvp = 0, Wp = 0;                         // lam_vdo of row i-1; adjoint of the vorticity of row s-1
#pragma unroll 1
  for (int r = oy - 3; r < yend + 8; ++r) {
    issue(r + 2);
    ring.wait();
    const int i = r - 2, s = r - 5;
    const unsigned ii = row_of(g, i) + xi, si = row_of(g, s) + xi;
    const bool ownr = own && i >= oy && i < yend;
    double lu = 0., lv = 0.;  // lam_udo, lam_vdo of row i over the domain
    if (dom && i >= 0 && i < g.ny) {
      lu = ring.get(r, F_LU);
      lv = ring.get(r, F_LV);
    }
    const double vc = ring.get(r, F_VC), cv = ring.get(r, F_CV), cus = ring.get(r, F_CS);
    // ---- forward: row r
    const double u1 = ring.get(r, F_U), v = ring.get(r, F_V), cu = ring.get(r, F_C);
    const double w = f - (u1 - u0) * rdy + (shfl_dn(v, 1) - v) * rdx;
    u0 = u1;
    {
      const double wl = shfl_up(w, 1), wr = shfl_dn(w, 1), cR = shfl_dn(cu, 1);
      const double den = 1. / (1. - dtdx * (cR - cu));
      lt.push(inner_e(w, dtdx * cu > 0. ? wl : w, dtdx * cR > 0. ? w : wr, den, rA));
    }
    lv_.push(v);
    // ---- interface i: the fluxes and their adjoints
    double lvL;  // of the layer-nlay vc of row i
    double W;    // of the vorticity of row s
    {
      const double luo = ownr ? lu : 0., cy = dtdx * cv;
      const double F = lt.flux(cy);
      double lc = 0.;
      const double lamt = lt.reverse(cy, dt * vc * luo, lc);
      radd(lam_vc, ii, dt * F * luo, in);
      lvL = dtdx * lc;
      // row s: the inner x sweep with the layer-nlay Courant numbers
      const double wl = shfl_up(w5, 1), wr = shfl_dn(w5, 1), cR = shfl_dn(cus, 1);
      const bool c0 = dtdx * cus > 0., c1 = dtdx * cR > 0.;
      const double den = 1. / (1. - dtdx * (cR - cus));
      double am, a0, ap, lden = 0.;
      inner_e_adj(w5, c0 ? wl : w5, c1 ? w5 : wr, c0, c1, den, rA, lamt, am, a0, ap, lden);
      W = a0 + dn0(am) + up0(ap);
      const double lw = dtdx * den * den * lden;
      radd(lam_uL, si, up0(lw) - lw, in);
    }
    w5 = w4; w4 = w3; w3 = w2; w2 = w1; w1 = w;
    {
      const double luL = shfl_up(lu, 1);
      const double lke = ownr ? -dtdx * ((lane > 0 ? luL : 0.) - lu) - dtdy * (lvp - lv) : 0.;
      const double vbL = .5 * (cv + shfl_up(cv, 1));
      const double cy = dtdy * vbL, F = lv_.flux(cy);
      double lc = 0.;
      const double lamv = lv_.reverse(cy, .5 * vbL * lke, lc);
      const double lvb = ownr ? .5 * (.5 * F * lke + dtdy * lc) : 0.;
      radd(lam_vL, ii, lvL + lvb + dn0(lvb), in);
      radd(lam_vd, si, lamv + rdx * (up0(W) - W), in);
      radd(lam_ud, si, rdy * (W - Wp), in);
    }
    Wp = W;
    lvp = lv;
  }
}

}  // namespace atm
