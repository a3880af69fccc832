// Radiation of the reference (src/mod_radiation.f90, src/mod_gas_optics.f90,
// src/mod_solar.f90) on the device, FP64 in both forms:
//   calculate_radiative_heating (:41-156): layer pressures and temperatures
//   of each column, then for each of the 16 g-points a shortwave
//   (solve_shortwave_column, :158-268) and a longwave
//   (solve_longwave_column, :270-347) two-stream solution, both closed by
//   the adding method of calculate_fluxes (:349-381), summed into net_flux.
// Built with --fmad=false and the portable exp/log/pow of atm_math.h:
// every value is the reference's expression in its order, so the results
// are those of the FP64 restatement.  The table searches are binary
// searches for the index the reference's linear scans stop at (the first
// grid point not below the argument), which is the same index.
//
// The reference's asymmetry factor is zero in both solutions and its longwave
// scattering is zero, so the terms they multiply are left out: with
// finite factors each omitted product is an exact zero or one (the shortwave's
// delta-Eddington rescaling changes nothing, the longwave's layers reflect
// nothing and its beta is one), and the remaining operations give the same bits.
#include "atm_math.h"
#include "atm_ops.h"
#include "atm_radiation.h"

namespace atm {
namespace {

// mod_constants.f90:8 -- pi is a default-real literal
constexpr double PI_F = (double)3.1415926535897932384626433f;
// mod_solar.f90:33: 600*(1.+.2/(1.+(radius/100000e3)**2)); .2 and 100000e3
// are default-real literals
constexpr double SOLAR_BASE = 600.;
constexpr double SOLAR_PEAK = (double).2f;
constexpr double SOLAR_SCALE = (double)100000e3f;

// first k with xs[k] >= x for x in [xs[0], xs[n-1]]: where `k = 1; do while
// (x > xs(k)); k = k + 1` stops
__device__ __forceinline__ int first_not_below(const double* __restrict__ xs, int n, double x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (xs[mid] >= x) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// lookup_1d (mod_gas_optics.f90:4556-4579) split in two: the bracket
// (where the reference's scan stops; outside the table the reference stops,
// :4562-4566, and the kernel flags it) and the interpolation at a known
// bracket.  The pressures, temperatures and level temperatures are the
// same for every g-point, so each column finds its brackets once.
__device__ __forceinline__ int bracket(double x, const double* __restrict__ xs, int n, bool& bad) {
  if (x < xs[0] || x > xs[n - 1] || x != x) {
    bad = true;
    return 1;
  }
  return first_not_below(xs, n, x);  // 0 only where x == xs[0], which interp_at returns exactly
}
// lookup_pT_table (mod_gas_optics.f90:4581-4609): the brackets of one layer
// packed as kp | kt1 << 16 | kt2 << 24 (pressure; temperature in rows kp
// and kp - 1; kt2 unused when p is a grid pressure; atm_set_gas_optics
// keeps n_p below 2^16 and n_t below 2^8)
__device__ __forceinline__ unsigned bracket_pt(const RadTables& tb, double p, double t, bool& bad) {
  const int np = tb.np, nt = tb.nt;
  if (p < tb.pressures[0] || p > tb.pressures[np - 1] || p != p) {
    bad = true;
    return 1u | 1u << 16 | 1u << 24;
  }
  const int kp = first_not_below(tb.pressures, np, p);
  const int kt1 = bracket(t, tb.temps + kp * nt, nt, bad);
  const int kt2 = p == tb.pressures[kp] ? 1 : bracket(t, tb.temps + (kp - 1) * nt, nt, bad);
  return (unsigned)kp | (unsigned)kt1 << 16 | (unsigned)kt2 << 24;
}
// The table values of one layer's lookup for one g-point, fetched a layer ahead
// of their use, as most of them come from L2.
struct Lookup {
  double y0, y1, x0, x1;  // row kp: values and temperatures kt1 - 1, kt1
  double v0, v1, z0, z1;  // row kp - 1: kt2 - 1, kt2
  double q0, q1;          // pressures kp - 1, kp
  __device__ __forceinline__ void fetch(const RadTables& tb, const double* __restrict__ table, unsigned code) {
    const int nt = tb.nt, ng = tb.ng, kp = code & 0xffff, k1 = (code >> 16) & 0xff, k2 = code >> 24;
    const int r1 = kp * nt, r2 = max(kp - 1, 0) * nt;
    const int a1 = r1 + k1, a0 = r1 + max(k1 - 1, 0), b1 = r2 + k2, b0 = r2 + max(k2 - 1, 0);
    y0 = __ldg(table + (long long)a0 * ng);
    y1 = __ldg(table + (long long)a1 * ng);
    v0 = __ldg(table + (long long)b0 * ng);
    v1 = __ldg(table + (long long)b1 * ng);
    x0 = __ldg(tb.temps + a0);
    x1 = __ldg(tb.temps + a1);
    z0 = __ldg(tb.temps + b0);
    z1 = __ldg(tb.temps + b1);
    q0 = __ldg(tb.pressures + max(kp - 1, 0));
    q1 = __ldg(tb.pressures + kp);
  }
  __device__ __forceinline__ double at(double p, double t) const {
    const double t1 = t == x1 ? y1 : (y1 * (x0 - t) + y0 * (t - x1)) / (x0 - x1);
    if (p == q1) return t1;
    const double t2 = t == z1 ? v1 : (v1 * (z0 - t) + v0 * (t - z1)) / (z0 - z1);
    return (t1 * (q0 - p) + t2 * (p - q1)) / (q0 - q1);
  }
};
// ... and of a lookup in the Planck table
struct PlanckLookup {
  double y0, y1, x0, x1;
  __device__ __forceinline__ void fetch(const RadTables& tb, const double* __restrict__ plk, int k) {
    const int k0 = max(k - 1, 0);
    y0 = __ldg(plk + (long long)k0 * tb.ng);
    y1 = __ldg(plk + (long long)k * tb.ng);
    x0 = __ldg(tb.plk_t + k0);
    x1 = __ldg(tb.plk_t + k);
  }
  __device__ __forceinline__ double at(double t) const {
    return t == x1 ? y1 : (y1 * (x0 - t) + y0 * (t - x1)) / (x0 - x1);
  }
};

// A block's columns: RC of them, 16 lanes each (a lane a g-point, in rounds of
// 16), so that a small domain fills the GPU and a column's layer properties,
// in shared memory, serve all its g-points.  What a lane keeps per layer for
// the adding method's sweeps (seven arrays) stays in local memory and mostly in
// DRAM (3.7 KB a lane at 64 layers), and the tables in L2: four blocks an SM wait
// on these loads, so each is issued ahead of its use.  Measured on B200 (ms;
// before: a thread a column, its g-points in turn): 64x64x20 1.65 -> 0.11,
// 192x160x48 6.77 -> 1.69, 512x512x64 23.7 -> 18.2, 1024x1024x64 87.9 -> 71.9
// (113 without the loads ahead).
constexpr int RG = 16, RC = 8;
constexpr int RP = 2;  // levels of the working arrays loaded ahead in the sweeps (1, 3 and 4: 91.9, 81.1 and 91.7 ms below)
constexpr int RB = 8;  // levels whose fluxes are gathered before they are summed over the g-points

// shared memory of one column, levels 1-based as in the reference
struct RadColumn {
  double *play, *tlay, *dm, *tlev, *sum[4], *buf;  // sum: upward and downward shortwave, longwave
  unsigned* code;
  int* kb;
};
__host__ __device__ inline int rad_doubles(int L) { return 8 * (L + 2) + 2 * RB * (RG + 1) + (L + 2); }

// The ordered sums over the g-points of one solution: the lanes of a column
// leave the fluxes of RB levels in buf, then each adds one level's, upward or
// downward, to the column's sum in the reference's order.
struct RadSums {
  const RadColumn& c;
  int which, lane, n;  // 0 shortwave, 2 longwave; lanes taking part in this round
  __device__ __forceinline__ void put(int L, int k, double fu, double fd) {
    const int slot = (L + 1 - k) % RB;
    c.buf[slot * (RG + 1) + lane] = fu;
    c.buf[(RB + slot) * (RG + 1) + lane] = fd;
    if (slot == RB - 1 || k == 1) {
      __syncwarp();
      const int level = k + slot - (lane % RB);
      if (level >= k) {
        double* s = c.sum[which + lane / RB] + level;
        const double* f = c.buf + lane * (RG + 1);
        double t = *s;
        for (int g = 0; g < n; ++g) t = t + f[g];
        *s = t;
      }
      __syncwarp();
    }
  }
};

// The layer properties and flux sums of a column that one thread has to itself
// (k_radiation_columns), and how its fluxes are added to them.
template <int LM>
struct OwnColumn {
  double play[LM + 1], tlay[LM + 1], dm[LM + 1], tlev[LM + 2], sum[4][LM + 2];
  unsigned code[LM + 1];
  int kb[LM + 2];
};
template <int LM>
struct OwnSums {
  OwnColumn<LM>& c;
  int which;
  __device__ __forceinline__ void put(int, int k, double fu, double fd) {
    c.sum[which][k] = c.sum[which][k] + fu;
    c.sum[which + 1][k] = c.sum[which + 1][k] + fd;
  }
};

// Per-lane working arrays of one g-point (1-based as in the reference).
template <int LM>
struct LayerArrays {
  double R[LM + 1], T[LM + 1], su[LM + 1], sd[LM + 1];  // reflectance (later times em), transmittance, sources (su later beta)
  double alb[LM + 2], em[LM + 2], beam[LM + 2];         // calculate_fluxes' albedo, emission_up; solar_beam
};

// solve_shortwave_column (mod_radiation.f90:158-268) for g-point g: the layer
// coefficients top-down (the direct beam is attenuated layer by layer), then
// calculate_fluxes (:349-381); the beam is added to the downward flux.
template <int LM, typename Col, typename Out>
__device__ __forceinline__ void shortwave(const RadTables& tb, int g, int L, const Col& col, double irradiance,
                                          double mu0, double sfc_albedo, LayerArrays<LM>& c, Out& out) {
  const double* tab = tb.sw_abs + g;
  const double k_sca = tb.sw_sca[g];
  double beam = mu0 * irradiance;
  c.beam[L + 1] = beam;
  Lookup nx;
  nx.fetch(tb, tab, col.code[L]);
  for (int k = L; k >= 1; --k) {
    const double k_abs = nx.at(col.play[k], col.tlay[k]);
    if (k > 1) nx.fetch(tb, tab, col.code[k - 1]);
    const double k_ext = k_abs + k_sca;
    const double tau = k_ext * col.dm[k];
    const double ssa = k_sca / k_ext;
    // direct to diffuse: hybrid modified Eddington-delta (Meador & Weaver 1980)
    double gamma1 = (7. - ssa * 4.) / 4.;
    double gamma2 = (-1. + ssa * 4.) / 4.;
    const double alpha1 = gamma1 * .5 + gamma2 * .5;
    const double alpha2 = gamma2 * .5 + gamma2 * .5;
    double lambda = sqrt(gamma1 * gamma1 - gamma2 * gamma2);
    const double lam_mu = lambda * mu0;
    const double e_minus = atm_exp(-(lambda * tau));
    const double e_2minus = e_minus * e_minus;
    const double direct_t = atm_exp(-(tau / mu0));
    double tmp1 = ssa / ((1. - lam_mu * lam_mu) * (lambda + gamma1 + (lambda - gamma1) * e_2minus));
    const double tmp2 = lambda * .5;
    const double diffuse_r = tmp1 * ((1. - lam_mu) * (alpha2 + tmp2) - (1. + lam_mu) * (alpha2 - tmp2) * e_2minus -
                                     2. * lambda * (.5 - alpha2 * mu0) * e_minus * direct_t);
    const double diffuse_t = tmp1 * (2. * lambda * (.5 + alpha1 * mu0) * e_minus -
                                     direct_t * ((1. + lam_mu) * (alpha1 + tmp2) - (1. - lam_mu) * (alpha1 - tmp2) * e_2minus));
    c.su[k] = diffuse_r * beam;
    c.sd[k] = diffuse_t * beam;
    beam = direct_t * beam;
    c.beam[k] = beam;
    // diffuse to diffuse: hemispheric constant (Meador & Weaver 1980) with
    // the backscatter of Ritter & Geleyn (1992); e_minus is the one above
    gamma1 = 2. * (1. - ssa * .5);
    gamma2 = ssa;
    lambda = sqrt(gamma1 * gamma1 - gamma2 * gamma2);
    tmp1 = 1. / (lambda + gamma1 + (lambda - gamma1) * e_2minus);
    c.R[k] = tmp1 * gamma2 * (1. - e_2minus);
    c.T[k] = 2. * tmp1 * lambda * e_minus;
  }
  double alb = sfc_albedo, em = 0.;
  c.alb[1] = alb;
  c.em[1] = em;
  {  // :357-363
    double Rn[RP], Tn[RP], un[RP], dn[RP];
    auto fetch = [&](int q, int k) {
      Rn[q] = c.R[k];
      Tn[q] = c.T[k];
      un[q] = c.su[k];
      dn[q] = c.sd[k];
    };
#pragma unroll
    for (int q = 0; q < RP; ++q)
      if (1 + q <= L) fetch(q, 1 + q);
    for (int k0 = 1; k0 <= L; k0 += RP) {
#pragma unroll
      for (int q = 0; q < RP; ++q) {
        const int k = k0 + q;
        if (k > L) break;
        const double R = Rn[q], T = Tn[q], su = un[q], sd = dn[q];
        if (k + RP <= L) fetch(q, k + RP);
        const double beta = 1. / (1. - R * alb);
        const double alb1 = R + (T * T) * beta * alb;
        const double em1 = su + T * beta * (em + sd * alb);
        c.R[k] = R * em;
        c.su[k] = beta;
        c.alb[k + 1] = alb1;
        c.em[k + 1] = em1;
        alb = alb1;
        em = em1;
      }
    }
  }
  double fdn = c.beam[L + 1];  // :365-380
  out.put(L, L + 1, alb * fdn + em, fdn + fdn);
  {
    double bn[RP], dn[RP], Tn[RP], rn[RP], an[RP], en[RP], mn_[RP];
    auto fetch = [&](int q, int k) {
      bn[q] = c.su[k];
      dn[q] = c.sd[k];
      Tn[q] = c.T[k];
      rn[q] = c.R[k];
      an[q] = c.alb[k];
      en[q] = c.em[k];
      mn_[q] = c.beam[k];
    };
#pragma unroll
    for (int q = 0; q < RP; ++q)
      if (L - q >= 1) fetch(q, L - q);
    for (int k0 = L; k0 >= 1; k0 -= RP) {
#pragma unroll
      for (int q = 0; q < RP; ++q) {
        const int k = k0 - q;
        if (k < 1) break;
        fdn = bn[q] * (dn[q] + Tn[q] * fdn + rn[q]);
        const double fu = an[q] * fdn + en[q], fd = fdn + mn_[q];
        if (k - RP >= 1) fetch(q, k - RP);
        out.put(L, k, fu, fd);
      }
    }
  }
}

// solve_longwave_column (mod_radiation.f90:270-347) for g-point g: no
// scattering, a Planck source linear in optical depth; the upward sweep of
// calculate_fluxes inside its layer loop (both go upward)
template <int LM, typename Col, typename Out>
__device__ __forceinline__ void longwave(const RadTables& tb, int g, int L, const Col& col, double ts, int kbs,
                                         double emissivity, LayerArrays<LM>& c, Out& out) {
  const double* tab = tb.lw_abs + g;
  const double* plk = tb.plk + g;
  Lookup nx;
  nx.fetch(tb, tab, col.code[1]);
  PlanckLookup pn;
  pn.fetch(tb, plk, kbs);
  const double surface_planckian = pn.at(ts);
  pn.fetch(tb, plk, col.kb[1]);
  double lp_k = pn.at(col.tlev[1]);
  pn.fetch(tb, plk, col.kb[2]);
  double alb = 1. - emissivity, em = emissivity * PI_F * surface_planckian;  // calculate_fluxes' arguments (:345)
  c.alb[1] = alb;
  c.em[1] = em;
  for (int k = 1; k <= L; ++k) {
    const double tau = nx.at(col.play[k], col.tlay[k]) * col.dm[k];
    const double lp_k1 = pn.at(col.tlev[k + 1]);
    if (k < L) {
      nx.fetch(tb, tab, col.code[k + 1]);
      pn.fetch(tb, plk, col.kb[k + 2]);
    }
    const double T = atm_exp(-(2. * tau));
    const double pdiff = (1. - T) * (lp_k - lp_k1) / (tau * 2.);
    const double su = PI_F * (lp_k1 - T * lp_k + pdiff);
    const double sd = PI_F * (lp_k - T * lp_k1 - pdiff);
    c.T[k] = T;
    c.sd[k] = sd;
    lp_k = lp_k1;
    const double em1 = su + T * (em + sd * alb);
    alb = (T * T) * alb;
    em = em1;
    c.alb[k + 1] = alb;
    c.em[k + 1] = em;
  }
  double fdn = 0.;
  out.put(L, L + 1, alb * fdn + em, fdn);
  double dn[RP], Tn[RP], an[RP], en[RP];
  auto fetch = [&](int q, int k) {
    dn[q] = c.sd[k];
    Tn[q] = c.T[k];
    an[q] = c.alb[k];
    en[q] = c.em[k];
  };
#pragma unroll
  for (int q = 0; q < RP; ++q)
    if (L - q >= 1) fetch(q, L - q);
  for (int k0 = L; k0 >= 1; k0 -= RP) {
#pragma unroll
    for (int q = 0; q < RP; ++q) {
      const int k = k0 - q;
      if (k < 1) break;
      fdn = dn[q] + Tn[q] * fdn;
      const double fu = an[q] * fdn + en[q];
      if (k - RP >= 1) fetch(q, k - RP);
      out.put(L, k, fu, fdn);
    }
  }
}

// The layer pressures and temperatures (mod_radiation.f90:54-103), a lane a
// level, then for each g-point, a lane each, the shortwave and longwave fluxes,
// added in the order g = 1, 2, ... into the four sums the reference keeps
// (:113-147), and net_flux = (down sw + down lw) - (up sw + up lw) (:149-152).
// The reference also overwrites plev, pkap, play and playkap of the shared
// fields here; every later reader recomputes them first, so they stay
// local.  Its domain is the interior plus 3 halo cells, whose values the
// halo exchange that follows replaces: the interior is computed here and
// atm_radiation_halo fills the halo.
template <int LM>
__global__ void __launch_bounds__(RG * RC, 4) k_radiation(Geom g, RadTables tb, RadArgs a) {
  extern __shared__ double rad_sm[];
  const int L = g.L, lane = threadIdx.x % RG, c0 = threadIdx.x / RG;
  const int col = blockIdx.x * RC + c0;
  const bool in = col < g.nx * g.ny;
  const int cc = in ? col : 0;
  const long long S = g.S, o = g.at(cc % g.nx, cc / g.nx);
  const unsigned group = 0xffffu << (threadIdx.x & 16);
  RadColumn c;
  double* q = rad_sm + (long long)c0 * rad_doubles(L);
  c.play = q;
  c.tlay = q += L + 2;
  c.dm = q += L + 2;
  c.tlev = q += L + 2;
  for (int i = 0; i < 4; ++i) c.sum[i] = q += L + 2;
  c.buf = q += L + 2;
  c.code = reinterpret_cast<unsigned*>(q + 2 * RB * (RG + 1));
  c.kb = reinterpret_cast<int*>(c.code + (L + 2));
  double *plev = c.sum[0], *pkap = c.sum[1];  // until the sums start
  {
    double p = a.ptop;  // the order of this sum fixes its bits: every lane forms it
    if (lane == 0) plev[L + 1] = p;
    for (int k = L; k >= 1; --k) {
      p = p + a.dp[o + (long long)(k - 1) * S];
      if (lane == 0) plev[k] = p;
    }
  }
  __syncwarp();
  for (int k = 1 + lane; k <= L + 1; k += RG) pkap[k] = k <= L ? atm_pow(plev[k], KAPPA) : a.pk_top;
  __syncwarp();
  for (int k = 1 + lane; k <= L; k += RG) {  // :54-84
    const double dpk = a.dp[o + (long long)(k - 1) * S];
    const double plog = atm_log(plev[k] / plev[k + 1]);
    c.play[k] = dpk / plog;
    const double playkap = (pkap[k + 1] - pkap[k]) / (-(plog * KAPPA));
    c.tlay[k] = a.pt[o + (long long)(k - 1) * S] * playkap;
    c.dm[k] = dpk / a.gravity;  // :118
  }
  __syncwarp();
  bool bad = false;
  for (int k = 1 + lane; k <= L + 1; k += RG) {
    // interpolation of T linear in log p; extrapolation to the bottom
    // (:95-102) and the model top (:86-93)
    const int m = k == 1 ? 1 : (k == L + 1 ? L - 1 : k - 1);
    const double p1 = atm_log(c.play[m]), p2 = atm_log(c.play[m + 1]), plog = atm_log(k == L + 1 ? a.ptop : plev[k]);
    const double t = (c.tlay[m] * (p2 - plog) + c.tlay[m + 1] * (plog - p1)) / (p2 - p1);
    c.tlev[k] = t;
    // the table brackets of every layer and level, shared by the g-points
    c.kb[k] = bracket(t, tb.plk_t, tb.npl, bad);
    if (k <= L) c.code[k] = bracket_pt(tb, c.play[k], c.tlay[k], bad);
  }
  const double ts = a.ts[o];
  const int kbs = bracket(ts, tb.plk_t, tb.npl, bad);
  bad = (__ballot_sync(0xffffffffu, bad) & group) != 0;
  for (int k = 1 + lane; k <= L + 1; k += RG)
    for (int i = 0; i < 4; ++i) c.sum[i][k] = 0.;  // :112-116
  __syncwarp();
  // solar_irradiance (mod_solar.f90:26-35)
  const double r = a.radius[cc] / SOLAR_SCALE;
  const double irradiance = SOLAR_BASE * (1. + SOLAR_PEAK / (1. + r * r));
  LayerArrays<LM> w;
  for (int g0 = 0; g0 < tb.ng; g0 += RG) {
    const int n = min(RG, tb.ng - g0), gp = g0 + min(lane, n - 1);
    RadSums sw{c, 0, lane, n}, lw{c, 2, lane, n};
    shortwave<LM>(tb, gp, L, c, tb.frac[gp] * irradiance, a.mu0, a.albedo, w, sw);
    longwave<LM>(tb, gp, L, c, ts, kbs, a.emissivity, w, lw);
  }
  if (in) {
    for (int k = 1 + lane; k <= L + 1; k += RG)
      a.nf[o + (long long)(k - 1) * S] = bad ? 0. : (c.sum[1][k] + c.sum[3][k]) - (c.sum[0][k] + c.sum[2][k]);
    if (bad && lane == 0) atomicOr(a.range_error, 1);
  }
}

// The same with a thread a column, its g-points in turn and its arrays in local
// memory: for tables of few g-points, whose other lanes k_radiation leaves idle,
// and for few layers, whose work is little beside what a block sets up.  BLOCKS an
// SM: 8 (64 registers) hide more of the local memory's latency where that many
// columns come, 4 take fewer instructions (us at 4 / 6 / 8: 3 g-points 40 layers
// 65536 columns 1081 / 1218 / 1265, 64 layers 262144 6633 / 6078 / 5057, 6 layers
// 262144 422 / 470 / 474).
template <int LM, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_radiation_columns(Geom g, RadTables tb, RadArgs a) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.nx * g.ny) return;
  const int L = g.L;
  const long long S = g.S, o = g.at(col % g.nx, col / g.nx);
  OwnColumn<LM> c;
  bool bad = false;
  {
    double pu = a.ptop, pku = a.pk_top, lu = atm_log(a.ptop);  // level k + 1: pressure, pkap, log p
    double lp2 = 0.;                                           // log play(k + 1)
    auto level = [&bad, &tb](OwnColumn<LM>& c, int k, int m, double lm, double lm1, double lk) {
      const double t = (c.tlay[m] * (lm1 - lk) + c.tlay[m + 1] * (lk - lm)) / (lm1 - lm);
      c.tlev[k] = t;
      c.kb[k] = bracket(t, tb.plk_t, tb.npl, bad);
    };
    const double ltop = lu;
    for (int k = L; k >= 1; --k) {  // :54-84
      const double dpk = a.dp[o + (long long)(k - 1) * S];
      const double p = pu + dpk, pk = atm_pow(p, KAPPA), plog = atm_log(p / pu);
      c.play[k] = dpk / plog;
      c.tlay[k] = a.pt[o + (long long)(k - 1) * S] * ((pku - pk) / (-(plog * KAPPA)));
      c.dm[k] = dpk / a.gravity;  // :118
      c.code[k] = bracket_pt(tb, c.play[k], c.tlay[k], bad);
      const double lp1 = atm_log(c.play[k]);
      // the level above, between layers k and k + 1; the model top extrapolated (:86-93)
      if (k < L) level(c, k + 1, k, lp1, lp2, lu);
      if (k == L - 1) level(c, L + 1, L - 1, lp1, lp2, ltop);
      pu = p;
      pku = pk;
      lu = atm_log(p);
      if (k == 1) level(c, 1, 1, lp1, lp2, lu);  // the bottom extrapolated (:95-102)
      lp2 = lp1;
    }
  }
  const double ts = a.ts[o];
  const int kbs = bracket(ts, tb.plk_t, tb.npl, bad);
  for (int k = 1; k <= L + 1; ++k)
    for (int i = 0; i < 4; ++i) c.sum[i][k] = 0.;  // :112-116
  // solar_irradiance (mod_solar.f90:26-35)
  const double r = a.radius[col] / SOLAR_SCALE;
  const double irradiance = SOLAR_BASE * (1. + SOLAR_PEAK / (1. + r * r));
  LayerArrays<LM> w;
  OwnSums<LM> sw{c, 0}, lw{c, 2};
  if (!bad)
    for (int gp = 0; gp < tb.ng; ++gp) {
      shortwave<LM>(tb, gp, L, c, tb.frac[gp] * irradiance, a.mu0, a.albedo, w, sw);
      longwave<LM>(tb, gp, L, c, ts, kbs, a.emissivity, w, lw);
    }
  for (int k = 1; k <= L + 1; ++k)
    a.nf[o + (long long)(k - 1) * S] = (c.sum[1][k] + c.sum[3][k]) - (c.sum[0][k] + c.sum[2][k]);
  if (bad) atomicOr(a.range_error, 1);
}

// Whether n columns take a thread each.  Both forms' times grow with the columns, the
// lanes' with the rounds of RG g-points, the threads' with the g-points and, for
// latency, less than in proportion below 112000 columns; a column's round costs about 11
// times a column's g-point in turn, more with many layers (fewer blocks an SM) and with
// very few.  Measured on B200 (us, a lane a g-point / a thread a column):
// 20 layers, 16384 columns 1 g-point 357/160, 3 358/323, 6 360/547; 262144 6 4911/2887, 10 4936/4582, 14 4965/6284;
// 64 layers, 4096 1 361/430; 36000 3 2689/1515, 6 2698/2746; 262144 10 18175/14698, 14 18359/20239, 20 33584/28461, 40 49700/59697;
// 128 layers, 160000 14 37249/33388, 16 37277/38637; 3 layers, 65536 16 308/219, 1048576 16 4840/2808.
inline bool rad_columns(long long n, int L, int ng) {
  const double round = L > 64 ? 15. : L > 32 ? 12. : 10.5 + 170. / (L * L);
  const double cols = n > 112500 ? (double)n : 45000. + .6 * (double)n;
  return (ng + 1.) * cols < round * ((ng + RG - 1) / RG) * (double)n;
}

template <int LM>
cudaError_t launch(const Geom& g, const RadTables& t, const RadArgs& a, cudaStream_t s) {
  const int n = g.nx * g.ny;
  if (rad_columns(n, g.L, t.ng)) {
    if (n > 148 * 1024 && g.L > 8) k_radiation_columns<LM, 8><<<(n + 127) / 128, 128, 0, s>>>(g, t, a);
    else k_radiation_columns<LM, 4><<<(n + 127) / 128, 128, 0, s>>>(g, t, a);
    return cudaGetLastError();
  }
  const size_t sm = (size_t)RC * rad_doubles(g.L) * sizeof(double);
  // what LM layers take whatever L is: launches on several threads set the same value
  const cudaError_t e = cudaFuncSetAttribute(k_radiation<LM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(RC * rad_doubles(LM) * sizeof(double)));
  if (e != cudaSuccess) return e;
  k_radiation<LM><<<(n + RC - 1) / RC, RG * RC, sm, s>>>(g, t, a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t radiative_heating(const Geom& g, const RadTables& t, const RadArgs& a, cudaStream_t s) {
  if (g.L <= 32) return launch<32>(g, t, a, s);
  if (g.L <= 64) return launch<64>(g, t, a, s);
  return launch<MAX_LAYERS>(g, t, a, s);
}

}  // namespace atm
