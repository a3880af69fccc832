// Adjoint kernels of the FP64 dynamical core next to the sweeps (which are
// reversed in atm_adj_march.cuh): corner interpolation, halos and the vertical
// remap.  Each recomputes what it needs of the forward with the forward's
// operations, hence takes the same branches; adjoints are accumulated with +=
// or atomics where several points feed one input.
#pragma once

#include "atm_kernels.cuh"

namespace atm {

// index (0, 1, 2) of the argument that mn3 / mx3 return
__device__ __forceinline__ int sel_mn3(double a, double b, double c) {
  int i = (b < a) ? 1 : 0;
  double t = (b < a) ? b : a;
  return (c < t) ? 2 : i;
}
__device__ __forceinline__ int sel_mx3(double a, double b, double c) {
  int i = (a < b) ? 1 : 0;
  double t = (a < b) ? b : a;
  return (t < c) ? 2 : i;
}

// ======================================================= halo adjoints ====
// Adjoint of the periodic ring fill (k_ring, copy = false): every ring
// point's adjoint is added to its periodic image in the interior and
// cleared.
__global__ void k_ring_fold(Geom g, double* f0, double* f1, double* f2, double* f3, int K) {
  stream_order();
  const int wide = g.nx + 2 * H;
  const int nband = 2 * H * wide;
  const int nring = nband + 2 * H * g.ny;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nring || (int)blockIdx.y >= K) return;
  int x, y;
  if (idx < nband) {
    int r = idx / wide;
    y = r < H ? r - H : g.ny + (r - H);
    x = idx % wide - H;
  } else {
    int q = idx - nband;
    y = q / (2 * H);
    int cc = q % (2 * H);
    x = cc < H ? cc - H : g.nx + (cc - H);
  }
  const int fld = blockIdx.z;
  double* f = fld == 0 ? f0 : fld == 1 ? f1 : fld == 2 ? f2 : f3;
  if (!f) return;
  const int k = blockIdx.y;
  const long long o = g.at(x, y, k);
  const double v = f[o];
  if (v == 0.) return;
  const int xs = x < 0 ? x + g.nx : (x >= g.nx ? x - g.nx : x);
  const int ys = y < 0 ? y + g.ny : (y >= g.ny ? y - g.ny : y);
  atomicAdd(f + g.at(xs, ys, k), v);
  f[o] = 0.;
}

// Adjoint of the ring copy old -> new time level (k_ring, copy = true)
// for the ring points that the following step did not overwrite: points
// of fields 0, 1 inside [-band01, n+band01)^2 and of fields 2, 3 inside
// [-band23, n+band23)^2 were recomputed and keep their adjoint.
__global__ void k_ring_copy_adj(Geom g, double* d0, double* d1, double* d2, double* d3, double* s0, double* s1,
                                double* s2, double* s3, int K, int band01, int band23) {
  stream_order();
  const int wide = g.nx + 2 * H;
  const int nband = 2 * H * wide;
  const int nring = nband + 2 * H * g.ny;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nring || (int)blockIdx.y >= K) return;
  int x, y;
  if (idx < nband) {
    int r = idx / wide;
    y = r < H ? r - H : g.ny + (r - H);
    x = idx % wide - H;
  } else {
    int q = idx - nband;
    y = q / (2 * H);
    int cc = q % (2 * H);
    x = cc < H ? cc - H : g.nx + (cc - H);
  }
  const int fld = blockIdx.z;
  const int band = fld < 2 ? band01 : band23;
  if (x >= -band && x < g.nx + band && y >= -band && y < g.ny + band) return;
  double* d = fld == 0 ? d0 : fld == 1 ? d1 : fld == 2 ? d2 : d3;
  double* s = fld == 0 ? s0 : fld == 1 ? s1 : fld == 2 ? s2 : s3;
  const long long o = g.at(x, y, blockIdx.y);
  s[o] += d[o];
  d[o] = 0.;
}

// ======================================================= remap adjoint ====
// Reverse mode of remap_column (src/mod_remap.f90:165-356): the forward
// vertical_ppm is recomputed with its intermediates kept (solve, back
// substitution, limited interface values), the same layer pairs are
// visited, and the adjoints flow back to the source values and to both
// coordinates.
// The column arrays of the adjoint of vertical_ppm: the forward's lvs (after
// the elimination), lvb (after the back substitution), lvc (limited) and
// gam, and the adjoints.  The monotone path forms each layer's edges and
// curvature on the fly (PPMLayers); RemapAdjFull also stores them, for the
// all-pairs path of non-monotone coordinates.
template <int LM>
struct RemapAdjWork {
  double gam[LM + 2], lvs[LM + 2], lvb[LM + 2], lvc[LM + 2];
  double LL[LM + 2], Lgam[LM + 2], Ltop[LM + 2], Lbtm[LM + 2];
};
template <int LM>
struct RemapAdjFull : RemapAdjWork<LM> {
  double top[LM + 2], btm[LM + 2], curv[LM + 2];
};

// vertical_ppm (src/mod_remap.f90:287-356) keeping lvs, lvb, lvc, the
// edges and the curvature; the operations are those of vertical_ppm in
// atm_kernels.cuh.
template <int LM>
__device__ void vppm_record(RemapAdjFull<LM>& w, int L, const double* var, const double* coord) {
  double* gam = w.gam;
  double* lv = w.lvs;
  double alpha, beta;
  alpha = (coord[L] - coord[L - 1]) / (coord[L + 1] - coord[L]);
  beta = alpha * (.5 + alpha);
  lv[L + 1] = (2. * alpha * (1. + alpha) * var[L] + var[L - 1]) / beta;
  gam[L] = (1. + alpha * (1.5 + alpha)) / beta;
  for (int k = L; k >= 2; --k) {
    alpha = (coord[k + 1] - coord[k]) / (coord[k] - coord[k - 1]);
    beta = 2. + 2. * alpha - gam[k];
    lv[k] = (3. * (var[k] + alpha * var[k - 1]) - lv[k + 1]) / beta;
    gam[k - 1] = alpha / beta;
  }
  beta = 1. + alpha * (1.5 + alpha);
  lv[1] = (2. * alpha * (1. + alpha) * var[1] + var[2] - beta * lv[2]) / (alpha * (.5 + alpha) - beta * gam[1]);
  double* b = w.lvb;
  b[1] = lv[1];
  for (int k = 2; k <= L + 1; ++k) b[k] = lv[k] - gam[k - 1] * b[k - 1];
  double* c = w.lvc;
  for (int k = 1; k <= L + 1; ++k) c[k] = b[k];
  c[L] = mn(c[L], mx(var[L], var[L - 1]));
  c[L] = mx(c[L], mn(var[L], var[L - 1]));
  c[2] = mn(c[2], mx(var[2], var[1]));
  c[2] = mx(c[2], mn(var[2], var[1]));
  for (int k = 2; k <= L - 1; ++k) {
    double lo = mn(var[k], var[k + 1]), hi = mx(var[k], var[k + 1]);
    if (k + 2 > L || gam[k + 2] * gam[k] > 0) {
      c[k + 1] = mn(c[k + 1], hi);
      c[k + 1] = mx(c[k + 1], lo);
    } else if (gam[k + 2] > 0) {
      c[k + 1] = mx(c[k + 1], lo);
    } else {
      c[k + 1] = mn(c[k + 1], hi);
    }
  }
  for (int k = 1; k <= L; ++k) {
    w.top[k] = c[k + 1];
    w.btm[k] = c[k];
  }
  for (int k = 2; k <= L - 1; ++k) {
    double pmp1 = var[k + 1] - 2. * gam[k];
    double lac1 = pmp1 + 1.5 * gam[k - 1];
    w.top[k + 1] = mn(mx(w.top[k + 1], mn3(var[k + 1], pmp1, lac1)), mx3(var[k + 1], pmp1, lac1));
    pmp1 = var[k + 1] + 2. * gam[k + 1];
    lac1 = pmp1 - 1.5 * gam[k];
    w.btm[k + 1] = mn(mx(w.btm[k + 1], mn3(var[k + 1], pmp1, lac1)), mx3(var[k + 1], pmp1, lac1));
  }
  for (int k = 1; k <= L; ++k) w.curv[k] = 6. * var[k] - 3. * (w.top[k] + w.btm[k]);
}

// adjoint of r = mn(mx(x0, mn3(a, b, c)), mx3(a, b, c)) for the edge limiter
// of src/mod_remap.f90:342-352 with a = var, b = var + s2 * gam(j2),
// c = b + s15 * gam(j15): returns the adjoint of x0.
__device__ __forceinline__ double edge_clamp_adj(double x0, double a, double b, double c, double lam, double& lvar,
                                                 double* Lgam, int j2, double s2, int j15, double s15) {
  const double lo = mn3(a, b, c), hi = mx3(a, b, c);
  const double inner = mx(x0, lo);
  int which;  // 0: x0, 1: lo, 2: hi
  if (hi < inner) which = 2;
  else if (x0 < lo) which = 1;
  else which = 0;
  if (which == 0) return lam;
  const int s = which == 1 ? sel_mn3(a, b, c) : sel_mx3(a, b, c);
  if (s == 0) {
    lvar += lam;
  } else {
    lvar += lam;
    Lgam[j2] += s2 * lam;
    if (s == 2) Lgam[j15] += s15 * lam;
  }
  return 0.;
}

// Adjoint of vertical_ppm given w.Ltop, w.Lbtm (curvature already folded
// into them and into Lvar): adds to Lvar (source values) and Lc (coordinate).
template <int LM>
__device__ void vppm_adj(RemapAdjWork<LM>& w, int L, const double* var, const double* coord, double* Lvar, double* Lc) {
  const double* gam = w.gam;
  double* LL = w.LL;
  double* Lgam = w.Lgam;
  for (int k = 0; k <= L + 1; ++k) {
    LL[k] = 0.;
    Lgam[k] = 0.;
  }
  // edge limiters of top/btm (:340-352), reverse order
  for (int k = L - 1; k >= 2; --k) {
    double lt = w.Ltop[k + 1];
    if (lt != 0.) {
      const double pmp1 = var[k + 1] - 2. * gam[k];
      const double lac1 = pmp1 + 1.5 * gam[k - 1];
      lt = edge_clamp_adj(w.lvc[k + 2], var[k + 1], pmp1, lac1, lt, Lvar[k + 1], Lgam, k, -2., k - 1, 1.5);
    }
    double lb = w.Lbtm[k + 1];
    if (lb != 0.) {
      const double pmp1 = var[k + 1] + 2. * gam[k + 1];
      const double lac1 = pmp1 - 1.5 * gam[k];
      lb = edge_clamp_adj(w.lvc[k + 1], var[k + 1], pmp1, lac1, lb, Lvar[k + 1], Lgam, k + 1, 2., k, -1.5);
    }
    w.Ltop[k + 1] = lt;
    w.Lbtm[k + 1] = lb;
  }
  for (int k = 1; k <= L; ++k) {
    LL[k + 1] += w.Ltop[k];
    LL[k] += w.Lbtm[k];
  }
  // interface-value limiters (:319-339): each entry's chain of clamps, reversed
  for (int j = 2; j <= L; ++j) {
    bool is_min[6];
    double bound[6];
    int vsel[6];
    int n = 0;
    auto min_hi = [&](int p, int q) {  // x = mn(x, mx(var[p], var[q]))
      is_min[n] = true;
      bool t = var[p] < var[q];
      bound[n] = t ? var[q] : var[p];
      vsel[n] = t ? q : p;
      ++n;
    };
    auto max_lo = [&](int p, int q) {  // x = mx(x, mn(var[p], var[q]))
      is_min[n] = false;
      bool t = var[q] < var[p];
      bound[n] = t ? var[q] : var[p];
      vsel[n] = t ? q : p;
      ++n;
    };
    if (j == L) { min_hi(L, L - 1); max_lo(L, L - 1); }
    if (j == 2) { min_hi(2, 1); max_lo(2, 1); }
    if (j >= 3) {
      const int k = j - 1;
      if (k + 2 > L || gam[k + 2] * gam[k] > 0) { min_hi(k, k + 1); max_lo(k, k + 1); }
      else if (gam[k + 2] > 0) max_lo(k, k + 1);
      else min_hi(k, k + 1);
    }
    bool sel[6];
    double x = w.lvb[j];
    for (int i = 0; i < n; ++i) {
      sel[i] = is_min[i] ? (bound[i] < x) : (x < bound[i]);
      if (sel[i]) x = bound[i];
    }
    double lam = LL[j];
    for (int i = n - 1; i >= 0 && lam != 0.; --i)
      if (sel[i]) {
        Lvar[vsel[i]] += lam;
        lam = 0.;
      }
    LL[j] = lam;
  }
  // back substitution (:317-318)
  for (int k = L + 1; k >= 2; --k) {
    LL[k - 1] -= gam[k - 1] * LL[k];
    Lgam[k - 1] -= w.lvb[k - 1] * LL[k];
  }
  // first interface value (:314-316); a2 is the alpha of the loop's last pass
  const double a2 = (coord[3] - coord[2]) / (coord[2] - coord[1]);
  double La2;
  {
    const double b0 = 1. + a2 * (1.5 + a2);
    const double D1 = a2 * (.5 + a2) - b0 * gam[1];
    const double LN1 = LL[1] / D1, LD1 = -w.lvs[1] / D1 * LL[1];
    Lvar[1] += 2. * a2 * (1. + a2) * LN1;
    Lvar[2] += LN1;
    double Lb0 = -w.lvs[2] * LN1;
    LL[2] -= b0 * LN1;
    La2 = (2. + 4. * a2) * var[1] * LN1 + (.5 + 2. * a2) * LD1;
    Lb0 -= gam[1] * LD1;
    Lgam[1] -= b0 * LD1;
    La2 += (1.5 + 2. * a2) * Lb0;
  }
  // elimination (:306-313), reverse order k = 2..L
  for (int k = 2; k <= L; ++k) {
    const double nn = coord[k + 1] - coord[k], dd = coord[k] - coord[k - 1];
    const double ak = nn / dd;
    const double bek = 2. + 2. * ak - gam[k];
    double La = (k == 2) ? La2 : 0.;
    La += Lgam[k - 1] / bek;
    double Lbe = -gam[k - 1] / bek * Lgam[k - 1];
    const double LN = LL[k] / bek;
    Lbe -= w.lvs[k] / bek * LL[k];
    Lvar[k] += 3. * LN;
    Lvar[k - 1] += 3. * ak * LN;
    La += 3. * var[k - 1] * LN;
    LL[k + 1] -= LN;
    La += 2. * Lbe;
    Lgam[k] -= Lbe;
    Lc[k + 1] += La / dd;
    Lc[k] -= La / dd;
    const double Ld = -ak / dd * La;
    Lc[k] += Ld;
    Lc[k - 1] -= Ld;
  }
  // top interface value and gam(nlay) (:301-305)
  {
    const double nn = coord[L] - coord[L - 1], dd = coord[L + 1] - coord[L];
    const double aL = nn / dd;
    const double bL = aL * (.5 + aL);
    const double LNL = LL[L + 1] / bL;
    double LbL = -w.lvs[L + 1] / bL * LL[L + 1];
    Lvar[L] += 2. * aL * (1. + aL) * LNL;
    Lvar[L - 1] += LNL;
    double LaL = (2. + 4. * aL) * var[L] * LNL;
    const double LG = Lgam[L] / bL;
    LbL -= gam[L] / bL * Lgam[L];
    LaL += (1.5 + 2. * aL) * LG;
    LaL += (.5 + 2. * aL) * LbL;
    Lc[L] += LaL / dd;
    Lc[L - 1] -= LaL / dd;
    const double Ldd = -aL / dd * LaL;
    Lc[L + 1] += Ldd;
    Lc[L] -= Ldd;
  }
}

// adjoint of one pair's contribution (remap_pair) given source layer k's
// edges, curvature and value: adds to Ltop/Lbtm (with the curvature folded
// in), Lsrc, Lsc, Ldc
template <int LM>
__device__ __forceinline__ void remap_pair_adj(RemapAdjWork<LM>& w, double btm, double top, double curv, double vk,
                                               double ldst, const double* sc, const double* dc, int k, int m,
                                               double* Lsrc, double* Lsc, double* Ldc) {
  const double dsrc = sc[k + 1] - sc[k];
  const double s1 = (dc[m] - sc[k]) / dsrc;
  const double s2 = (dc[m + 1] - sc[k]) / dsrc;
  const double ddst = dc[m + 1] - dc[m];
  const double IF = dsrc / ddst;
  const double tmp3 = 2. * s1 * s1;
  double Ls1 = 0., Ls2 = 0., LIF = 0., Lb = 0., Lt = 0., Lcv = 0.;
  if (dc[m + 1] <= sc[k + 1] && sc[k + 1] < dc[m] && dc[m] < sc[k]) {
    const double t1 = s1 - 1., t2 = s1 + 1.;
    const double A = 3. * (btm * t1 - top * t2) + curv * (tmp3 - t2);
    const double f = t1 / 6. * IF * ldst;
    Lb += f * 3. * t1;
    Lt -= f * 3. * t2;
    Lcv += f * (tmp3 - t2);
    LIF += t1 / 6. * A * ldst;
    Ls1 += (A / 6. * IF + t1 / 6. * IF * (3. * (btm - top) + curv * (4. * s1 - 1.))) * ldst;
  }
  if (sc[k + 1] < dc[m + 1] && dc[m + 1] < sc[k] && sc[k] <= dc[m]) {
    const double B = btm * (2. - s2) + s2 * (top + curv * (1. - C2_3 * s2));
    const double f = s2 / 2. * IF * ldst;
    Lb += f * (2. - s2);
    Lt += f * s2;
    Lcv += f * s2 * (1. - C2_3 * s2);
    LIF += s2 / 2. * B * ldst;
    Ls2 += (.5 * B * IF + s2 / 2. * IF * (-btm + top + curv * (1. - 2. * C2_3 * s2))) * ldst;
  }
  if (dc[m + 1] <= sc[k + 1] && sc[k] <= dc[m]) {
    Lsrc[k] += IF * ldst;
    LIF += vk * ldst;
  }
  if (sc[k + 1] < dc[m + 1] && dc[m] < sc[k]) {
    const double t1 = s1 + s2;
    const double C = 3. * (btm * (t1 - 2.) - top * t1) + curv * (tmp3 + t1 * (2. * s2 - 3.));
    const double f = (s1 - s2) / 6. * IF * ldst;
    Lb += f * 3. * (t1 - 2.);
    Lt -= f * 3. * t1;
    Lcv += f * (tmp3 + t1 * (2. * s2 - 3.));
    LIF += (s1 - s2) / 6. * C * ldst;
    const double dC1 = 3. * (btm - top) + curv * (4. * s1 + 2. * s2 - 3.);
    const double dC2 = 3. * (btm - top) + curv * (2. * s2 - 3. + 2. * t1);
    Ls1 += (C * IF / 6. + (s1 - s2) / 6. * IF * dC1) * ldst;
    Ls2 += (-C * IF / 6. + (s1 - s2) / 6. * IF * dC2) * ldst;
  }
  // curvature = 6 var - 3 (top + btm)
  Lsrc[k] += 6. * Lcv;
  w.Ltop[k] += Lt - 3. * Lcv;
  w.Lbtm[k] += Lb - 3. * Lcv;
  const double Ldsrc = -(Ls1 * s1 + Ls2 * s2) / dsrc + LIF / ddst;
  Ldc[m] += Ls1 / dsrc + LIF * IF / ddst;
  Ldc[m + 1] += Ls2 / dsrc - LIF * IF / ddst;
  Lsc[k] += -(Ls1 + Ls2) / dsrc - Ldsrc;
  Lsc[k + 1] += Ldsrc;
}

// All-pairs adjoint of remap_column for coordinates that are not monotone
// (every source layer against every target layer, as the reference loops),
// with its own column arrays.
template <int LM>
__device__ __noinline__ void remap_column_adj_full(int L, const double* src_var, const double* Ldst, const double* sc,
                                                   const double* dc, double* Lsrc, double* Lsc, double* Ldc) {
  RemapAdjFull<LM> w;
  vppm_record<LM>(w, L, src_var, sc);
  for (int k = 0; k <= L + 1; ++k) {
    w.Ltop[k] = 0.;
    w.Lbtm[k] = 0.;
  }
  for (int k = 1; k <= L; ++k)
    for (int m = 1; m <= L; ++m) {
      if (sc[k + 1] >= dc[m] || sc[k] <= dc[m + 1] || Ldst[m] == 0.) continue;
      remap_pair_adj<LM>(w, w.btm[k], w.top[k], w.curv[k], src_var[k], Ldst[m], sc, dc, k, m, Lsrc, Lsc, Ldc);
    }
  vppm_adj<LM>(w, L, src_var, sc, Lsrc, Lsc);
}

// Adjoint of remap_column: given the adjoint Ldst of the remapped values,
// adds to Lsrc (source values), Lsc (source coordinate), Ldc (target).
// Monotone coordinates (the usual case): the elimination of vertical_ppm
// as the forward's streaming remap does it (ppm_eliminate), then the pairs
// in the forward merge's order with each source layer's edges and curvature
// formed as the merge reaches it (PPMLayers, which also yields the back
// substituted and limited interface values the reverse of vertical_ppm
// reads); the same operations as vertical_ppm, so the same values.
template <int LM>
__device__ void remap_column_adj(RemapAdjWork<LM>& w, int L, const double* src_var, const double* Ldst, const double* sc,
                                 const double* dc, double* Lsrc, double* Lsc, double* Ldc) {
  bool mono = true;
  for (int k = 1; k <= L; ++k) mono = mono && (sc[k + 1] <= sc[k]) && (dc[k + 1] <= dc[k]);
  if (!mono) {
    remap_column_adj_full<LM>(L, src_var, Ldst, sc, dc, Lsrc, Lsc, Ldc);
    return;
  }
  const ColArr csc{const_cast<double*>(sc), 1}, clv{w.lvs, 1}, cgam{w.gam, 1};
  {
    int kc = L + 2, kv = L + 1;
    ppm_eliminate<false>(L, [&]() { return sc[--kc]; }, [&]() { return src_var[--kv]; }, csc, clv, cgam);
  }
  for (int k = 0; k <= L + 1; ++k) {
    w.Ltop[k] = 0.;
    w.Lbtm[k] = 0.;
  }
  auto var = [&](int k) { return src_var[k]; };
  PPMLayers<decltype(var)> ly(clv, cgam, L, var);
  w.lvb[1] = ly.lvf;
  w.lvc[1] = ly.lvc;
  auto advance = [&]() {  // to the next layer; its top interface values
    ly.next();
    w.lvb[ly.k + 1] = ly.lvf;
    w.lvc[ly.k + 1] = ly.lvc;
  };
  int k0 = 1;
  for (int m = 1; m <= L; ++m) {
    while (k0 <= L && sc[k0 + 1] >= dc[m]) ++k0;
    if (Ldst[m] == 0.) continue;
    for (int k = k0; k <= L && sc[k] > dc[m + 1]; ++k) {
      while (ly.k < k) advance();
      remap_pair_adj<LM>(w, ly.btm, ly.top, ly.curv, ly.vk, Ldst[m], sc, dc, k, m, Lsrc, Lsc, Ldc);
    }
  }
  while (ly.k < L) advance();
  vppm_adj<LM>(w, L, src_var, sc, Lsrc, Lsc);
}

// remap_column of the energy for coordinates that are not monotone, with
// its own column arrays
template <int LM>
__device__ __noinline__ void remap_energy_pairs(int L, const double* en, double* er, const double* plev,
                                                const double* tpl) {
  PPMWork<LM> wf;
  remap_column<LM>(wf, L, en, er, plev, tpl, nullptr, 1, nullptr);
}

// Adjoint of k_remap_energy (src/mod_remap.f90:42-78, 111-161) on the
// interior: adjoints of the remapped dp, pt, ud, vd in; adjoints of the
// pre-remap dp, pt (this column), ud, vd (its A-grid neighbours) and of the
// remapped face winds urem, vrem out.
// One thread per column, its arrays in local memory: more than 64 layers, many
// columns (remap_adj_columns), and columns whose coordinates are not monotone
// (atm_remap_adj.cuh has the others).
template <int LM>
__device__ __noinline__ void remap_energy_adj_at(const Geom& g, const RemapArgs& ra, const double* dp, const double* pt,
                                                 const double* ud, const double* vd, const double* urem,
                                                 const double* vrem, const double* gzs, const double* lam_dpo,
                                                 const double* lam_pto, double* lam_dp, double* lam_pt, double* lam_ud,
                                                 double* lam_vd, double* lam_ur, double* lam_vr, int i, int j) {
  const int L = g.L;
  const long long S = g.S;
  const long long o = g.at(i, j);
  const int P = g.P;
  double plev[LM + 2], pk[LM + 2], tpl[LM + 2], tpk[LM + 2];
  double en[LM + 2], ptr[LM + 2];
  double Lplev[LM + 2], Ltpl[LM + 2], Lpk[LM + 2], Ltpk[LM + 2], Ler[LM + 2];
  RemapAdjWork<LM> wk;
  // forward recomputation, as k_remap_energy
  plev[L + 1] = ra.ptop;
  pk[L + 1] = ra.pk_top;
  double lyk[LM + 2], tlyk[LM + 2];
  for (int k = L; k >= 1; --k) {
    plev[k] = plev[k + 1] + dp[o + (long long)(k - 1) * S];
    pk[k] = atm_pow(plev[k], KAPPA);
    double plog = atm_log(pk[k + 1] / pk[k]);
    lyk[k] = (pk[k + 1] - pk[k]) / plog;
  }
  tpl[L + 1] = ra.ptop;
  tpk[L + 1] = ra.pk_top;
  for (int k = L; k >= 1; --k) {
    tpl[k] = ra.ak[k - 1] + ra.bk[k - 1] * (plev[1] - ra.ptop);
    tpk[k] = atm_pow(tpl[k], KAPPA);
    double plog = atm_log(tpk[k + 1] / tpk[k]);
    tlyk[k] = (tpk[k + 1] - tpk[k]) / plog;
  }
  {
    double gz0 = gzs[o];  // gz(k), streamed upward
    for (int k = 1; k <= L; ++k) {
      long long ok = o + (long long)(k - 1) * S;
      const double gz1 = gz0 + CP_DRY * pt[ok] * (pk[k] - pk[k + 1]);
      double ua = (.25 * (ud[ok] + ud[ok + P]) + .125 * (ud[ok - 1] + ud[ok - 1 + P] + ud[ok + 1] + ud[ok + 1 + P]));
      double va = (.25 * (vd[ok] + vd[ok + 1]) + .125 * (vd[ok - P] + vd[ok + 1 - P] + vd[ok + P] + vd[ok + 1 + P]));
      en[k] = CV_DRY * pt[ok] * lyk[k] + .5 * (gz1 + gz0 + ua * ua + va * va);
      gz0 = gz1;
    }
  }
  {
    // the remapped energy er(m), ascending, and the recovered pt (:127-150)
    double gzr = gzs[o];
    auto put = [&](int m, double erm) {
      long long ok = o + (long long)(m - 1) * S;
      double ua = (.25 * (urem[ok] + urem[ok + P]) + .125 * (urem[ok - 1] + urem[ok - 1 + P] + urem[ok + 1] + urem[ok + 1 + P]));
      double va = (.25 * (vrem[ok] + vrem[ok + 1]) + .125 * (vrem[ok - P] + vrem[ok + 1 - P] + vrem[ok + P] + vrem[ok + 1 + P]));
      ptr[m] = (erm - gzr - .5 * (ua * ua + va * va)) / (CV_DRY * tlyk[m] + .5 * CP_DRY * (tpk[m] - tpk[m + 1]));
      gzr = gzr + CP_DRY * ptr[m] * (tpk[m] - tpk[m + 1]);
    };
    bool mono = true;
    for (int k = 1; k <= L; ++k) mono = mono && (plev[k + 1] <= plev[k]) && (tpl[k + 1] <= tpl[k]);
    if (mono) {  // the forward's streaming remap (the energy kernel's path)
      const ColArr cpl{plev, 1}, clv{wk.lvs, 1}, cgam{wk.gam, 1};
      int kc = L + 2, kv = L + 1;
      ppm_eliminate<false>(L, [&]() { return plev[--kc]; }, [&]() { return en[--kv]; }, cpl, clv, cgam);
      remap_merge(L, cpl, clv, cgam, [&](int k) { return en[k]; }, [&](int k) { return tpl[k]; }, put, nullptr, 1);
    } else {  // all pairs, into Ler as scratch (it is cleared below)
      remap_energy_pairs<LM>(L, en, Ler, plev, tpl);
      for (int m = 1; m <= L; ++m) put(m, Ler[m]);
    }
  }
  for (int k = 0; k <= L + 1; ++k) {
    Lplev[k] = 0.; Ltpl[k] = 0.; Lpk[k] = 0.; Ltpk[k] = 0.; Ler[k] = 0.;
  }
  // outputs: dp = tpl(k) - tpl(k+1) (:156-161)
  for (int k = 1; k <= L; ++k) {
    long long ok = o + (long long)(k - 1) * S;
    const double ld = lam_dpo[ok];
    Ltpl[k] += ld;
    Ltpl[k + 1] -= ld;
  }
  // pt recovery and the remapped geopotential (:130-150), reverse
  {
    double lgz = 0.;  // adjoint of gz_remap(k+1)
    for (int k = L; k >= 1; --k) {
      long long ok = o + (long long)(k - 1) * S;
      const double dtp = tpk[k] - tpk[k + 1];
      const double Dk = CV_DRY * tlyk[k] + .5 * CP_DRY * dtp;
      const double lp = lam_pto[ok] + CP_DRY * dtp * lgz;
      Ltpk[k] += CP_DRY * ptr[k] * lgz;
      Ltpk[k + 1] -= CP_DRY * ptr[k] * lgz;
      const double ln = lp / Dk;  // adjoint of the numerator
      Ler[k] += ln;
      lgz -= ln;
      const double LD = -ptr[k] / Dk * lp;
      // tlyk(k) = (tpk(k+1) - tpk(k)) / log(tpk(k+1) / tpk(k))
      const double lg = log(tpk[k + 1] / tpk[k]);
      const double Ly = CV_DRY * LD;
      Ltpk[k + 1] += Ly * (1. - tlyk[k] / tpk[k + 1]) / lg;
      Ltpk[k] += Ly * (-1. + tlyk[k] / tpk[k]) / lg;
      Ltpk[k] += .5 * CP_DRY * LD;
      Ltpk[k + 1] -= .5 * CP_DRY * LD;
      // ua, va of the remapped face winds
      const double ua = (.25 * (urem[ok] + urem[ok + P]) + .125 * (urem[ok - 1] + urem[ok - 1 + P] + urem[ok + 1] + urem[ok + 1 + P]));
      const double va = (.25 * (vrem[ok] + vrem[ok + 1]) + .125 * (vrem[ok - P] + vrem[ok + 1 - P] + vrem[ok + P] + vrem[ok + 1 + P]));
      const double lu = -ua * ln, lv = -va * ln;
      if (lu != 0.) {
        atomicAdd(lam_ur + ok, .25 * lu);
        atomicAdd(lam_ur + ok + P, .25 * lu);
        atomicAdd(lam_ur + ok - 1, .125 * lu);
        atomicAdd(lam_ur + ok - 1 + P, .125 * lu);
        atomicAdd(lam_ur + ok + 1, .125 * lu);
        atomicAdd(lam_ur + ok + 1 + P, .125 * lu);
      }
      if (lv != 0.) {
        atomicAdd(lam_vr + ok, .25 * lv);
        atomicAdd(lam_vr + ok + 1, .25 * lv);
        atomicAdd(lam_vr + ok - P, .125 * lv);
        atomicAdd(lam_vr + ok + 1 - P, .125 * lv);
        atomicAdd(lam_vr + ok + P, .125 * lv);
        atomicAdd(lam_vr + ok + 1 + P, .125 * lv);
      }
    }
  }
  // the energy remap (:107-110)
  double Lsrc[LM + 2];
  for (int k = 0; k <= L + 1; ++k) Lsrc[k] = 0.;
  remap_column_adj<LM>(wk, L, en, Ler, plev, tpl, Lsrc, Lplev, Ltpl);
  // target pressures (:57-71): tpk = tpl**kappa, tpl = ak + bk (ps - ptop)
  for (int k = 1; k <= L; ++k) {
    Ltpl[k] += Ltpk[k] * KAPPA * tpk[k] / tpl[k];
    Lplev[1] += ra.bk[k - 1] * Ltpl[k];
  }
  // energy (:72-78), hydrostatic gz (:53-56), playkap (:46-52)
  double Lpt[LM + 2];
  {
    for (int k = 1; k <= L; ++k) {
      long long ok = o + (long long)(k - 1) * S;
      const double le = Lsrc[k];
      Lpt[k] = CV_DRY * lyk[k] * le;
      // lyk(k) = (pk(k+1) - pk(k)) / log(pk(k+1) / pk(k))
      const double ly = CV_DRY * pt[ok] * le;
      const double lg = log(pk[k + 1] / pk[k]);
      Lpk[k + 1] += ly * (1. - lyk[k] / pk[k + 1]) / lg;
      Lpk[k] += ly * (-1. + lyk[k] / pk[k]) / lg;
      // the adjoint of en(k) (Lsrc(k)) also reaches .5 (gz(k+1) + gz(k)) and the kinetic energy
      const double ua = (.25 * (ud[ok] + ud[ok + P]) + .125 * (ud[ok - 1] + ud[ok - 1 + P] + ud[ok + 1] + ud[ok + 1 + P]));
      const double va = (.25 * (vd[ok] + vd[ok + 1]) + .125 * (vd[ok - P] + vd[ok + 1 - P] + vd[ok + P] + vd[ok + 1 + P]));
      const double lu = ua * le, lv = va * le;
      if (lu != 0.) {
        atomicAdd(lam_ud + ok, .25 * lu);
        atomicAdd(lam_ud + ok + P, .25 * lu);
        atomicAdd(lam_ud + ok - 1, .125 * lu);
        atomicAdd(lam_ud + ok - 1 + P, .125 * lu);
        atomicAdd(lam_ud + ok + 1, .125 * lu);
        atomicAdd(lam_ud + ok + 1 + P, .125 * lu);
      }
      if (lv != 0.) {
        atomicAdd(lam_vd + ok, .25 * lv);
        atomicAdd(lam_vd + ok + 1, .25 * lv);
        atomicAdd(lam_vd + ok - P, .125 * lv);
        atomicAdd(lam_vd + ok + 1 - P, .125 * lv);
        atomicAdd(lam_vd + ok + P, .125 * lv);
        atomicAdd(lam_vd + ok + 1 + P, .125 * lv);
      }
    }
    // gz(k+1) = gz(k) + cp pt(k) (pk(k) - pk(k+1)); d en(k) / d gz(k), gz(k+1) = .5
    double lz = 0.;
    for (int k = L; k >= 1; --k) {
      long long ok = o + (long long)(k - 1) * S;
      lz += .5 * Lsrc[k];  // gz(k+1)
      if (k + 1 <= L) lz += .5 * Lsrc[k + 1];  // gz(k+1) is also the lower level of layer k+1
      Lpt[k] += CP_DRY * (pk[k] - pk[k + 1]) * lz;
      Lpk[k] += CP_DRY * pt[ok] * lz;
      Lpk[k + 1] -= CP_DRY * pt[ok] * lz;
    }
  }
  // pk = plev**kappa; plev(k) = plev(k+1) + dp(k)
  for (int k = 1; k <= L; ++k) Lplev[k] += Lpk[k] * KAPPA * pk[k] / plev[k];
  double acc = 0.;
  for (int k = 1; k <= L; ++k) {
    long long ok = o + (long long)(k - 1) * S;
    acc += Lplev[k];
    lam_dp[ok] += acc;
    lam_pt[ok] += Lpt[k];
  }
}

// 16 blocks of 64 threads per SM (64 registers; more columns in flight to
// hide the local-memory latency of the column arrays)
template <int LM>
__global__ void __launch_bounds__(64, 16) k_remap_energy_adj(Geom g, RemapArgs ra, const double* dp,
                                                         const double* pt, const double* ud,
                                                         const double* vd, const double* urem,
                                                         const double* vrem, const double* gzs,
                                                         const double* lam_dpo,
                                                         const double* lam_pto,
                                                         const double* lam_udo,
                                                         const double* lam_vdo, double* lam_dp,
                                                         double* lam_pt, double* lam_ud, double* lam_vd, double* lam_ur,
                                                         double* lam_vr) {
  stream_order();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.nx * g.ny) return;
  const int i = col % g.nx, j = col / g.nx;
  const long long o = g.at(i, j);
  // ud = urem and vd = vrem (:156-161); the column's energy and pressure
  // adjoints are zero unless its new dp or pt carry an adjoint
  bool any = false;
  for (int k = 0; k < g.L; ++k) {
    const long long ok = o + (long long)k * g.S;
    if (lam_udo[ok] != 0.) atomicAdd(lam_ur + ok, lam_udo[ok]);
    if (lam_vdo[ok] != 0.) atomicAdd(lam_vr + ok, lam_vdo[ok]);
    any = any || lam_dpo[ok] != 0. || lam_pto[ok] != 0.;
  }
  if (any)
    remap_energy_adj_at<LM>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_dp, lam_pt, lam_ud, lam_vd,
                            lam_ur, lam_vr, i, j);
}

// Adjoint of k_remap_winds (src/mod_remap.f90:80-105) of direction dir at a
// point of [-1, nx] x [-1, ny]: the adjoint lr of the remapped wind in; that of
// the wind f of the column (lf) and of dp of the four columns that form its
// source and target interface pressures out.
template <int LM>
__device__ __noinline__ void remap_winds_adj_at(const Geom& g, const RemapArgs& ra, const double* dp, const double* f,
                                                const double* lr, double* lam_dp, double* lf, int i, int j, int dir) {
  const int L = g.L;
  double sc[LM + 2], dc[LM + 2], var[LM + 2], Ld[LM + 2], Lv[LM + 2], Ls[LM + 2], Lt[LM + 2];
  RemapAdjWork<LM> wk;
  const long long o = g.at(i, j), oa = o;
  const long long ob = dir == 0 ? g.at(i, j - 1) : g.at(i - 1, j);
  const long long oc = dir == 0 ? g.at(i, j + 1) : g.at(i + 1, j);
  const long long od = dir == 0 ? g.at(i, j - 2) : g.at(i - 2, j);
  double pa = ra.ptop, pb = ra.ptop, pc = ra.ptop, pd = ra.ptop;
  bool any = false;
  for (int k = L + 1; k >= 1; --k) {
    if (k <= L) {
      const long long kk = (long long)(k - 1) * g.S;
      pa = pa + dp[oa + kk];
      pb = pb + dp[ob + kk];
      pc = pc + dp[oc + kk];
      pd = pd + dp[od + kk];
      var[k] = f[o + kk];
      Ld[k] = lr[o + kk];
      any = any || Ld[k] != 0.;
    }
    sc[k] = C7_12 * (pa + pb) - C1_12 * (pc + pd);
  }
  if (!any) return;
  for (int k = 1; k <= L + 1; ++k) {
    double ta, tb, tc, td;
    if (k <= L) {
      const double a = ra.ak[k - 1], b = ra.bk[k - 1];
      ta = a + b * (pa - ra.ptop);
      tb = a + b * (pb - ra.ptop);
      tc = a + b * (pc - ra.ptop);
      td = a + b * (pd - ra.ptop);
    } else {
      ta = tb = tc = td = ra.ptop;
    }
    dc[k] = C7_12 * (ta + tb) - C1_12 * (tc + td);
  }
  for (int k = 0; k <= L + 1; ++k) { Lv[k] = 0.; Ls[k] = 0.; Lt[k] = 0.; }
  remap_column_adj<LM>(wk, L, var, Ld, sc, dc, Lv, Ls, Lt);
  for (int k = 1; k <= L; ++k) lf[o + (long long)(k - 1) * g.S] += Lv[k];
  // sc(k) = 7/12 (pa + pb) - 1/12 (pc + pd), p(k) = ptop + sum of dp(m >= k);
  // dc(k) = 7/12 (ta + tb) - 1/12 (tc + td), t = ak + bk (ps - ptop)
  double Z = 0.;
  for (int k = 1; k <= L; ++k) Z += ra.bk[k - 1] * Lt[k];
  double P = 0.;
  for (int m = 1; m <= L; ++m) {
    P += Ls[m];
    const double v = P + Z;
    if (v == 0.) continue;
    const long long kk = (long long)(m - 1) * g.S;
    atomicAdd(lam_dp + oa + kk, C7_12 * v);
    atomicAdd(lam_dp + ob + kk, C7_12 * v);
    atomicAdd(lam_dp + oc + kk, -C1_12 * v);
    atomicAdd(lam_dp + od + kk, -C1_12 * v);
  }
}

// (blockIdx.y: the direction)
template <int LM>
__global__ void __launch_bounds__(64, 16) k_remap_winds_adj(Geom g, RemapArgs ra, const double* dp,
                                                        const double* ud, const double* vd,
                                                        const double* lam_ur,
                                                        const double* lam_vr, double* lam_dp,
                                                        double* lam_ud, double* lam_vd) {
  stream_order();
  const int w = g.nx + 2, h = g.ny + 2;
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= w * h) return;
  const int i = -1 + col % w, j = -1 + col / w, dir = blockIdx.y;
  remap_winds_adj_at<LM>(g, ra, dp, dir == 0 ? ud : vd, dir == 0 ? lam_ur : lam_vr, lam_dp, dir == 0 ? lam_ud : lam_vd,
                         i, j, dir);
}

}  // namespace atm
