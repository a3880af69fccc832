// Reverse of the vertical remap (src/mod_remap.f90:27-163) in the shared-level
// form of atm_remap.cuh: a block owns 32 columns, its warps share the levels,
// the column arrays lie in shared memory.
//
// The forward is recomputed with the forward's operations (hence its limiter
// branches and layer pairs).  The reverse of a column is, like the forward, a
// few linear chains -- back substitution, elimination, running sums -- run by
// one warp with their coefficients formed beforehand, between stages that are
// independent per level: the layer pairs (each source layer gathers from the
// targets that overlap it), the limiters, the powers and logarithms.  What a
// level passes to its neighbours goes through an array and a barrier.  The
// target coordinate is linear in the surface pressures, so its adjoint is one
// number per column.
//
// Measured on B200 (the reverse of a remap with the forward winds it needs, ms;
// before: one thread a column, about twenty column arrays in local memory, waits
// of 16 to 18 cycles an issued instruction on them): 64x64x20 0.80 -> 0.15,
// 301x203x40 3.83 -> 2.08, 512x512x32 7.46 -> 5.61.  Now the chains' barriers (5
// cycles an issued instruction at two blocks an SM).  Before the layers' edges and the
// target coordinate were kept: 0.15 / 2.19 / 5.98; with that, 4 warps a block: 0.22 /
// 3.25 / 7.19; 16: 0.13 / 2.18 / 5.86; 8 warps at three blocks (80 registers,
// spilling): 0.16 / 2.41 / 5.81.
#pragma once

#include "atm_adjoint.cuh"
#include "atm_remap.cuh"

namespace atm {

constexpr int RMA_WARPS = 8, RMA_PART = RMA_WARPS < 8 ? 8 : RMA_WARPS;

// edges of layer k from the unlimited interface values A and coefficients B;
// cb, ct: the limited interface values below and above
template <typename FV>
__device__ __forceinline__ void adj_edges(int k, int L, ShCol A, ShCol B, const FV& var, double vk, double& cb,
                                          double& ct, double& btm, double& top) {
  cb = k == 1 ? A[1] : remap_interface(k, L, A, B, var);
  ct = k == L ? A[L + 1] : remap_interface(k + 1, L, A, B, var);
  btm = cb;
  top = ct;
  if (k >= 3) {
    const double gk1 = B[k];
    double pmp1 = vk - 2. * gk1;
    double lac1 = pmp1 + 1.5 * B[k - 1];
    top = mn(mx(top, mn3(vk, pmp1, lac1)), mx3(vk, pmp1, lac1));
    pmp1 = vk + 2. * B[k + 1];
    lac1 = pmp1 - 1.5 * gk1;
    btm = mn(mx(btm, mn3(vk, pmp1, lac1)), mx3(vk, pmp1, lac1));
  }
}

// vertical_ppm's elimination and back substitution: on return A[k], k = 1..L+1,
// the unlimited interface values, B[k+1] = gam(k), k = 1..L
template <typename FV>
__device__ __forceinline__ void adj_solve(int L, ShCol sc, ShCol A, ShCol B, const FV& var, int warp) {
  for (int k = 2 + warp; k <= L; k += RMA_WARPS) {
    const double c1 = sc[k];
    const double alpha = (sc[k + 1] - c1) / (c1 - sc[k - 1]);
    A[k] = 3. * (var(k) + alpha * var(k - 1));
    B[k] = alpha;
  }
  __syncthreads();
  if (warp == 0) remap_solve<double>(L, sc, A, B, var(1), var(2), var(L - 1), var(L));
  __syncthreads();
}

// the reverse of one edge clamp: the adjoint of x0; gains of the layer's value,
// of the coefficient in b and of the one that c has beside it
__device__ __forceinline__ double clamp_adj(double x0, double a, double b, double c, double lam, double& lv, double& l2,
                                            double s2, double& l15, double s15) {
  const double lo = mn3(a, b, c), hi = mx3(a, b, c), inner = mx(x0, lo);
  if (!(hi < inner) && !(x0 < lo)) return lam;
  const int s = hi < inner ? sel_mx3(a, b, c) : sel_mn3(a, b, c);
  lv += lam;
  if (s != 0) l2 += s2 * lam;
  if (s == 2) l15 += s15 * lam;
  return 0.;
}

// Reverse of remap_column (monotone coordinates) for the levels k = 1 + warp +
// i * RMA_WARPS of the lane's column: from the adjoint ldst(m) of the remapped
// values, those of the source values (Lv) and of the source coordinate (Ls),
// and Z += sum of bk(m) times that of the target coordinate dc(m), this
// thread's part.  A, B from adj_solve; LL, Lg, T scratch, consumed like A and B
// (dc may read T: it is written after the pairs).
template <int LM, typename FV, typename FD, typename FL, typename FB>
__device__ __forceinline__ void remap_adj_core(int L, ShCol sc, ShCol A, ShCol B, ShCol LL, ShCol Lg, ShCol T,
                                               double (*ex)[RM_LANES], const FV& var, const FD& dc, const FL& ldst,
                                               const FB& bk, int warp, double (&Lv)[(LM + RMA_WARPS - 1) / RMA_WARPS],
                                               double (&Ls)[(LM + RMA_WARPS - 1) / RMA_WARPS], double& Z) {
  constexpr int N = (LM + RMA_WARPS - 1) / RMA_WARPS;
  const int lane = threadIdx.x & 31;
  double up[N], e2[N], g1[N], g2[N];  // to LL(k+1), Ls(k+1), Lg(k-1), Lg(k-2)
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    Lv[i] = Ls[i] = up[i] = e2[i] = g1[i] = g2[i] = 0.;
    if (k > L) continue;
    const double vk = var(k), sk = sc[k], sk1 = sc[k + 1];
    double cb, ct, btm, top;
    adj_edges(k, L, A, B, var, vk, cb, ct, btm, top);
    const double cv = 6. * vk - 3. * (top + btm), dsrc = sk1 - sk, rs = 1. / dsrc;
    double Lb = 0., Lt = 0., Lcv = 0., Lsrc = 0., Ldsrc = 0., Lsk = 0.;
    int m = k;  // the first target whose lower level lies below the layer's base, looked for from k
    while (m > 1 && dc(m) < sk) --m;
    double d0 = dc(m), d1 = dc(m + 1);
    while (m <= L && !(d1 < sk)) {
      ++m;
      d0 = d1;
      if (m <= L) d1 = dc(m + 1);
    }
    for (; m <= L && d0 > sk1; ++m) {
      const double ld = ldst(m);
      if (ld != 0.) {
        const double rd = 1. / (d1 - d0), IF = dsrc * rd;
        const double s1 = (d0 - sk) * rs, s2 = (d1 - sk) * rs;
        const bool over = d1 <= sk1, under = sk <= d0;
        double Ls1 = 0., Ls2 = 0., LIF = 0.;
        if (over && under) {
          Lsrc += IF * ld;
          LIF = vk * ld;
        } else if (over) {
          const double t1 = s1 - 1., t2 = s1 + 1., w = 2. * s1 * s1 - t2;
          const double q = 3. * (btm * t1 - top * t2) + cv * w, h = t1 * (1. / 6.), f = h * IF * ld;
          Lb += f * 3. * t1;
          Lt -= f * 3. * t2;
          Lcv += f * w;
          LIF = h * q * ld;
          Ls1 = (q * (1. / 6.) * IF + h * IF * (3. * (btm - top) + cv * (4. * s1 - 1.))) * ld;
        } else if (under) {
          const double w = 1. - C2_3 * s2, q = btm * (2. - s2) + s2 * (top + cv * w), h = s2 * .5, f = h * IF * ld;
          Lb += f * (2. - s2);
          Lt += f * s2;
          Lcv += f * s2 * w;
          LIF = h * q * ld;
          Ls2 = (.5 * q * IF + h * IF * (-btm + top + cv * (1. - 2. * C2_3 * s2))) * ld;
        } else {
          const double t1 = s1 + s2, w = 2. * s1 * s1 + t1 * (2. * s2 - 3.);
          const double q = 3. * (btm * (t1 - 2.) - top * t1) + cv * w, h = (s1 - s2) * (1. / 6.), f = h * IF * ld;
          Lb += f * 3. * (t1 - 2.);
          Lt -= f * 3. * t1;
          Lcv += f * w;
          LIF = h * q * ld;
          const double b = 3. * (btm - top), q6 = q * IF * (1. / 6.);
          Ls1 = (q6 + h * IF * (b + cv * (4. * s1 + 2. * s2 - 3.))) * ld;
          Ls2 = (h * IF * (b + cv * (2. * s2 - 3. + 2. * t1)) - q6) * ld;
        }
        Ldsrc += LIF * rd - (Ls1 * s1 + Ls2 * s2) * rs;
        Lsk -= (Ls1 + Ls2) * rs;
        const double y = LIF * IF * rd;
        Z += bk(m) * (Ls1 * rs + y) + bk(m + 1) * (Ls2 * rs - y);
      }
      d0 = d1;
      if (m < L) d1 = dc(m + 2);
    }
    Lv[i] = Lsrc + 6. * Lcv;  // curvature = 6 var - 3 (top + btm)
    Lt -= 3. * Lcv;
    Lb -= 3. * Lcv;
    Ls[i] = Lsk - Ldsrc;
    e2[i] = Ldsrc;
    double g0 = 0.;
    if (k >= 3) {  // the edge limiters (:340-352)
      const double gk1 = B[k];
      if (Lt != 0.) {
        const double pmp1 = vk - 2. * gk1;
        Lt = clamp_adj(ct, vk, pmp1, pmp1 + 1.5 * B[k - 1], Lt, Lv[i], g1[i], -2., g2[i], 1.5);
      }
      if (Lb != 0.) {
        const double pmp1 = vk + 2. * B[k + 1];
        Lb = clamp_adj(cb, vk, pmp1, pmp1 - 1.5 * gk1, Lb, Lv[i], g0, 2., g1[i], -1.5);
      }
    }
    up[i] = Lt;
    LL[k] = Lb;
    Lg[k] = g0;
    if (k == L) LL[L + 1] = 0.;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k > L) continue;
    LL[k + 1] += up[i];
    T[k + 1] = e2[i];
    if (k >= 3) Lg[k - 1] += g1[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k > L || k < 2) continue;
    if (k >= 3) Lg[k - 2] += g2[i];
    Ls[i] += T[k];
    // the limiters of interface k (:319-339): the last clamp that held passes the adjoint on
    const double lam = LL[k];
    double below = 0.;
    if (lam != 0.) {
      double x = A[k];
      const double va = var(k - 1), vb = var(k);
      int last = 0;  // 1: layer k-1, 2: layer k
      auto clamp_hi = [&](bool t) {  // x = mn(x, the larger), t: it is layer k's
        const double b = t ? vb : va;
        if (b < x) {
          x = b;
          last = t ? 2 : 1;
        }
      };
      auto clamp_lo = [&](bool t) {  // x = mx(x, the smaller)
        const double b = t ? vb : va;
        if (x < b) {
          x = b;
          last = t ? 2 : 1;
        }
      };
      if (k == L || k == 2) {
        clamp_hi(!(vb < va));
        clamp_lo(!(va < vb));
      }
      if (k >= 3) {
        const bool both = k == L || B[k + 2] * B[k] > 0;
        const bool lo = both || B[k + 2] > 0, hi = both || !lo;
        if (hi) clamp_hi(va < vb);
        if (lo) clamp_lo(vb < va);
      }
      if (last) LL[k] = 0.;
      if (last == 2) Lv[i] += lam;
      if (last == 1) below = lam;
    }
    e2[i] = below;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k <= L && k >= 2) T[k] = e2[i];
  }
  if (warp == 0) {  // the back substitution (:317-318)
    double l = LL[L + 1];
    for (int k = L + 1; k >= 2; --k) {
      l = LL[k - 1] - B[k] * l;
      LL[k - 1] = l;
    }
  }
  __syncthreads();
  // coefficients of the elimination's reverse: p = 1/beta, q = gam(k-1) p, s = (value before substitution) p
  double q[N], s[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    q[i] = s[i] = 0.;
    if (k > L) continue;
    if (k < L) Lv[i] += T[k + 1];
    Lg[k] -= A[k] * LL[k + 1];
    if (k >= 2) {
      const double c1 = sc[k];
      const double a = (sc[k + 1] - c1) / (c1 - sc[k - 1]);
      e2[i] = 1. / (2. + 2. * a - B[k + 1]);
      q[i] = B[k] * e2[i];
      s[i] = (A[k] + B[k] * A[k - 1]) * e2[i];
    }
  }
  const double gam1 = B[2], gamL = B[L + 1];
  const double lvs1 = A[1], lvs2 = A[2] + gam1 * lvs1, lvsT = A[L + 1] + gamL * A[L];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k > L || k < 2) continue;
    T[k] = e2[i];
    B[k] = q[i];
    A[k] = s[i];
  }
  __syncthreads();
  if (warp == 0) {
    // first interface value (:314-316); a2 is the alpha of the loop's last pass
    const double a2 = (sc[3] - sc[2]) / (sc[2] - sc[1]), b0 = 1. + a2 * (1.5 + a2);
    const double rD = 1. / (a2 * (.5 + a2) - b0 * gam1);
    const double LN1 = LL[1] * rD, LD1 = -lvs1 * LN1;
    const double Lb0 = -lvs2 * LN1 - gam1 * LD1;
    ex[0][lane] = 2. * a2 * (1. + a2) * LN1;  // to layer 1
    ex[1][lane] = LN1;                        // to layer 2
    ex[2][lane] = (2. + 4. * a2) * var(1) * LN1 + (.5 + 2. * a2) * LD1 + (1.5 + 2. * a2) * Lb0;  // of a2
    double l = LL[2] - b0 * LN1, gm = Lg[1] - b0 * LD1;
    LL[2] = l;
    Lg[1] = gm;
    for (int k = 2; k <= L; ++k) {  // the elimination (:306-313)
      gm = Lg[k] + (B[k] * gm + A[k] * l);
      l = LL[k + 1] - T[k] * l;
      Lg[k] = gm;
      LL[k + 1] = l;
    }
    // top interface value and gam(nlay) (:301-305)
    const double rd = 1. / (sc[L + 1] - sc[L]), aL = (sc[L] - sc[L - 1]) * rd, rb = 1. / (aL * (.5 + aL));
    const double LNL = l * rb, LG = gm * rb;
    const double LbL = -lvsT * LNL - gamL * LG;
    const double La = (2. + 4. * aL) * var(L) * LNL + (1.5 + 2. * aL) * LG + (.5 + 2. * aL) * LbL;
    ex[3][lane] = 2. * aL * (1. + aL) * LNL;  // to layer L
    ex[4][lane] = LNL;                        // to layer L-1
    ex[5][lane] = La * rd + aL * rd * La;     // to the coordinate of L
    ex[6][lane] = -La * rd;                   // ... of L-1
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k > L || k < 2) continue;
    const double c1 = sc[k], rdd = 1. / (c1 - sc[k - 1]), a = (sc[k + 1] - c1) * rdd;
    const double p = T[k], l = LL[k], gm = Lg[k - 1];
    const double LN = p * l, Lbe = -(B[k] * gm + A[k] * l);
    double La = gm * p + 3. * var(k - 1) * LN + 2. * Lbe;
    if (k == 2) La += ex[2][lane];
    const double x = La * rdd;
    Lv[i] += 3. * LN;
    Ls[i] -= x + a * x;
    A[k] = 3. * a * LN;  // to layer k-1
    B[k] = a * x;        // to the coordinate of k-1
    T[k] = x;            // ... of k+1
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RMA_WARPS;
    if (k > L) continue;
    if (k < L) {
      Lv[i] += A[k + 1];
      Ls[i] += B[k + 1];
    }
    if (k >= 3) Ls[i] += T[k - 1];
    if (k == 1) Lv[i] += ex[0][lane];
    if (k == 2) Lv[i] += ex[1][lane];
    if (k == L) {
      Lv[i] += ex[3][lane];
      Ls[i] += ex[5][lane];
    }
    if (k == L - 1) {
      Lv[i] += ex[4][lane];
      Ls[i] += ex[6][lane];
    }
  }
}

// the sum over the block's warps of each lane's v
__device__ __forceinline__ double warps_sum(double v, double (*part)[RM_LANES], int warp, int lane) {
  part[warp][lane] = v;
  __syncthreads();
  double s = 0.;
  for (int q = 0; q < RMA_WARPS; ++q) s += part[q][lane];
  return s;
}

// Reverse of the wind remap (remap_winds_adj_at): blockIdx.y the direction.
// Six column arrays.
template <int LM>
__device__ __forceinline__ void remap_winds_adj_block(const Geom& g, const RemapArgs& ra, const double* __restrict__ dp,
                                                      const double* __restrict__ ud, const double* __restrict__ vd,
                                                      const double* __restrict__ lam_ur,
                                                      const double* __restrict__ lam_vr, double* lam_dp,
                                                      double* lam_ud, double* lam_vd) {
  constexpr int N = (LM + RMA_WARPS - 1) / RMA_WARPS;
  extern __shared__ double rm_sm[];
  __shared__ double part[RMA_PART][RM_LANES];
  __shared__ int bad[RM_LANES], act[RM_LANES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dir = blockIdx.y;
  const int w = g.nx + 2, h = g.ny + 2, L = g.L, st = (L + 2) * RM_LANES;
  const int col = blockIdx.x * RM_LANES + lane;
  const bool in = col < w * h;
  const int i = -1 + (in ? col % w : 0), j = -1 + (in ? col / w : 0);
  const long long S = g.S, oa = g.at(i, j);
  const double* f = dir == 0 ? ud : vd;
  const double* lr = dir == 0 ? lam_ur : lam_vr;
  const ShCol sc{rm_sm + lane}, A{rm_sm + st + lane}, B{rm_sm + 2 * st + lane}, LL{rm_sm + 3 * st + lane},
      Lg{rm_sm + 4 * st + lane}, T{rm_sm + 5 * st + lane};
  bool any = false;
  if (in)
    for (int k = 1 + warp; k <= L; k += RMA_WARPS) any = any || lr[oa + (long long)(k - 1) * S] != 0.;
  if (warp == 0) act[lane] = 0;
  if (!__syncthreads_or(any)) return;  // no adjoint reaches the block's columns
  if (any) act[lane] = 1;
  const long long ob = dir == 0 ? g.at(i, j - 1) : g.at(i - 1, j);
  const long long oc = dir == 0 ? g.at(i, j + 1) : g.at(i + 1, j);
  const long long od = dir == 0 ? g.at(i, j - 2) : g.at(i - 2, j);
  if (warp == 0) {
    double pa = ra.ptop, pb = ra.ptop, pc = ra.ptop, pd = ra.ptop;
    double prev = C7_12 * (pa + pb) - C1_12 * (pc + pd);
    sc[L + 1] = prev;
    bool mono = true;
#pragma unroll 4
    for (int k = L; k >= 1; --k) {
      const long long kk = (long long)(k - 1) * S;
      pa = pa + dp[oa + kk];
      pb = pb + dp[ob + kk];
      pc = pc + dp[oc + kk];
      pd = pd + dp[od + kk];
      const double c = C7_12 * (pa + pb) - C1_12 * (pc + pd);
      mono = mono && (prev <= c);
      sc[k] = c;
      prev = c;
    }
    part[0][lane] = pa;
    part[1][lane] = pb;
    part[2][lane] = pc;
    part[3][lane] = pd;
    bad[lane] = mono ? 0 : 1;
  }
  __syncthreads();
  const double pa = part[0][lane], pb = part[1][lane], pc = part[2][lane], pd = part[3][lane];
  auto dc = [&](int k) {
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
    return C7_12 * (ta + tb) - C1_12 * (tc + td);
  };
  for (int k = 1 + warp; k <= L + 1; k += RMA_WARPS) T[k] = dc(k);  // until the core's scratch
  auto var = [&](int k) { return f[oa + (long long)(k - 1) * S]; };
  auto ldst = [&](int k) { return lr[oa + (long long)(k - 1) * S]; };
  auto bk = [&](int k) { return k <= L ? ra.bk[k - 1] : 0.; };
  adj_solve(L, sc, A, B, var, warp);
  {
    bool mono = true;
    for (int k = 1 + warp; k <= L; k += RMA_WARPS) mono = mono && (T[k + 1] <= T[k]);
    if (!mono) bad[lane] = 1;
  }
  auto td = [&](int k) { return T[k]; };
  double Lv[N], Ls[N], Z = 0.;
  // (ex: the partial sums' array, not read again before the core's barriers)
  remap_adj_core<LM>(L, sc, A, B, LL, Lg, T, part, var, td, ldst, bk, warp, Lv, Ls, Z);
  __syncthreads();
  Z = warps_sum(Z, part, warp, lane);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k <= L) LL[k] = Ls[q];
  }
  __syncthreads();
  if (warp == 0) {  // sc(k) holds the layers m >= k
    double P = Z;
    for (int k = 1; k <= L; ++k) {
      P += LL[k];
      LL[k] = P;
    }
  }
  __syncthreads();
  if (!in || !act[lane]) return;
  if (bad[lane]) {  // coordinates that are not monotone: the all-pairs reverse
    if (warp == 0) remap_winds_adj_at<LM>(g, ra, dp, f, lr, lam_dp, dir == 0 ? lam_ud : lam_vd, i, j, dir);
    return;
  }
  double* lf = dir == 0 ? lam_ud : lam_vd;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k > L) continue;
    const long long kk = (long long)(k - 1) * S;
    if (Lv[q] != 0.) lf[oa + kk] += Lv[q];
    const double v = LL[k];
    if (v == 0.) continue;
    atomicAdd(lam_dp + oa + kk, C7_12 * v);
    atomicAdd(lam_dp + ob + kk, C7_12 * v);
    atomicAdd(lam_dp + oc + kk, -C1_12 * v);
    atomicAdd(lam_dp + od + kk, -C1_12 * v);
  }
}
template <int LM>
__global__ void __launch_bounds__(RM_LANES * RMA_WARPS, 2) k_remap_winds_adj_split(
    Geom g, RemapArgs ra, const double* dp, const double* ud, const double* vd, const double* lam_ur,
    const double* lam_vr, double* lam_dp, double* lam_ud, double* lam_vd) {
  stream_order();
  remap_winds_adj_block<LM>(g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud, lam_vd);
}

// Reverse of the energy remap (remap_energy_adj_at).  Eight column arrays; each
// thread keeps the powers of its levels in registers.
template <int LM>
__device__ __forceinline__ void remap_energy_adj_block(
    const Geom& g, const RemapArgs& ra, const double* __restrict__ dp, const double* __restrict__ pt,
    const double* __restrict__ ud, const double* __restrict__ vd, const double* __restrict__ urem,
    const double* __restrict__ vrem, const double* __restrict__ gzs, const double* __restrict__ lam_dpo,
    const double* __restrict__ lam_pto, const double* __restrict__ lam_udo, const double* __restrict__ lam_vdo,
    double* lam_dp, double* lam_pt, double* lam_ud, double* lam_vd, double* lam_ur, double* lam_vr) {
  constexpr int N = (LM + RMA_WARPS - 1) / RMA_WARPS;
  extern __shared__ double rm_sm[];
  __shared__ double part[RMA_PART][RM_LANES];
  __shared__ int bad[RM_LANES], act[RM_LANES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int L = g.L, P = g.P, st = (L + 2) * RM_LANES;
  const int col = blockIdx.x * RM_LANES + lane;
  const bool in = col < g.nx * g.ny;
  const int i = in ? col % g.nx : 0, j = in ? col / g.nx : 0;
  const long long S = g.S, o = g.at(i, j);
  const ShCol sc{rm_sm + lane}, A{rm_sm + st + lane}, B{rm_sm + 2 * st + lane}, en{rm_sm + 3 * st + lane},
      er{rm_sm + 4 * st + lane}, LL{rm_sm + 5 * st + lane}, Lg{rm_sm + 6 * st + lane}, T{rm_sm + 7 * st + lane};
  // ud = urem and vd = vrem (:156-161); the column's energy and pressure
  // adjoints are zero unless its new dp or pt carry an adjoint
  bool any = false;
  if (in)
    for (int k = 1 + warp; k <= L; k += RMA_WARPS) {
      const long long ok = o + (long long)(k - 1) * S;
      const double lu = lam_udo[ok], lv = lam_vdo[ok];
      if (lu != 0.) atomicAdd(lam_ur + ok, lu);
      if (lv != 0.) atomicAdd(lam_vr + ok, lv);
      any = any || lam_dpo[ok] != 0. || lam_pto[ok] != 0.;
    }
  if (warp == 0) act[lane] = 0;
  if (!__syncthreads_or(any)) return;
  if (any) act[lane] = 1;
  // forward recomputation, as k_remap_energy_split
  if (warp == 0) {
    double pl = ra.ptop;
    sc[L + 1] = pl;
    bool mono = true;
#pragma unroll 4
    for (int k = L; k >= 1; --k) {
      const double pn = pl + dp[o + (long long)(k - 1) * S];
      mono = mono && (pl <= pn);
      sc[k] = pn;
      pl = pn;
    }
    bad[lane] = mono ? 0 : 1;
  }
  __syncthreads();
  const double ps = sc[1];
  auto tpl = [&](int k) { return k <= L ? ra.ak[k - 1] + ra.bk[k - 1] * (ps - ra.ptop) : ra.ptop; };
  {
    bool mono = true;
    for (int k = 1 + warp; k <= L; k += RMA_WARPS) {
      A[k] = atm_pow(sc[k], KAPPA);
      T[k] = atm_pow(tpl(k), KAPPA);
      mono = mono && (tpl(k + 1) <= tpl(k));
    }
    if (warp == RMA_WARPS - 1) A[L + 1] = T[L + 1] = ra.pk_top;
    if (!mono) bad[lane] = 1;
  }
  __syncthreads();
  if (warp == 0) {  // gz (:70-75)
    double z = gzs[o], pk0 = A[1];
    B[1] = z;
#pragma unroll 4
    for (int k = 1; k <= L; ++k) {
      const double pk1 = A[k + 1];
      z = z + CP_DRY * pt[o + (long long)(k - 1) * S] * (pk0 - pk1);
      B[k + 1] = z;
      pk0 = pk1;
    }
  }
  __syncthreads();
  auto wind2 = [&](const double* u, const double* v, long long ok) {
    const double ua = (.25 * (u[ok] + u[ok + P]) + .125 * (u[ok - 1] + u[ok - 1 + P] + u[ok + 1] + u[ok + 1 + P]));
    const double va = (.25 * (v[ok] + v[ok + 1]) + .125 * (v[ok - P] + v[ok + 1 - P] + v[ok + P] + v[ok + 1 + P]));
    return make_double2(ua, va);
  };
  // the reverse of wind2 for the adjoints lu, lv of ua, va
  auto wind2_adj = [&](double* u, double* v, long long ok, double lu, double lv) {
    if (lu != 0.) {
      atomicAdd(u + ok, .25 * lu);
      atomicAdd(u + ok + P, .25 * lu);
      atomicAdd(u + ok - 1, .125 * lu);
      atomicAdd(u + ok - 1 + P, .125 * lu);
      atomicAdd(u + ok + 1, .125 * lu);
      atomicAdd(u + ok + 1 + P, .125 * lu);
    }
    if (lv != 0.) {
      atomicAdd(v + ok, .25 * lv);
      atomicAdd(v + ok + 1, .25 * lv);
      atomicAdd(v + ok - P, .125 * lv);
      atomicAdd(v + ok + 1 - P, .125 * lv);
      atomicAdd(v + ok + P, .125 * lv);
      atomicAdd(v + ok + 1 + P, .125 * lv);
    }
  };
  double pk0[N], pk1[N], lyk[N], tk0[N], tk1[N], Dk[N], ke[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k > L) continue;
    const long long ok = o + (long long)(k - 1) * S;
    pk0[q] = A[k];
    pk1[q] = A[k + 1];
    lyk[q] = (pk1[q] - pk0[q]) / atm_log(pk1[q] / pk0[q]);
    double2 w = wind2(ud, vd, ok);
    en[k] = CV_DRY * pt[ok] * lyk[q] + .5 * (B[k + 1] + B[k] + w.x * w.x + w.y * w.y);
    tk0[q] = T[k];
    tk1[q] = T[k + 1];
    const double tlyk = (tk1[q] - tk0[q]) / atm_log(tk1[q] / tk0[q]);
    w = wind2(urem, vrem, ok);
    Dk[q] = CV_DRY * tlyk + .5 * CP_DRY * (tk0[q] - tk1[q]);
    ke[q] = .5 * (w.x * w.x + w.y * w.y);
  }
  __syncthreads();
  auto var = [&](int k) { return en[k]; };
  adj_solve(L, sc, A, B, var, warp);
  for (int k = 1 + warp; k <= L; k += RMA_WARPS) {  // the layers' edges, for the remapped energy
    double cb, ct, btm, top;
    adj_edges(k, L, A, B, var, en[k], cb, ct, btm, top);
    LL[k] = btm;
    Lg[k] = top;
  }
  __syncthreads();
  for (int m = 1 + warp; m <= L; m += RMA_WARPS) {
    const double d0 = tpl(m), d1 = tpl(m + 1);
    int k = m;
    while (k > 1 && !(sc[k] >= d0)) --k;
    while (k <= L && sc[k + 1] >= d0) ++k;
    double acc = 0.;
    for (; k <= L && sc[k] > d1; ++k) {
      const double vk = en[k], btm = LL[k], top = Lg[k];
      pair_add_case(acc, btm, top, 6. * vk - 3. * (top + btm), vk, sc[k], sc[k + 1], d0, d1);
    }
    er[m] = acc;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k > L) continue;
    LL[k] = ke[q];
    Lg[k] = Dk[q];
  }
  __syncthreads();
  if (warp == 0) {
    // the recovered pt (:127-150) into er, then its reverse and the remapped
    // geopotential's: the adjoint of er into LL, of gz_remap(m+1) into Lg
    double gzr = gzs[o];
    for (int m = 1; m <= L; ++m) {
      const double ptr = (er[m] - gzr - LL[m]) / Lg[m];
      gzr = gzr + CP_DRY * ptr * (T[m] - T[m + 1]);
      er[m] = ptr;
    }
    double lgz = 0.;
#pragma unroll 4
    for (int m = L; m >= 1; --m) {
      const double rD = 1. / Lg[m];
      const double ln = (lam_pto[o + (long long)(m - 1) * S] + CP_DRY * (T[m] - T[m + 1]) * lgz) * rD;
      LL[m] = ln;
      Lg[m] = lgz;
      lgz -= ln;
    }
  }
  __syncthreads();
  double Z = 0.;  // of ps through the target levels
  const bool live = in && act[lane] && !bad[lane];
  // the adjoint of tpk(k) as one of ps: tpk = tpl**kappa, tpl = ak + bk (ps - ptop) (:57-71)
  auto to_ps = [&](int k, double tk) { return k <= L ? ra.bk[k - 1] * KAPPA * tk / tpl(k) : 0.; };
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int m = 1 + warp + q * RMA_WARPS;
    if (m > L) continue;
    const long long ok = o + (long long)(m - 1) * S;
    const double ptr = er[m], ln = LL[m], lgz = Lg[m], dtp = tk0[q] - tk1[q];
    const double ld = lam_dpo[ok];  // dp = tpl(k) - tpl(k+1) (:156-161)
    Z += ra.bk[m - 1] * ld - (m < L ? ra.bk[m] * ld : 0.);
    const double LD = -ptr * ln;
    // tlyk = (tk1 - tk0) / log(tk1 / tk0)
    const double tlyk = (Dk[q] - .5 * CP_DRY * dtp) * (1. / CV_DRY);
    const double y = CV_DRY * LD * tlyk / -dtp;
    const double l0 = CP_DRY * ptr * lgz + y * (-1. + tlyk / tk0[q]) + .5 * CP_DRY * LD;
    const double l1 = -CP_DRY * ptr * lgz + y * (1. - tlyk / tk1[q]) - .5 * CP_DRY * LD;
    Z += l0 * to_ps(m, tk0[q]) + l1 * to_ps(m + 1, tk1[q]);
    if (live) {
      const double2 w = wind2(urem, vrem, ok);
      wind2_adj(lam_ur, lam_vr, ok, -w.x * ln, -w.y * ln);
    }
    er[m] = ln;  // (the level's own value, read above)
    T[m] = tpl(m);
  }
  __syncthreads();
  auto ldst = [&](int k) { return er[k]; };
  auto td = [&](int k) { return k <= L ? T[k] : ra.ptop; };
  auto bk = [&](int k) { return k <= L ? ra.bk[k - 1] : 0.; };
  double Lv[N], Ls[N];
  remap_adj_core<LM>(L, sc, A, B, LL, Lg, T, part, var, td, ldst, bk, warp, Lv, Ls, Z);
  __syncthreads();
  Z = warps_sum(Z, part, warp, lane);
  // energy (:72-78), hydrostatic gz (:53-56), playkap (:46-52)
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k <= L) er[k] = Lv[q];
  }
  __syncthreads();
  if (warp == 0) {  // of gz(k+1): half of layer k's, all of those above
    double lz = 0.;
    for (int k = L; k >= 1; --k) {
      const double le = er[k];
      LL[k] = lz + .5 * le;
      lz += le;
    }
  }
  __syncthreads();
  double Lpt[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k > L) continue;
    const long long ok = o + (long long)(k - 1) * S;
    const double le = Lv[q], lz = LL[k], t = pt[ok], d = pk1[q] - pk0[q];
    const double ly = lyk[q], y = CV_DRY * t * le * ly / d;  // lyk = d / log(pk1 / pk0)
    Lpt[q] = CV_DRY * ly * le - CP_DRY * d * lz;
    Ls[q] += (y * (-1. + ly / pk0[q]) + CP_DRY * t * lz) * KAPPA * pk0[q] / sc[k];  // pk = plev**kappa
    T[k + 1] = k < L ? (y * (1. - ly / pk1[q]) - CP_DRY * t * lz) * KAPPA * pk1[q] / sc[k + 1] : 0.;
    if (live) {
      const double2 w = wind2(ud, vd, ok);
      wind2_adj(lam_ud, lam_vd, ok, w.x * le, w.y * le);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int k = 1 + warp + q * RMA_WARPS;
    if (k <= L) Lg[k] = Ls[q] + (k > 1 ? T[k] : Z);
  }
  __syncthreads();
  if (warp == 0) {  // plev(k) = plev(k+1) + dp(k)
    double acc = 0.;
    for (int k = 1; k <= L; ++k) {
      acc += Lg[k];
      Lg[k] = acc;
    }
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int k = 1 + warp + q * RMA_WARPS;
      if (k > L) continue;
      const long long ok = o + (long long)(k - 1) * S;
      lam_dp[ok] += Lg[k];
      lam_pt[ok] += Lpt[q];
    }
  } else if (in && act[lane] && warp == 0) {  // not monotone: the all-pairs reverse
    remap_energy_adj_at<LM>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_dp, lam_pt, lam_ud, lam_vd,
                              lam_ur, lam_vr, i, j);
  }
}
template <int LM>
__global__ void __launch_bounds__(RM_LANES * RMA_WARPS, 2) k_remap_energy_adj_split(
    Geom g, RemapArgs ra, const double* dp, const double* pt, const double* ud, const double* vd, const double* urem,
    const double* vrem, const double* gzs, const double* lam_dpo, const double* lam_pto, const double* lam_udo,
    const double* lam_vdo, double* lam_dp, double* lam_pt, double* lam_ud, double* lam_vd, double* lam_ur,
    double* lam_vr) {
  stream_order();
  remap_energy_adj_block<LM>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_udo, lam_vdo, lam_dp,
                             lam_pt, lam_ud, lam_vd, lam_ur, lam_vr);
}

}  // namespace atm
