// The vertical remap of a domain (src/mod_remap.f90:27-163): a block owns 32
// columns (lane = column), its warps share the levels, and the column arrays
// live in shared memory ([level][lane], no bank conflicts).
//
// A column's remap is a few chains whose order fixes the bits -- the pressure
// sums, the elimination and forward substitution of vertical_ppm, the
// geopotential -- between stages that are independent per level: the powers and
// logarithms, the quotients of the elimination, the limited edges, and above
// all the overlaps of each target layer with the source layers.  One warp runs
// the chains for its 32 columns, all warps share the rest.  With one thread a
// column (remap_winds_at, remap_energy_at of atm_kernels.cuh, which the
// persistent ensemble kernel keeps) the column arrays lay in local memory and
// every stage of every level waited for the one before.  Every value comes from
// the same operations in the same order as there.
#pragma once

#include "atm_kernels.cuh"

namespace atm {

constexpr int RM_WARPS = 8;  // 4 and 16 warps: 256x256x32 winds 0.28 and 0.33 ms against 0.22, energy 0.30 and 0.27 against 0.23
constexpr int RM_LANES = 32;

// bytes of a block's shared memory with n column arrays of levels 0 .. L+1
inline size_t remap_smem(int L, int n) { return (size_t)n * (L + 2) * RM_LANES * sizeof(double); }

// one column array: element k of the lane's column
struct ShCol {
  double* p;
  __device__ __forceinline__ double& operator[](int k) const { return p[k * RM_LANES]; }
};

// a value as the column array type E keeps it
template <typename E>
__device__ __forceinline__ double kept(double v) { return (double)(E)v; }

// vertical_ppm's elimination and forward substitution of one column by its
// thread (ppm_eliminate, PPMLayers): on entry A[k] = 3 (var(k) + alpha var(k-1))
// and B[k] = alpha(k) for k = 2..L; on return A[k], k = 1..L+1, the interface
// values and B[k+1] = gam(k), k = 1..L, each kept as E where the streaming
// remap stores it.
template <typename E>
__device__ __forceinline__ void remap_solve(int L, ShCol sc, ShCol A, ShCol B, double v1, double v2, double vL1,
                                            double vL) {
  const double a0 = (sc[L] - sc[L - 1]) / (sc[L + 1] - sc[L]);
  double beta = a0 * (.5 + a0);
  double lv = (2. * a0 * (1. + a0) * vL + vL1) / beta;
  A[L + 1] = kept<E>(lv);
  double g = (1. + a0 * (1.5 + a0)) / beta;
  B[L + 1] = kept<E>(g);
  double alpha = 0.;
  double an = B[L], nn = A[L];
  for (int k = L; k >= 2; --k) {
    alpha = an;
    const double n = nn;
    if (k > 2) {
      an = B[k - 1];
      nn = A[k - 1];
    }
    beta = 2. + 2. * alpha - g;
    lv = (n - lv) / beta;
    A[k] = kept<E>(lv);
    g = alpha / beta;
    B[k] = kept<E>(g);
  }
  beta = 1. + alpha * (1.5 + alpha);
  double f = kept<E>((2. * alpha * (1. + alpha) * v1 + v2 - beta * lv) / (alpha * (.5 + alpha) - beta * g));
  A[1] = f;
  for (int k = 1; k <= L; ++k) {
    f = A[k + 1] - B[k + 1] * f;
    A[k + 1] = f;
  }
}

// the limited value of interface j (between layers j-1 and j), 2 <= j <= L
template <typename FV>
__device__ __forceinline__ double remap_interface(int j, int L, ShCol A, ShCol B, const FV& var) {
  double c = A[j];
  const double vk = var(j - 1), vk1 = var(j);
  const double lo = mn(vk, vk1), hi = mx(vk, vk1);
  if (j == L || j == 2) {
    c = mn(c, mx(vk1, vk));
    c = mx(c, mn(vk1, vk));
  }
  if (j >= 3) {
    if (j == L || B[j + 2] * B[j] > 0) {
      c = mn(c, hi);
      c = mx(c, lo);
    } else if (B[j + 2] > 0) {
      c = mx(c, lo);
    } else {
      c = mn(c, hi);
    }
  }
  return c;
}

// the edges of layer k from the limited interface values A
template <typename FV>
__device__ __forceinline__ void remap_edges(int k, ShCol A, ShCol B, const FV& var, double& btm, double& top) {
  btm = A[k];
  top = A[k + 1];
  if (k >= 3) {
    const double vk = var(k), gk1 = B[k];
    double pmp1 = vk - 2. * gk1;
    double lac1 = pmp1 + 1.5 * B[k - 1];
    top = mn(mx(top, mn3(vk, pmp1, lac1)), mx3(vk, pmp1, lac1));
    pmp1 = vk + 2. * B[k + 1];
    lac1 = pmp1 - 1.5 * gk1;
    btm = mn(mx(btm, mn3(vk, pmp1, lac1)), mx3(vk, pmp1, lac1));
  }
}

// From the source coordinate sc and the variable var(k): the edges of every
// layer, A[k] = bottom, B[k] = top.  All threads of the block.
template <int LM, typename E, typename FV>
__device__ __forceinline__ void remap_ppm(int L, ShCol sc, ShCol A, ShCol B, const FV& var, int warp) {
  for (int k = 2 + warp; k <= L; k += RM_WARPS) {
    const double c1 = sc[k];
    const double alpha = (sc[k + 1] - c1) / (c1 - sc[k - 1]);
    A[k] = 3. * (var(k) + alpha * var(k - 1));
    B[k] = alpha;
  }
  __syncthreads();
  if (warp == 0) remap_solve<E>(L, sc, A, B, var(1), var(2), var(L - 1), var(L));
  __syncthreads();
  for (int j = 2 + warp; j <= L; j += RM_WARPS) A[j] = remap_interface(j, L, A, B, var);
  __syncthreads();
  constexpr int N = (LM + RM_WARPS - 1) / RM_WARPS;
  double b[N], t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RM_WARPS;
    if (k <= L) remap_edges(k, A, B, var, b[i], t[i]);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int k = 1 + warp + i * RM_WARPS;
    if (k <= L) {
      A[k] = b[i];
      B[k] = t[i];
    }
  }
  __syncthreads();
}

// The remapped value of target layer m between its interfaces d0 >= d1: the
// overlapping source layers in ascending order (both coordinates descend).
// tr, when non-null, receives the layer's trace entry (remap_column).
template <typename FV>
__device__ __forceinline__ double remap_layer(int m, int L, ShCol sc, ShCol A, ShCol B, const FV& var, double d0,
                                              double d1, int* tr) {
  int k0 = m;  // the first source layer whose top lies above d0, looked for from m
  while (k0 > 1 && !(sc[k0] >= d0)) --k0;
  while (k0 <= L && sc[k0 + 1] >= d0) ++k0;
  double acc = 0.;
  int first = -1, last = -1, w0 = -1, w1 = -1, cnt = 0;
  for (int k = k0; k <= L; ++k) {
    const double sk = sc[k];
    if (!(sk > d1)) break;
    const double btm = A[k], top = B[k], vk = var(k);
    const int which = pair_add_case(acc, btm, top, 6. * vk - 3. * (top + btm), vk, sk, sc[k + 1], d0, d1);
    if (first < 0) {
      first = k;
      w0 = which;
    }
    last = k;
    w1 = which;
    ++cnt;
  }
  if (tr) {
    tr[0] = first;
    tr[1] = last;
    tr[2] = w0;
    tr[3] = w1;
    tr[4] = cnt;
  }
  return acc;
}

// Winds on the cell faces over [isd-1, ied+1]^2 (remap_winds_at): blockIdx.y the
// direction.  Three column arrays: the coordinate, and the elimination's values
// and coefficients, later the edges.  E as in remap_winds_at.
template <typename T, int LM, typename E = double>
__global__ void __launch_bounds__(RM_LANES * RM_WARPS, 4) k_remap_winds_split(
    Geom g, RemapArgs ra, const T* dp, const T* ud, const T* vd,
    T* urem, T* vrem, int* trace, Status* st) {
  stream_order();
  extern __shared__ double rm_sm[];
  __shared__ double ps[4][RM_LANES];
  __shared__ int bad[RM_LANES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dir = blockIdx.y;
  const int w = g.nx + 2, h = g.ny + 2, L = g.L;
  const int col = blockIdx.x * RM_LANES + lane;
  const bool in = col < w * h;
  const int i = -1 + (in ? col % w : 0), j = -1 + (in ? col / w : 0);
  const long long S = g.S;
  const T* f = dir == 0 ? ud : vd;
  T* r = dir == 0 ? urem : vrem;
  const long long oa = g.at(i, j);
  const ShCol sc{rm_sm + lane}, A{rm_sm + (L + 2) * RM_LANES + lane}, B{rm_sm + 2 * (L + 2) * RM_LANES + lane};
  if (warp == 0) {
    // source coordinate: running sums from the model top of the face's four
    // columns (src/mod_remap.f90:42-44,84-85)
    const long long ob = dir == 0 ? g.at(i, j - 1) : g.at(i - 1, j);
    const long long oc = dir == 0 ? g.at(i, j + 1) : g.at(i + 1, j);
    const long long od = dir == 0 ? g.at(i, j - 2) : g.at(i - 2, j);
    constexpr int NB = 4;  // levels loaded ahead
    T na[NB], nb[NB], nc[NB], nd[NB];
    auto fetch = [&](int u, int k) {
      if (k < 1) return;
      const long long kk = (long long)(k - 1) * S;
      na[u] = dp[oa + kk];
      nb[u] = dp[ob + kk];
      nc[u] = dp[oc + kk];
      nd[u] = dp[od + kk];
    };
#pragma unroll
    for (int u = 0; u < NB; ++u) fetch(u, L - u);
    double pa = ra.ptop, pb = ra.ptop, pc = ra.ptop, pd = ra.ptop;
    double prev = C7_12 * (pa + pb) - C1_12 * (pc + pd);
    sc[L + 1] = prev;
    bool mono = true;
    for (int k0 = L; k0 >= 1; k0 -= NB) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int k = k0 - u;
        if (k < 1) break;
        pa = pa + (double)na[u];
        pb = pb + (double)nb[u];
        pc = pc + (double)nc[u];
        pd = pd + (double)nd[u];
        fetch(u, k - NB);
        const double c = C7_12 * (pa + pb) - C1_12 * (pc + pd);
        mono = mono && (prev <= c);
        sc[k] = c;
        prev = c;
      }
    }
    ps[0][lane] = pa;
    ps[1][lane] = pb;
    ps[2][lane] = pc;
    ps[3][lane] = pd;
    bad[lane] = mono ? 0 : 1;
  }
  __syncthreads();
  const double pa = ps[0][lane], pb = ps[1][lane], pc = ps[2][lane], pd = ps[3][lane];
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
  auto var = [&](int k) { return (double)f[oa + (long long)(k - 1) * S]; };
  remap_ppm<LM, E>(L, sc, A, B, var, warp);
  int* tr = nullptr;
  if (trace && in) tr = trace + ((long long)dir * h * w + (long long)(j + 1) * w + (i + 1)) * L * 5;  // [3][ny+2][nx+2][L][5]
  bool mono = true;
  for (int m = 1 + warp; m <= L; m += RM_WARPS) {
    const double d0 = dc(m), d1 = dc(m + 1);
    mono = mono && (d1 <= d0);
    const double v = remap_layer(m, L, sc, A, B, var, d0, d1, tr ? tr + (m - 1) * 5 : nullptr);
    if (in) r[oa + (long long)(m - 1) * S] = T(v);
  }
  if (!mono) bad[lane] = 1;
  __syncthreads();
  // coordinates that are not monotone: the reference's all-pairs search instead
  if (warp == 0 && in && bad[lane]) remap_winds_full<T, LM>(g, ra, dp, f, r, tr, st, i, j, dir);
}

// Energy remap and potential-temperature recovery on the interior
// (remap_energy_at).  Four column arrays, in turn: levels; pkap, the
// elimination's values, bottom edges, the recovery's denominators; geopotential,
// coefficients, top edges, pkap steps; energy, remapped energy.
template <typename T, int LM, typename PW = PortablePow>
__global__ void __launch_bounds__(RM_LANES * RM_WARPS, 3) k_remap_energy_split(
    Geom g, RemapArgs ra, const T* dp, const T* pt, const T* ud,
    const T* vd, const T* urem, const T* vrem, const double* gzs,
    T* dpo, T* pto, T* udo, T* vdo, int* trace, Status* st) {
  stream_order();
  extern __shared__ double rm_sm[];
  __shared__ int bad[RM_LANES];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int L = g.L, P = g.P;
  const int col = blockIdx.x * RM_LANES + lane;
  const bool in = col < g.nx * g.ny;
  const int i = in ? col % g.nx : 0, j = in ? col / g.nx : 0;
  const long long S = g.S, o = g.at(i, j);
  const ShCol sc{rm_sm + lane}, A{rm_sm + (L + 2) * RM_LANES + lane}, B{rm_sm + 2 * (L + 2) * RM_LANES + lane},
      en{rm_sm + 3 * (L + 2) * RM_LANES + lane};
  constexpr int NB = 8;
  if (warp == 0) {  // levels (src/mod_remap.f90:42-44)
    T dn[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) dn[u] = L - u >= 1 ? dp[o + (long long)(L - u - 1) * S] : T(0);
    double pl = ra.ptop;
    sc[L + 1] = pl;
    bool mono = true;
    for (int k0 = L; k0 >= 1; k0 -= NB) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int k = k0 - u;
        if (k < 1) break;
        const double pn = pl + (double)dn[u];
        if (k - NB >= 1) dn[u] = dp[o + (long long)(k - NB - 1) * S];
        mono = mono && (pl <= pn);
        sc[k] = pn;
        pl = pn;
      }
    }
    bad[lane] = mono ? 0 : 1;
  }
  __syncthreads();
  const double ps = sc[1];
  for (int k = 1 + warp; k <= L; k += RM_WARPS) A[k] = PW::kappa(sc[k]);  // pkap (:46)
  if (warp == RM_WARPS - 1) A[L + 1] = ra.pk_top;
  auto tpl = [&](int k) { return k <= L ? ra.ak[k - 1] + ra.bk[k - 1] * (ps - ra.ptop) : ra.ptop; };  // target levels (:57-59)
  {
    bool mono = true;
    for (int k = 1 + warp; k <= L; k += RM_WARPS) mono = mono && (tpl(k + 1) <= tpl(k));
    if (!mono) bad[lane] = 1;
  }
  __syncthreads();
  if (warp == 0) {  // gz (:70-75)
    T pn[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) pn[u] = u < L ? pt[o + (long long)u * S] : T(0);
    double z = gzs[o], pk0 = A[1];
    B[1] = z;
    for (int k0 = 1; k0 <= L; k0 += NB) {
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int k = k0 + u;
        if (k > L) break;
        const double pk1 = A[k + 1];
        z = z + CP_DRY * (double)pn[u] * (pk0 - pk1);
        if (k + NB <= L) pn[u] = pt[o + (long long)(k + NB - 1) * S];
        B[k + 1] = z;
        pk0 = pk1;
      }
    }
  }
  __syncthreads();
  // kinetic energy of the A-grid winds of face winds u, v (:116-121)
  auto wind2 = [&](const T* u, const T* v, long long ok) {
    const double ua = (.25 * ((double)u[ok] + (double)u[ok + P]) +
                       .125 * ((double)u[ok - 1] + (double)u[ok - 1 + P] + (double)u[ok + 1] + (double)u[ok + 1 + P]));
    const double va = (.25 * ((double)v[ok] + (double)v[ok + 1]) +
                       .125 * ((double)v[ok - P] + (double)v[ok + 1 - P] + (double)v[ok + P] + (double)v[ok + 1 + P]));
    return make_double2(ua, va);
  };
  for (int k = 1 + warp; k <= L; k += RM_WARPS) {  // total energy (:111-125)
    const long long ok = o + (long long)(k - 1) * S;
    const double pk0 = A[k], pk1 = A[k + 1];
    const double plog = PW::log(pk1 / pk0);
    const double lyk = (pk1 - pk0) / plog;
    const double2 w = wind2(ud, vd, ok);
    en[k] = CV_DRY * (double)pt[ok] * lyk + .5 * (B[k + 1] + B[k] + w.x * w.x + w.y * w.y);
  }
  __syncthreads();
  auto var = [&](int k) { return en[k]; };
  remap_ppm<LM, double>(L, sc, A, B, var, warp);
  int* tr = nullptr;
  if (trace && in) {
    const int w = g.nx + 2, h = g.ny + 2;
    tr = trace + ((long long)2 * h * w + (long long)(j + 1) * w + (i + 1)) * L * 5;
  }
  const bool full = bad[lane] != 0;  // not monotone: the reference's all-pairs search
  constexpr int N = (LM + RM_WARPS - 1) / RM_WARPS;
  double er[N] = {};
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int m = 1 + warp + q * RM_WARPS;
    if (m <= L && !full) er[q] = remap_layer(m, L, sc, A, B, var, tpl(m), tpl(m + 1), tr ? tr + (m - 1) * 5 : nullptr);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int m = 1 + warp + q * RM_WARPS;
    if (m <= L) {
      en[m] = er[q];
      sc[m] = PW::kappa(tpl(m));
    }
  }
  if (warp == RM_WARPS - 1) sc[L + 1] = ra.pk_top;
  __syncthreads();
  // remapped energy -> potential temperature (:127-161): what each level's
  // recovery needs beside the geopotential below it
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int m = 1 + warp + q * RM_WARPS;
    if (m <= L) {
      const double k0 = sc[m], k1 = sc[m + 1];
      const double plog = PW::log(k1 / k0);
      const double tlyk = (k1 - k0) / plog;
      A[m] = CV_DRY * tlyk + .5 * CP_DRY * (k0 - k1);
      B[m] = k0 - k1;
      const double2 w = wind2(urem, vrem, o + (long long)(m - 1) * S);
      er[q] = .5 * (w.x * w.x + w.y * w.y);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; ++q) {
    const int m = 1 + warp + q * RM_WARPS;
    if (m <= L) sc[m] = er[q];
  }
  __syncthreads();
  if (warp == 0) {
    double gzr = gzs[o];
    for (int m = 1; m <= L; ++m) {
      const double ptr = (en[m] - gzr - sc[m]) / A[m];
      gzr = gzr + CP_DRY * ptr * B[m];
      en[m] = ptr;
    }
  }
  __syncthreads();
  if (full) {
    if (warp == 0 && in)
      remap_energy_full<T, LM, PW>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, dpo, pto, udo, vdo, tr, st, i, j);
    return;
  }
  if (!in) return;
  bool nonfinite = false;
  for (int m = 1 + warp; m <= L; m += RM_WARPS) {
    const long long ok = o + (long long)(m - 1) * S;
    const T dpn = T(tpl(m) - tpl(m + 1)), tn = T(en[m]), un = urem[ok], vn = vrem[ok];
    dpo[ok] = dpn;
    pto[ok] = tn;
    udo[ok] = un;
    vdo[ok] = vn;
    nonfinite = nonfinite || !(finite_(dpn) && finite_(tn) && finite_(un) && finite_(vn));
  }
  flag_nonfinite(&st->nonfinite_remap, nonfinite);
}

// One thread a column, for domains that fill the GPU with them: 16 blocks of 64
// threads per SM (a 64-register budget, the column arrays in local memory
// either way), as more columns in flight hide more of the local-memory latency
// (1024x1024x64, winds / energy: 4.09 / 4.34 ms, 4.51 / 5.00 at 12 blocks, 4.53 /
// 4.39 at 20).
template <typename T, int LM, typename E = double>
__global__ void __launch_bounds__(64, 16) k_remap_winds(Geom g, RemapArgs ra, const T* dp,
                                                        const T* ud, const T* vd,
                                                        T* urem, T* vrem, int* trace,
                                                        Status* st) {
  stream_order();
  remap_winds_at<T, LM, E>(g, ra, dp, ud, vd, urem, vrem, trace, st, blockIdx.x * blockDim.x + threadIdx.x,
                           blockIdx.y);
}
template <typename T, int LM, typename PW = PortablePow>
__global__ void __launch_bounds__(64, 16) k_remap_energy(Geom g, RemapArgs ra, const T* dp,
                                                         const T* pt, const T* ud,
                                                         const T* vd, const T* urem,
                                                         const T* vrem, const double* gzs,
                                                         T* dpo, T* pto, T* udo,
                                                         T* vdo, int* trace, Status* st) {
  stream_order();
  remap_energy_at<T, LM, PW>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, dpo, pto, udo, vdo, trace, st,
                             blockIdx.x * blockDim.x + threadIdx.x);
}

// Columns up to which the split kernels are the faster ones.  Their blocks wait
// for one warp's chains, which other blocks hide only while few columns wait: so
// the limit is a number of columns a block that an SM holds (by the column
// arrays' shared memory, at most `most` by registers), less where the layers leave
// some of the block's warps without work.  Measured on B200, FP64 form (us, split
// against one thread a column; columns in thousands), winds:
//   3 layers 4.1 11/12, 9.2 14/12; 8 layers 9.2 19/23, 16 21/22, 26 27/23; 20 layers 16 38/47, 26 52/53;
//   32 and 64 (four blocks) 26 74/89, 157/191, 37 103/100, 223/205;
//   80 and 96 (three) 16 174/222, 220/267, 26 248/242, 312/292; 112 and 128 (two) 9.2 210/284, 250/329, 16 316/317, 375/365
// and energy:
//   3 layers 9.2 15/19, 16 23/19; 8 layers 26 31/37, 37 41/39; 20 layers 37 86/100, 50 118/114;
//   32 and 64 (three blocks) 50 171/193, 372/402, 66 213/211, 467/436;
//   80 and 96 (two) 26 368/450, 458/551, 37 500/476, 619/580; 112 and 128 (one) 16 553/608, 633/704, 26 817/650, 952/753
// With a limit that did not know the layers, a remap of 256x256x128 took 2.70 ms, of
// 272x272x96 1.61; a thread a column 1.82 and 1.41.
inline int remap_blocks(int L, int n, int most) {
  const int b = (int)(228 * 1024 / (remap_smem(L, n) + 2304));  // the kernels' own variables and the block's reserve
  return b < most ? b : most;
}
inline long long remap_winds_few(int L) { return 148LL * 56 * remap_blocks(L, 3, 4) * (L < 32 ? L : 32) / 32; }
// (more than two blocks of the 65- to 128-layer instance gain nothing: 65 layers 26
// 240/358, 50 472/408; with three, columns that share the GPU with other kernels do
// better in the split form also beyond the tie, so the line lies at its far end: eight
// ensemble members 10.89 ms with it, 11.02 at 53000 columns, a gradient of 301x203x40
// 30.13 and 30.34)
inline long long remap_energy_few(int L) {
  const int b = remap_blocks(L, 4, L > 64 ? 2 : 3);
  return 148LL * (b > 2 ? 512 : 120 * b) * (L < 28 ? L + 8 : 36) / 36;
}

// Shared memory above the default limit, which the kernel's own variables count
// against too: always what the kernel's largest layer count takes, so that
// launches of different layer counts on several threads set the same value.
template <typename K>
inline cudaError_t remap_smem_attr(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <typename T, int LM, typename E = double>
cudaError_t launch_remap_winds(const Geom& g, const RemapArgs& ra, const T* dp, const T* ud, const T* vd, T* urem,
                               T* vrem, int* trace, Status* st, cudaStream_t s) {
  const int n = (g.nx + 2) * (g.ny + 2);
  if (n > remap_winds_few(g.L)) {
    launch(k_remap_winds<T, LM, E>, dim3((n + 63) / 64, 2), 64, 0, s, g, ra, dp, ud, vd, urem, vrem, trace, st);
    return cudaGetLastError();
  }
  const size_t sm = remap_smem(g.L, 3);
  const cudaError_t e = remap_smem_attr(k_remap_winds_split<T, LM, E>, remap_smem(LM, 3));
  if (e != cudaSuccess) return e;
  launch(k_remap_winds_split<T, LM, E>, dim3((n + RM_LANES - 1) / RM_LANES, 2), RM_LANES * RM_WARPS, sm, s, 
      g, ra, dp, ud, vd, urem, vrem, trace, st);
  return cudaGetLastError();
}
template <typename T, int LM, typename PW = PortablePow>
cudaError_t launch_remap_energy(const Geom& g, const RemapArgs& ra, const T* dp, const T* pt, const T* ud, const T* vd,
                                const T* urem, const T* vrem, const double* gzs, T* dpo, T* pto, T* udo, T* vdo,
                                int* trace, Status* st, cudaStream_t s) {
  const int n = g.nx * g.ny;
  if (n > remap_energy_few(g.L)) {
    launch(k_remap_energy<T, LM, PW>, (n + 63) / 64, 64, 0, s, g, ra, dp, pt, ud, vd, urem, vrem, gzs, dpo, pto, udo, vdo,
                                                           trace, st);
    return cudaGetLastError();
  }
  const size_t sm = remap_smem(g.L, 4);
  const cudaError_t e = remap_smem_attr(k_remap_energy_split<T, LM, PW>, remap_smem(LM, 4));
  if (e != cudaSuccess) return e;
  launch(k_remap_energy_split<T, LM, PW>, (n + RM_LANES - 1) / RM_LANES, RM_LANES * RM_WARPS, sm, s, 
      g, ra, dp, pt, ud, vd, urem, vrem, gzs, dpo, pto, udo, vdo, trace, st);
  return cudaGetLastError();
}

}  // namespace atm
