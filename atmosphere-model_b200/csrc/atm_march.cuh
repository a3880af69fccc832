// Column-marching sweep kernels of the B200 dynamical core, both forms.
//
// A warp owns a strip of one layer: 32 consecutive x columns (lane = column)
// of which the middle 26 are outputs (3 halo columns on each side feed the
// PPM stencils), and a number of output rows that it walks through in
// ascending y.  Each lane keeps the y-direction stencil values of its column
// (the last few rows of every stage) in registers, so that every stage of the
// reference's layer loop is evaluated once per cell instead of once per
// cell of every overlapping tile halo; x-direction neighbours come from the
// neighbouring lanes by warp shuffles.  The warps of a block are independent
// (no block-wide barrier); each row's inputs are copied into the warp's part of
// shared memory two rows ahead (FeedRing).
//
// The sweeps are bound by the latency of their FP64 (FP32) chains at the warps
// that the registers leave, then by instruction issue (HBM traffic is the
// fields read and written once, 0.5 ms of a kernel at 1024x1024x64), so the
// formulas are arranged for the fewest instructions that give the reference's
// bits: a difference of two neighbours is formed once and serves the slopes of
// both cells and the two edges between them (YLine, xline_flux), each cell's
// edges are formed and limited once, exact products are fused, and the
// division by three needs no branch.  Measured on B200 at 1024x1024x64 (ms a
// launch, C mass / C momentum / D mass / D momentum; first: FP64 sweeps on 32 x
// 4-8 shared-memory tiles, FP32 marching with per-flux edges; then marching
// with each row loaded a row ahead into registers; now):
//   FP64  4.24 / 4.03 / 4.58 / 4.92  ->  1.93 / 2.61 / 2.38 / 2.69  ->  1.73 / 2.17 / 2.05 / 2.39
//   FP32  1.63 / 2.02 / 1.70 / 2.29  ->  1.23 / 1.65 / 1.27 / 1.60  ->  1.16 / 1.37 / 1.24 / 1.56
//
// Every value is the reference's expression (src/mod_sw_dyn.f90) up to the
// sign of a zero; FP64 instances are bit-identical to the FP64 restatement.
// The persistent ensemble kernel runs the same strip functions with plain
// loads (RO = false), as it reads fields that it wrote earlier in the same
// launch.
#pragma once

#include <type_traits>

#include "atm_kernels.cuh"

namespace atm {

constexpr int MW = 32;              // lanes (columns) of a strip
constexpr int MXH = 3;              // halo columns on each side
constexpr int MOUT = MW - 2 * MXH;  // output columns of a strip
constexpr int MWARPS = 4;           // independent strips (warps) per block at most (atm_strips.h)

// Register budget (blocks of four warps per SM) and rows per loop body of each
// marching kernel.  The row windows shift by one register a row; unrolling by
// n rows does n shifts at once (a window of w doubles costs 2w/n moves a row).
// Measured on B200 at 1024x1024x64 (ms, C mass / C momentum / D mass / D
// momentum), rows fed through shared memory:
//   FP64, 3 blocks (168 registers), 1 / 2 / 3 / 4 rows: 1.93 2.18 2.26 2.42 /
//     1.78 2.33 2.32 2.44 / 1.77 2.31 2.25 2.43 / 1.75 2.43 2.20 2.52;
//     4 blocks (128 registers) with the windows of the inputs read back from
//     shared memory instead of kept in registers, 1 / 2 rows: 1.91 2.35 2.13
//     2.66 / 1.84 2.65 2.17 3.18: taken for D mass
//   FP32, 4 blocks (128 registers), 1 / 2 / 3 / 4 rows: 1.22 1.47 1.34 1.62 /
//     1.18 1.41 1.30 1.57 / 1.22 1.45 1.30 1.59 / 1.15 1.39 1.33 1.63
enum { MK_CMASS, MK_DMASS, MK_CMOM, MK_DMOM };
template <typename T, int K>
struct MarchL {
  static constexpr bool F32 = std::is_same_v<T, float>;
  static constexpr int min_blocks = F32 || K == MK_DMASS ? 4 : 3;
  static constexpr int unroll = F32 ? (K == MK_DMOM ? 2 : K == MK_DMASS ? 3 : 4) : K == MK_CMASS ? 4 : 1;
};

template <typename T>
__device__ __forceinline__ T shfl_dn(T v, int d) {
  return __shfl_down_sync(0xffffffffu, v, d);
}
template <typename T>
__device__ __forceinline__ T shfl_up(T v, int d) {
  return __shfl_up_sync(0xffffffffu, v, d);
}

// a * b + c.  The mixed form's translation unit is compiled without
// contraction (so that every kernel inlining these functions rounds them
// alike), and its FP32 arithmetic asks for its fused operations here; in
// FP64 the unfused expression, whose value equals the formula as written
// (an IEEE sum does not depend on the order of its two operands).
__device__ __forceinline__ float fmadd(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmadd(double a, double b, double c) { return a * b + c; }

// a * b + c where a * b is exact (a a power of two): one fused operation in
// either type, with the value of the two separate ones.
__device__ __forceinline__ float fmx(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmx(double a, double b, double c) { return __fma_rn(a, b, c); }

// v with its sign flipped where s is negative
__device__ __forceinline__ double xsign(double v, double s) {
  return __hiloint2double(__double2hiint(v) ^ (__double2hiint(s) & 0x80000000), __double2loint(v));
}
__device__ __forceinline__ float xsign(float v, float s) {
  return __int_as_float(__float_as_int(v) ^ (__float_as_int(s) & 0x80000000));
}
// min and max that return NaN where an argument is NaN (one instruction in
// FP32; in FP64 the compare-and-select of mn and mx, which keeps a NaN first
// argument)
__device__ __forceinline__ float mn_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float mx_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ double mn_nan(double a, double b) { return mn(a, b); }
__device__ __forceinline__ double mx_nan(double a, double b) { return mx(a, b); }

// Monotone slope of a cell (src/mod_sw_dyn.f90:870-875) from the differences
// dm = q(0) - q(-1), dp = q(+1) - q(0) and dqi = (q(+1) - q(-1)) / 4.
// The reference bounds |dqi| by dmax = max(q(+1), q(0), q(-1)) - q(0) and dmin =
// q(0) - min(...): where dm and dp agree in sign these two are |dm| and |dp|
// (the same rounded differences), elsewhere one of them is zero.  So the
// magnitude is the least of |dqi| and of dm, dp counted positive along dqi,
// and not below zero: the same value from half the compares and selects, and
// each difference serves two cells and the edges between them.
template <typename T>
__device__ __forceinline__ T slope_d(T dm, T dp, T dqi) {
  const T m = mn_nan(mn_nan(fab(dqi), xsign(dm, dqi)), xsign(dp, dqi));
  return cpsign(mx_nan(m, T(0)), dqi);
}

// x / 3 in FP64, equal to the IEEE quotient for every x, without a branch:
// the corrected quotient of div_const, whose remainder e is exact (a multiple
// of the smallest subnormal, and x / 3 is never near half an ulp from two
// doubles, so the correction rounds rightly among subnormals too); a zero
// remainder (zeros among them) and a NaN one (infinities) keep q.
__device__ __forceinline__ double third(double x) {
  constexpr double r = 1.0 / 3;
  const double q = x * r;
  const double e = __fma_rn(-q, 3.0, x);
  return fabs(e) > 0. ? __fma_rn(e, r, q) : q;
}
__device__ __forceinline__ float third(float x) { return div_const<3>(x); }

// The constrained limiter (src/mod_sw_dyn.f90:878-911) of a cell's raw edge anomalies with
// its raw slope dqi.
__device__ __forceinline__ double lim_min(double lim, double e) { return mn(lim, fabs(e)); }
__device__ __forceinline__ float lim_min(float lim, float e) { return fminf(lim, fabsf(e)); }
template <typename T>
__device__ __forceinline__ void limit_con(T dqi, T& eL, T& eR) {
  const T lim = T(2) * fab(dqi);
  eL = -cpsign(lim_min(lim, eL), dqi);
  eR = cpsign(lim_min(lim, eR), dqi);
}
// The same with the positivity filter of PPM_NONNEGATIVE.  Both edges are at
// most 2 |dqi| in magnitude, so where q0 > 6 |dqi| neither floor at -q0 holds
// and the parabola's minimum, above q0 - 2 |dqi|, is positive: nothing
// changes and the filter (and its division) is skipped.
template <typename T>
__device__ __forceinline__ void limit_nn(T q0, T dqi, T& eL, T& eR) {
  limit_con(dqi, eL, eR);
  if (q0 > T(6) * fab(dqi)) return;
  eL = mx(eL, -q0);
  eR = mx(eR, -q0);
  const T a = eR - eL;
  const T b = T(-3) * (eR + eL);
  if ((fab(a) < -b) && (q0 + a * a / (T(4) * b) + div_const<12>(b) < T(0))) {
    if (eL * eR > T(0)) {
      eL = T(0);
      eR = T(0);
    } else if (eL > eR) {
      eL = T(2) * fab(eR);
    } else {
      eR = T(2) * fab(eL);
    }
  }
}

// Upwind flux with Courant number c at the interface between cells m and 0
// from their values and edges (src/mod_sw_dyn.f90:781-868).
template <typename T>
__device__ __forceinline__ T flux_e(T c, T qm, T eLm, T eRm, T q0, T eL0, T eR0) {
  const bool pos = c > T(0);
  const T sa = fab(c);
  const T k1 = fmx(T(-2), sa, T(1)) * (T(1) - sa);
  const T k2 = sa * (sa - T(1));
  return fmadd(k2, pos ? eLm : eR0, fmadd(k1, pos ? eRm : eL0, pos ? qm : q0));
}
// PPM_CONSTRAINED: the upwind value itself where both cells' edges are
// one-sided (flat_e of each)
template <typename T>
__device__ __forceinline__ bool flat_e(T eL, T eR) {
  return T(3) * fab(eL + eR) > fab(eL - eR);
}
template <typename T>
__device__ __forceinline__ T flux_con_e(T c, T qm, T eLm, T eRm, T q0, T eL0, T eR0, bool flat) {
  const T f = flux_e(c, qm, eLm, eRm, q0, eL0, eR0);
  return flat ? ((c > T(0)) ? qm : q0) : f;
}

// t = .5 (q + den (q - rA (f1 - f0))), the piecewise-constant inner sweep
template <typename T>
__device__ __forceinline__ T inner_e(T q, T f0, T f1, T den, T rA) {
  return T(.5) * fmadd(den, fmadd(-rA, f1 - f0, q), q);
}

// A line of one quantity along y, fed a value a row: the windows of its last
// rows and the edges of its cells, formed once a cell.  After push() of row r:
// q0 .. q3 are rows r .. r-3, (L2, R2) and (L3, R3) the final edges of cells
// r-2 and r-3, so that flux() is the flux at the interface between them.
template <typename T, int V>
struct YLine {
  T q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  T dif = 0, mono = 0, dqi = 0, rawL = 0;  // q0 - q1; slope, dqi and raw lower edge of cell r-1
  T L2 = 0, R2 = 0, L3 = 0, R3 = 0;
  bool flat2 = false, flat3 = false;
  __device__ __forceinline__ void push(T v) {
    const T dn = v - q0;
    const T dq = (v - q1) * T(0.25);
    const T m = slope_d(dif, dn, dq);       // cell r-1
    const T h = third(mono - m);            // between cells r-2 and r-1
    L3 = L2;
    R3 = R2;
    L2 = rawL;
    R2 = fmx(T(.5), dif, h);
    rawL = fmx(T(-.5), dif, h);
    if (V == PPM_CON) {
      limit_con(dqi, L2, R2);
      flat3 = flat2;
      flat2 = flat_e(L2, R2);
    }
    if (V == PPM_NN) limit_nn(q1, dqi, L2, R2);
    q3 = q2; q2 = q1; q1 = q0; q0 = v;
    dif = dn;
    mono = m;
    dqi = dq;
  }
  __device__ __forceinline__ T flux(T c) const {
    if (V == PPM_CON) return flux_con_e(c, q3, L3, R3, q2, L2, R2, flat2 && flat3);
    return flux_e(c, q3, L3, R3, q2, L2, R2);
  }
};

// A line along x, one cell a lane: the flux at the interface between the
// lane's cell and the cell of the lane below.
template <typename T, int V>
__device__ __forceinline__ T xline_flux(T q, T c) {
  const T qL = shfl_up(q, 1), qR = shfl_dn(q, 1);
  const T dm = q - qL;
  const T dqi = (qR - qL) * T(0.25);
  const T m = slope_d(dm, qR - q, dqi);
  const T h = third(shfl_up(m, 1) - m);
  const T rI = fmx(T(.5), dm, h);  // raw upper edge of the cell below
  T eL = fmx(T(-.5), dm, h);       // raw lower edge of the cell
  T eR = shfl_dn(rI, 1);
  if (V == PPM_UNC) return flux_e(c, qL, shfl_up(eL, 1), rI, q, eL, eR);
  if (V == PPM_NN) {
    limit_nn(q, dqi, eL, eR);
    return flux_e(c, qL, shfl_up(eL, 1), shfl_up(eR, 1), q, eL, eR);
  }
  limit_con(dqi, eL, eR);
  const unsigned fl = __ballot_sync(0xffffffffu, flat_e(eL, eR));
  const int lane = threadIdx.x & (MW - 1);
  const bool flat = lane > 0 && ((fl >> (lane - 1)) & 3u) == 3u;
  return flux_con_e(c, qL, shfl_up(eL, 1), shfl_up(eR, 1), q, eL, eR, flat);
}

// The unconstrained flux at the interface above the lane's cell, with the
// lane's Courant number.
template <typename T>
__device__ __forceinline__ T xline_flux_above(T q, T c) {
  const T qL = shfl_up(q, 1), qR = shfl_dn(q, 1);
  const T dp = qR - q;
  const T m = slope_d(q - qL, dp, (qR - qL) * T(0.25));
  const T h = third(m - shfl_dn(m, 1));
  const T rI = fmx(T(.5), dp, h);   // upper edge of the cell
  const T lI = fmx(T(-.5), dp, h);  // lower edge of the cell above
  return flux_e(c, q, shfl_up(lI, 1), rI, qR, lI, shfl_dn(rI, 1));
}

// Column accessor of one level of a stored field: the value at (x, y) with x
// the lane's column, both brought into the stored (halo-padded) array, so
// that rows and lanes past it read some stored value (they only feed outputs
// outside the kernel's range).  A level holds fewer than 2^32
// elements (three levels of 17 fields of that size exceed the device memory).
__device__ __forceinline__ unsigned col_of(const Geom& g, int x) {
  return (unsigned)(min(max(x, -H), g.nx + H - 1) + H + XOFF);
}
__device__ __forceinline__ unsigned row_of(const Geom& g, int y) {
  return (unsigned)(min(max(y, -H), g.ny + H - 1) + H) * (unsigned)g.P;
}

// The inputs of a strip's rows, brought ahead of the row that works on them.
// Ring: into shared memory by asynchronous copies two rows ahead, NF values a
// lane and row; the first N8 fields keep eight rows, the others four.  Each
// lane copies its own column and may read its neighbours' (d = -1, 1; past
// the warp's ends some other value, which only feeds halo lanes).  early()
// and late() issue the copies of one row.  Loads a row ahead into registers left
// the FP64 sweeps waiting on them for 0.6 to 1.5 cycles an issued instruction:
// 9.6 -> 8.6 ms a step of 1024x1024x64.
template <int NF, int N8> constexpr int FEED_BYTES = (N8 * 8 + (NF - N8) * 4) * MW * 8;  // of a warp
template <int NF, int N8>
struct FeedRing {
  char* p;
  unsigned s;
  __device__ __forceinline__ explicit FeedRing(char* sm) {
    p = sm + (threadIdx.x >> 5) * FEED_BYTES<NF, N8>;
    s = (unsigned)__cvta_generic_to_shared(p);
  }
  __device__ __forceinline__ static int slot(int r, int f) {
    return (f < N8 ? (r & 7) * N8 + f : N8 * 8 + (r & 3) * (NF - N8) + (f - N8)) * (MW * 8);
  }
  template <typename E>
  __device__ __forceinline__ void early(int r, int f, const E* q) const {
    const unsigned to = s + slot(r, f) + (threadIdx.x & (MW - 1)) * sizeof(E);
    if constexpr (sizeof(E) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(q) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(q) : "memory");
  }
  template <typename E>
  __device__ __forceinline__ void late(int r, int f, const E* q) const {
    early(r, f, q);
  }
  __device__ __forceinline__ static void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  template <typename A, typename B>
  __device__ __forceinline__ void start(const A& e, const B& l, int j) const {
    e(j);
    l(j);
    commit();
    e(j + 1);
    l(j + 1);
    commit();
  }
  // the values of row j are there (all but the newest two groups have landed, in every lane)
  template <typename A, typename B>
  __device__ __forceinline__ void next(const A& e, const B& l, int j, int jend) const {
    if (j + 2 < jend) {
      e(j + 2);
      l(j + 2);
    }
    commit();
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncwarp();
  }
  template <typename E>
  __device__ __forceinline__ E get(int r, int f, int d = 0) const {
    return *reinterpret_cast<const E*>(p + slot(r, f) + ((int)(threadIdx.x & (MW - 1)) + d) * (int)sizeof(E));
  }
};
// Registers, for fields that the launch itself writes: early() a row ahead,
// late() at the row's start; neighbours by shuffles.
template <int NF, int N8>
struct FeedRegs {
  double cur[NF], nxt[NF];
  __device__ __forceinline__ explicit FeedRegs(char*) {}
  __device__ __forceinline__ static double bits(double v) { return v; }
  __device__ __forceinline__ static double bits(float v) { return __hiloint2double(0, __float_as_int(v)); }
  template <typename E>
  __device__ __forceinline__ void early(int, int f, const E* q) {
    nxt[f] = bits(*q);
  }
  template <typename E>
  __device__ __forceinline__ void late(int, int f, const E* q) {
    cur[f] = bits(*q);
  }
  template <typename A, typename B>
  __device__ __forceinline__ void start(const A& e, const B&, int j) {
    e(j);
  }
  template <typename A, typename B>
  __device__ __forceinline__ void next(const A& e, const B& l, int j, int) {
#pragma unroll
    for (int f = 0; f < NF; ++f) cur[f] = nxt[f];
    e(j + 1);
    l(j);
  }
  template <typename E>
  __device__ __forceinline__ E get(int, int f, int d = 0) const {
    E v;
    if constexpr (sizeof(E) == 8) v = cur[f];
    else v = __int_as_float(__double2loint(cur[f]));
    return d < 0 ? shfl_up(v, 1) : d > 0 ? shfl_dn(v, 1) : v;
  }
};
template <bool RO, int NF, int N8>
using Feed = std::conditional_t<RO, FeedRing<NF, N8>, FeedRegs<NF, N8>>;

// ---------------------------------------------------------------- mass ----
// The C-grid (CGRID) or D-grid mass and potential-temperature sweep of one
// layer (src/mod_sw_dyn.f90:96-268 and 439-598): S the state type, C the
// C-grid fields' type, T the sweep arithmetic.  The FP64 form has S = C = T =
// double; the mixed form keeps the state in double, the C-grid fields in
// float and sweeps in float.  Output region [lo, nx-1+hi] x [lo, ny-1+hi];
// strips of tys rows.
template <typename T, bool CGRID, typename S, typename C>
struct MassM {
  using UB = std::conditional_t<CGRID, S, C>;  // u, v inputs
  using O = std::conditional_t<CGRID, C, S>;   // outputs
};

template <bool RO, bool CGRID, bool SAME> constexpr int MASS_NF = SAME || RO ? (CGRID ? 5 : 4) : 7;
template <bool CGRID, bool SAME> constexpr int MASS_N8 = !CGRID ? 3 : SAME ? 0 : 2;
template <typename T, bool CGRID, typename S, typename C, bool RO = true>
__device__ __forceinline__ void mass_strip(const Geom& g, const Consts& c, const S* dp, const S* pt,
                                           const typename MassM<T, CGRID, S, C>::UB* u,
                                           const typename MassM<T, CGRID, S, C>::UB* v, const double* heat,
                                           typename MassM<T, CGRID, S, C>::O* dpo,
                                           typename MassM<T, CGRID, S, C>::O* pto, int lo, int hi, int* nonfinite,
                                           int sx, int sy, int k, int tys, char* sm) {
  using UB = typename MassM<T, CGRID, S, C>::UB;
  using O = typename MassM<T, CGRID, S, C>::O;
  constexpr int V = CGRID ? PPM_UNC : PPM_NN;
  constexpr bool SAME = std::is_same_v<S, T>;
  constexpr bool KEPT = SAME && RO && !CGRID;  // windows of dp, pt read back from the ring
  const int lane = threadIdx.x & (MW - 1);
  const int ox = lo + sx * MOUT;
  const int oy = lo + sy * tys;
  const int xhi = g.nx - 1 + hi, yhi = g.ny - 1 + hi;
  if (ox > xhi) return;  // the whole warp is past the region
  const int x = ox - MXH + lane;
  const bool out_lane = lane >= MXH && lane < MXH + MOUT && x <= xhi;
  const T dt = T(c.dt), dtdx = T(c.dtdx), dtdy = T(c.dtdy), rA = T(c.rA);
  const T rdx2 = T(c.rdx2), rdy2 = T(c.rdy2), m2rdxy = T(-2.) * T(c.rdx2rdy2);
  const T dxv = dtdx * T(c.vdx), dyv = dtdy * T(c.vdy), vdx = T(c.vdx), vdy = T(c.vdy);
  const long long kS = (long long)k * g.S;
  dp += kS;
  pt += kS;
  u += kS;
  v += kS;
  const unsigned xi = col_of(g, x), xr = col_of(g, x + 1);

  // register windows of the column, named by their row offset from the
  // newest row j of the current iteration
  T d3 = 0, d2 = 0, d1 = 0, d0 = 0;               // dp(j-3 .. j)
  T p3 = 0, p2 = 0, p1 = 0, p0 = 0;               // pt(j-3 .. j)
  T ds2 = 0, ds1 = 0, ds0 = 0;                    // dp(x+1) + dp(x-1), rows j-2 .. j
  T ps2 = 0, ps1 = 0, ps0 = 0;                    // ... of pt
  YLine<T, V> ld_, lp_;                           // the inner x sweeps of dp and pt along y
  T fd1 = 0, fd0 = 0, fp1 = 0, fp0 = 0;           // piecewise-constant y fluxes of dp, pt at interfaces j-3, j-2
  T fy1 = 0, fy0 = 0, fq1 = 0, fq0 = 0;           // y fluxes of dp and pt at interfaces j-3, j-2
  T ld2 = 0, ld1 = 0, ld0 = 0, lq2 = 0, lq1 = 0, lq0 = 0;  // Laplacians of dp, pt at rows j-4 .. j-2
  T uc3 = 0, uc2 = 0, uc1 = 0, uc0 = 0;           // C-grid u at rows j-3 .. j
  T vc1 = 0, vc0 = 0;                             // C-grid v at rows j-3, j-2
  T us = 0;                                       // D-grid u(x, j) + u(x-1, j) (C grid)
  T va_o = 0, vb_o = 0;                           // D-grid v at (x, j-3), (x+1, j-3) (C grid)
  if constexpr (CGRID) {
    const T a = T(u[row_of(g, oy - 3) + xi]);
    us = a + shfl_up(a, 1);
    const unsigned rv = row_of(g, oy - 6);
    va_o = T(v[rv + xi]);
    vb_o = T(v[rv + xr]);
  }
  bool bad = false;
  const int jend = min(oy + tys, yhi + 1) + 3;
  enum { F_DP, F_PT, F_U, F_V, F_VB, F_DU, F_PU };
  Feed<RO, MASS_NF<RO, CGRID, SAME>, MASS_N8<CGRID, SAME>> feed(sm);
  auto early = [&](int j) {
    const unsigned r = row_of(g, j) + xi, rv = row_of(g, j - 2);
    feed.early(j, F_DP, dp + r);
    feed.early(j, F_PT, pt + r);
    feed.early(j, F_U, u + (CGRID ? row_of(g, j + 1) + xi : r));
    feed.early(j, F_V, v + (rv + xi));
    if constexpr (CGRID) feed.early(j, F_VB, v + (rv + xr));
  };
  auto late = [&](int j) {  // the state values of row y (the update in the state's type)
    if constexpr (!SAME && !RO) {
      const unsigned r = row_of(g, j - 3) + xi;
      feed.late(j, F_DU, dp + r);
      feed.late(j, F_PU, pt + r);
    }
  };
  feed.start(early, late, oy - 3);
#pragma unroll MarchL<T, CGRID ? MK_CMASS : MK_DMASS>::unroll
  for (int j = oy - 3; j < jend; ++j) {
    // ---- row j: inputs, C-grid u, the inner x sweep (mod_sw_dyn.f90:109-117, 176-185; 503-511)
    const int y = j - 3;
    const unsigned oi = row_of(g, y) + xi;
    feed.next(early, late, j, jend);
    S d_upd = 0, p_upd = 0;  // the state values of row y
    if constexpr (!SAME) {
      d_upd = RO ? feed.template get<S>(y, F_DP) : feed.template get<S>(j, F_DU);
      p_upd = RO ? feed.template get<S>(y, F_PT) : feed.template get<S>(j, F_PU);
    }
    const T dn = T(feed.template get<S>(j, F_DP)), pn = T(feed.template get<S>(j, F_PT));
    const T ua_c = T(feed.template get<UB>(j, F_U)), va_c = T(feed.template get<UB>(j, F_V));
    const T vb_c = CGRID ? T(feed.template get<UB>(j, F_VB)) : T(0);
    T ucn;
    if constexpr (CGRID) {  // .5 (.5 (u + u(x-1)) + .5 (the row above)): the halvings are exact
      const T s = ua_c + shfl_up(ua_c, 1);
      ucn = T(.25) * (us + s);
      us = s;
    } else {
      ucn = ua_c;
    }
    const T ucR = shfl_dn(ucn, 1);
    T dL, dR, pL, pR;
    if constexpr (KEPT) {
      dL = feed.template get<S>(j, F_DP, -1);
      dR = feed.template get<S>(j, F_DP, 1);
      pL = feed.template get<S>(j, F_PT, -1);
      pR = feed.template get<S>(j, F_PT, 1);
    } else {
      dL = shfl_up(dn, 1);
      dR = shfl_dn(dn, 1);
      pL = shfl_up(pn, 1);
      pR = shfl_dn(pn, 1);
    }
    T txn, tpn;
    {
      const bool c0 = dtdx * ucn > T(0), c1 = dtdx * ucR > T(0);
      const T den = T(1) / fmadd(-dtdx, ucR - ucn, T(1));
      txn = inner_e(dn, c0 ? dL : dn, c1 ? dn : dR, den, rA);
      tpn = inner_e(pn, c0 ? pL : pn, c1 ? pn : pR, den, rA);
    }
    // shift the windows to the new row
    if constexpr (KEPT) {
      d1 = feed.template get<S>(j - 1, F_DP);
      d2 = feed.template get<S>(j - 2, F_DP);
      d3 = feed.template get<S>(y, F_DP);
      p1 = feed.template get<S>(j - 1, F_PT);
      p2 = feed.template get<S>(j - 2, F_PT);
      p3 = feed.template get<S>(y, F_PT);
      ds2 = feed.template get<S>(j - 2, F_DP, 1) + feed.template get<S>(j - 2, F_DP, -1);
      ps2 = feed.template get<S>(j - 2, F_PT, 1) + feed.template get<S>(j - 2, F_PT, -1);
    } else {
      d3 = d2; d2 = d1; d1 = d0; d0 = dn;
      p3 = p2; p2 = p1; p1 = p0; p0 = pn;
      ds2 = ds1; ds1 = ds0; ds0 = dR + dL;
      ps2 = ps1; ps1 = ps0; ps0 = pR + pL;
    }
    if constexpr (RO && !CGRID) {
      uc3 = T(feed.template get<UB>(y, F_U));
    } else {
      uc3 = uc2; uc2 = uc1; uc1 = uc0; uc0 = ucn;
    }
    ld_.push(txn);
    lp_.push(tpn);
    // C-grid v of row j-2 (:109-117)
    vc1 = vc0;
    if constexpr (CGRID) {
      vc0 = T(.25) * ((va_c + va_o) + (vb_c + vb_o));
      va_o = va_c;
      vb_o = vb_c;
    } else {
      vc0 = va_c;
    }
    {  // inner and outer y sweeps' fluxes at the interface below row j-2
      const T cy = dtdx * vc0;
      const bool pos = cy > T(0);
      fd1 = fd0; fp1 = fp0;
      fd0 = pos ? d3 : d2;
      fp0 = pos ? p3 : p2;
      fy1 = fy0; fq1 = fq0;
      fy0 = ld_.flux(cy) * cy;
      fq0 = lp_.flux(cy);
    }
    // Laplacians of row j-2 (:158-173)
    ld2 = ld1; ld1 = ld0;
    lq2 = lq1; lq1 = lq0;
    ld0 = fmadd(d1 + d3, rdy2, fmadd(ds2, rdx2, d2 * m2rdxy));
    lq0 = fmadd(p1 + p3, rdy2, fmadd(ps2, rdx2, p2 * m2rdxy));
    if (y >= oy) {  // (the rows below are the strip's warm-up)
      // ---- row y: inner y sweep, the outer x sweep, the update
      const T den = T(1) / fmadd(-dtdy, vc0 - vc1, T(1));
      const T tyd = inner_e(d3, fd1, fd0, den, rA);
      const T typ = inner_e(p3, fp1, fp0, den, rA);
      const T cx = dtdx * uc3;
      const T fxd = xline_flux<T, V>(tyd, cx) * cx;
      const T fxp = xline_flux<T, V>(typ, cx);
      const T fxd1 = shfl_dn(fxd, 1), fxp1 = shfl_dn(fxp, 1);
      const T lxm = shfl_up(ld1, 1), lxp = shfl_dn(ld1, 1);
      const T qxm = shfl_up(lq1, 1), qxp = shfl_dn(lq1, 1);
      if (out_lane && y <= yhi) {
        // updates, mod_sw_dyn.f90:163-172,193-202,230-237,258-267 (C); 490-499,519-528,555-562,582-591 (D)
        O vo, qo;
        if constexpr (SAME) {  // the reference's operations, in order
          const T d = d3;
          T vv = d - (fxd1 - fxd + dxv * (fmx(T(-2), ld1, lxp) + lxm));
          vv = vv - (fy0 - fy1 + dyv * (fmx(T(-2), ld1, ld0) + ld2));
          T q = d * p3 - (fxp1 * fxd1 - fxp * fxd + vdx * ((qxp - lq1) * fxd1 - (lq1 - qxm) * fxd));
          q = q - (fq0 * fy0 - fq1 * fy1 + vdy * ((lq0 - lq1) * fy0 - (lq1 - lq2) * fy1));
          if (heat) q = q + dt * d * T(heat[kS + oi]);
          q = q / vv;
          vo = O(vv);
          qo = O(q);
        } else {
          // the same update in flux form: interface fluxes (advective plus
          // vorticity-damping) in the sweep type, their differences applied to
          // the state's type, so that mass and dp*pt telescope in S
          const T Fx0 = fmadd(dxv, ld1 - lxm, fxd), Fx1 = fmadd(dxv, lxp - ld1, fxd1);
          const T Fy0 = fmadd(dyv, ld1 - ld2, fy1), Fy1 = fmadd(dyv, ld0 - ld1, fy0);
          const T Hx0 = fmadd(vdx, lq1 - qxm, fxp) * fxd, Hx1 = fmadd(vdx, qxp - lq1, fxp1) * fxd1;
          const T Hy0 = fmadd(vdy, lq1 - lq2, fq1) * fy1, Hy1 = fmadd(vdy, lq0 - lq1, fq0) * fy0;
          const S d = d_upd;
          const S vv = d - ((S(Fx1) - S(Fx0)) + (S(Fy1) - S(Fy0)));
          S q = d * p_upd - ((S(Hx1) - S(Hx0)) + (S(Hy1) - S(Hy0)));
          if (heat) q = q + S(c.dt) * d * S(heat[kS + oi]);
          q = q / vv;
          vo = O(vv);
          qo = O(q);
        }
        dpo[kS + oi] = vo;
        pto[kS + oi] = qo;
        const bool inside = x >= 0 && x < g.nx && y >= 0 && y < g.ny;
        bad = bad || (inside && !(finite_(vo) && finite_(qo)));
      }
    }
  }
  if (nonfinite) flag_nonfinite(nonfinite, bad);
}

// shared memory of a warp, and of a block beside its warps' (the values past
// the ends of the first and last warps' rows)
constexpr int FEED_PAD = 16;
template <typename T, bool CGRID, typename S>
constexpr int MASS_SMEM = FEED_BYTES<MASS_NF<true, CGRID, std::is_same_v<S, T>>, MASS_N8<CGRID, std::is_same_v<S, T>>>;

// one warp per strip: across x within the block and blockIdx.x, blockIdx.y
// across y, blockIdx.z the layer
__device__ __forceinline__ int strip_x() { return (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); }
template <typename T, bool CGRID, typename S, typename C>
__global__ void __launch_bounds__(MW * MWARPS, MarchL<T, CGRID ? MK_CMASS : MK_DMASS>::min_blocks) k_mass_m(Geom g, Consts c, const S* dp,
                                                         const S* pt,
                                                         const typename MassM<T, CGRID, S, C>::UB* u,
                                                         const typename MassM<T, CGRID, S, C>::UB* v,
                                                         const double* heat,
                                                         typename MassM<T, CGRID, S, C>::O* dpo,
                                                         typename MassM<T, CGRID, S, C>::O* pto, int lo,
                                                         int hi, int* nonfinite, int tys) {
  stream_order();
  extern __shared__ __align__(16) char feed_sm[];
  mass_strip<T, CGRID, S, C>(g, c, dp, pt, u, v, heat, dpo, pto, lo, hi, nonfinite, strip_x(), blockIdx.y, blockIdx.z,
                             tys, feed_sm + 8);
}

// ======================================================== C-grid momentum ==
// The C-grid momentum update of one layer (src/mod_sw_dyn.f90:294-414):
// kinetic energy from PPM fluxes of the C-grid winds with the
// layer-nlay A-grid winds (:299-317), absolute vorticity (:319-323), the
// pressure-gradient force (:325-339) and the vorticity-flux updates of uc
// and vc (:344-412).  Outputs on the interior; strips of tys rows.
constexpr int CMOM_NF = 10;
template <typename T, typename S, typename C, bool RO = true>
__device__ __forceinline__ void c_mom_strip(const Geom& g, const Consts& c, const S* ud, const S* vd,
                                            const double* pkap, const double* gz, C* uc, C* vc, int sx, int sy, int k,
                                            int tys, char* sm) {
  constexpr int UNC = PPM_UNC;
  const int lane = threadIdx.x & (MW - 1);
  const int ox = sx * MOUT;
  const int oy = sy * tys;
  if (ox >= g.nx) return;  // the whole warp is past the region
  const int x = ox - MXH + lane;
  const bool out_lane = lane >= MXH && lane < MXH + MOUT && x < g.nx;
  const T dt = T(c.dt), dtdx = T(c.dtdx), dtdy = T(c.dtdy), rA = T(c.rA);
  const T rdx = T(c.rdx), rdy = T(c.rdy), f = T(c.coriolis);
  const T rdx2 = T(c.rdx2), rdy2 = T(c.rdy2), m2rdxy = T(-2.) * T(c.rdx2rdy2);
  const T vdx = T(c.vdx), vdy = T(c.vdy);
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const S *uk = ud + kS, *vk = vd + kS, *uL = ud + LS, *vL = vd + LS;
  const double *pka = pkap + kS, *pkb = pka + g.S, *gza = gz + kS, *gzb = gza + g.S;
  const unsigned xi = col_of(g, x), xl = col_of(g, x - 1), xr = col_of(g, x + 1);

  // register windows of the column, named by their row offset from the
  // newest row j of the iteration
  unsigned r = row_of(g, oy - 3);
  T u_x = T(uk[r + xi]), u_xm = T(uk[r + xl]);  // ud(x, j), ud(x-1, j)
  r = row_of(g, oy - 4);
  T v_x = T(vk[r + xi]), v_xp = T(vk[r + xr]);  // vd(x, j-1), vd(x+1, j-1)
  T uw3 = 0, uw2 = 0, uw1 = 0, uw0 = 0;  // ud(x, j-3 .. j)
  T vw4 = 0, vw3 = 0, vw2 = 0, vw1 = 0, vw0 = 0;  // vd(x, j-4 .. j)
  T a3 = 0, a2 = 0, a1 = 0, a0 = 0;      // C-grid u of this layer, rows j-3 .. j
  YLine<T, UNC> lb;                      // C-grid v of this layer along y
  YLine<T, UNC> lt;                      // the inner x sweep of the vorticity along y
  T w3 = 0, w2 = 0, w1 = 0, w0 = 0;      // absolute vorticity, rows j-3 .. j
  T ws2 = 0, ws1 = 0, ws0 = 0;           // its x(+1) + x(-1), rows j-2 .. j
  T fw1 = 0, fw0 = 0;                    // its piecewise-constant y flux at interfaces j-3, j-2
  T lp1 = 0, lp0 = 0;                    // Laplacian of the vorticity, rows j-3, j-2
  T ke1 = 0, ke0 = 0;                    // kinetic energy, rows j-4, j-3
  double pk0m = 0, pk1m = 0, gz0m = 0, gz1m = 0;  // pkap, gz at k and k+1, row j-4
  // layer-nlay ud at row y and vd at rows y-1, y of the first kinetic-energy row y = oy-1
  T uL1 = T(uL[row_of(g, oy - 1) + xi]);
  T vL2 = T(vL[row_of(g, oy - 2) + xi]), vL1 = T(vL[row_of(g, oy - 1) + xi]);
  const int jend = min(oy + tys, g.ny) + 3;
  enum { F_U, F_UM, F_V, F_VP, F_P0, F_P1, F_G0, F_G1, F_UN, F_VN };
  Feed<RO, CMOM_NF, 0> feed(sm);
  auto early = [&](int j) {
    const unsigned ru = row_of(g, j + 1), rv = row_of(g, j);
    feed.early(j, F_U, uk + (ru + xi));
    feed.early(j, F_UM, uk + (ru + xl));
    feed.early(j, F_V, vk + (rv + xi));
    feed.early(j, F_VP, vk + (rv + xr));
  };
  auto late = [&](int j) {  // the pressure terms of row y = j-3, layer-nlay winds of row y+1
    const unsigned oi = row_of(g, j - 3) + xi, ri = row_of(g, j - 2) + xi;
    feed.late(j, F_P0, pka + oi);
    feed.late(j, F_P1, pkb + oi);
    feed.late(j, F_G0, gza + oi);
    feed.late(j, F_G1, gzb + oi);
    feed.late(j, F_UN, uL + ri);
    feed.late(j, F_VN, vL + ri);
  };
  feed.start(early, late, oy - 3);
#pragma unroll MarchL<T, MK_CMOM>::unroll
  for (int j = oy - 3; j < jend; ++j) {
    const int y = j - 3;
    const unsigned oi = row_of(g, y) + xi;
    feed.next(early, late, j, jend);
    // ---- row j: C-grid winds of the layer (:110-117), vorticity (:319-323),
    // inner x sweep of the vorticity (:353-367)
    const T un = T(feed.template get<S>(j, F_U)), unm = T(feed.template get<S>(j, F_UM));
    const T vn = T(feed.template get<S>(j, F_V)), vnp = T(feed.template get<S>(j, F_VP));
    const T ucn = T(.25) * ((u_x + u_xm) + (un + unm));  // the reference's halvings are exact
    const T vcn = T(.25) * ((vn + v_x) + (vnp + v_xp));
    const T vor = fmadd(vcn - shfl_up(vcn, 1), rdx, fmadd(-(ucn - a0), rdy, f));
    const T vl = shfl_up(vor, 1), vr = shfl_dn(vor, 1);
    T tun;
    {
      const T den = T(1) / fmadd(-dtdx, u_x - u_xm, T(1));
      tun = inner_e(vor, (dtdx * u_xm > T(0)) ? vl : vor, (dtdx * u_x > T(0)) ? vor : vr, den, rA);
    }
    uw3 = uw2; uw2 = uw1; uw1 = uw0; uw0 = u_x;
    u_x = un;
    u_xm = unm;
    v_x = vn;
    v_xp = vnp;
    vw4 = vw3; vw3 = vw2; vw2 = vw1; vw1 = vw0; vw0 = vn;
    a3 = a2; a2 = a1; a1 = a0; a0 = ucn;
    w3 = w2; w2 = w1; w1 = w0; w0 = vor;
    ws2 = ws1; ws1 = ws0; ws0 = vr + vl;
    const T b3 = lb.q2;  // C-grid v of row j-3
    lb.push(vcn);
    lt.push(tun);
    // the vorticity's inner y sweep at the interface below row j-2 (vd(x, j-3)), its Laplacian at row j-2
    fw1 = fw0;
    fw0 = (dtdx * vw3 > T(0)) ? w3 : w2;
    lp1 = lp0;
    lp0 = fmadd(w1 + w3, rdy2, fmadd(ws2, rdx2, w2 * m2rdxy));
    if (y >= oy - 1) {  // (the rows below are the strip's warm-up)
      // ---- row y: kinetic energy (:299-317) with the layer-nlay A-grid winds
      // (:110-125 at k = nlay), recomputed where they are read
      const T uL0 = T(feed.template get<S>(j, F_UN)), vL0 = T(feed.template get<S>(j, F_VN));
      T ken;
      {
        const T ub = T(.5) * (uL1 + shfl_up(uL1, 1));
        const T ucl = T(.5) * (ub + T(.5) * (uL0 + shfl_up(uL0, 1)));
        const T ua = T(.5) * (ucl + T(.25) * (shfl_dn(uL1, 1) + uL1 + shfl_dn(uL0, 1) + uL0));
        const T vb = T(.5) * (vL1 + vL2);
        const T vL1r = shfl_dn(vL1, 1);
        const T vcl = T(.5) * (vb + T(.5) * (vL1r + shfl_dn(vL2, 1)));
        const T va = T(.5) * (vcl + T(.25) * (vL0 + vL1 + shfl_dn(vL0, 1) + vL1r));
        const T kv = va * lb.flux(dtdy * va);
        // the flux at the interface above the lane's cell: that of the next lane's lower interface
        const T fx = xline_flux_above<T>(a3, dtdx * ua);
        ken = T(.5) * fmadd(ua, fx, kv);
      }
      uL1 = uL0;
      vL2 = vL1;
      vL1 = vL0;
      ke1 = ke0;
      ke0 = ken;
      const double pk0 = feed.template get<double>(j, F_P0), pk1 = feed.template get<double>(j, F_P1);
      const double gz0 = feed.template get<double>(j, F_G0), gz1 = feed.template get<double>(j, F_G1);
      const double pk0l = shfl_up(pk0, 1), pk1l = shfl_up(pk1, 1), gz0l = shfl_up(gz0, 1), gz1l = shfl_up(gz1, 1);
      const double pk0d = pk0m, pk1d = pk1m, gz0d = gz0m, gz1d = gz1m;  // row y-1
      pk0m = pk0; pk1m = pk1; gz0m = gz0; gz1m = gz1;
      if (y >= oy) {
        // ---- row y: inner y sweep of the vorticity (:388-397), its x sweep, the updates
        const T den = T(1) / fmadd(-dtdy, vw3 - vw4, T(1));
        const T tvn = inner_e(w3, fw1, fw0, den, rA);
        const T ke_l = shfl_up(ke0, 1);
        const T lp_r = shfl_dn(lp1, 1);
        const T udx = uw3, vdx_ = vw3;
        const T fx = xline_flux_above<T>(tvn, dtdx * udx);
        if (out_lane && y < g.ny) {
          const double pgx = ((pk0 - pk1l) * (gz0l - gz1) + (pk0l - pk1) * (gz1l - gz0)) / (pk0 - pk1l + pk0l - pk1);
          const double pgy = ((pk0 - pk1d) * (gz0d - gz1) + (pk0d - pk1) * (gz1d - gz0)) / (pk0 - pk1d + pk0d - pk1);
          const T fy = lt.flux(dtdx * vdx_);
          uc[kS + oi] = C(fmadd(-dtdx, ke0 - ke_l - T(pgx), fmadd(dt, fmadd(vdy, lp0 - lp1, vdx_ * fy), a3)));
          vc[kS + oi] = C(fmadd(-dtdy, ke0 - ke1 - T(pgy), fmadd(-dt, fmadd(vdx, lp_r - lp1, udx * fx), b3)));
        }
      }
    }
  }
}

template <typename T, typename S, typename C>
__global__ void __launch_bounds__(MW * MWARPS, MarchL<T, MK_CMOM>::min_blocks) k_c_mom_m(Geom g, Consts c, const S* ud,
                                                          const S* vd, const double* pkap,
                                                          const double* gz, C* uc,
                                                          C* vc, int tys) {
  stream_order();
  extern __shared__ __align__(16) char feed_sm[];
  c_mom_strip<T, S, C>(g, c, ud, vd, pkap, gz, uc, vc, strip_x(), blockIdx.y, blockIdx.z, tys, feed_sm);
}

// ======================================================== D-grid momentum ==
// The D-grid momentum update of one layer (src/mod_sw_dyn.f90:634-771):
// kinetic energy from constrained-PPM fluxes of ud, vd with the
// layer-nlay B-grid winds (:639-657, 441-444), vorticity (:659-663), the
// B-grid pressure-gradient force (:665-679), del^4 divergence damping
// (:682-702) and the vorticity-flux updates (:708-769).  Outputs on the
// interior; strips of tys rows.
template <bool SAME> constexpr int DMOM_NF = SAME ? 10 : 12;
template <typename T, typename S, typename C, bool RO = true>
__device__ __forceinline__ void d_mom_strip(const Geom& g, const Consts& c, const S* ud, const S* vd, const C* uc,
                                            const C* vc, const double* pkapb, const double* gzb, S* udo, S* vdo,
                                            int* nonfinite, int sx, int sy, int k, int tys, char* sm) {
  constexpr int CON = PPM_CON;
  constexpr bool SAME = std::is_same_v<S, T>;
  const int lane = threadIdx.x & (MW - 1);
  const int ox = sx * MOUT;
  const int oy = sy * tys;
  if (ox >= g.nx) return;  // the whole warp is past the region
  const int x = ox - MXH + lane;
  const bool out_lane = lane >= MXH && lane < MXH + MOUT && x < g.nx;
  const T dt = T(c.dt), dtdx = T(c.dtdx), dtdy = T(c.dtdy), rA = T(c.rA);
  const T rdx = T(c.rdx), rdy = T(c.rdy), f = T(c.coriolis);
  const T rdx2 = T(c.rdx2), rdy2 = T(c.rdy2), m2rdxy = T(-2.) * T(c.rdx2rdy2);
  const T vdx = T(c.vdx), vdy = T(c.vdy), divdamp = T(c.divdamp);
  const long long kS = (long long)k * g.S, LS = (long long)(g.L - 1) * g.S;
  const S *uk = ud + kS, *vk = vd + kS;
  const C *uL = uc + LS, *vL = vc + LS, *ucK = uc + kS, *vcK = vc + kS;
  const double *pba = pkapb + kS, *pbb = pba + g.S, *gba = gzb + kS, *gbb = gba + g.S;
  const unsigned xi = col_of(g, x);

  // register windows of the column, named by their row offset from the
  // newest row j of the iteration
  unsigned r = row_of(g, oy - 3) + xi;
  T s3 = 0, s2 = 0, s1 = 0, s0 = T(uk[r]);  // ud(x, j-3 .. j)
  T v0 = T(vk[r]), v3 = 0;                  // vd(x, j), vd(x, j-3)
  YLine<T, CON> lv;                                 // vd along y
  lv.q0 = v0;
  T q2 = 0, q1 = 0, q0 = 0;                         // divergence, rows j-2 .. j
  T qs1 = 0, qs0 = 0;                               // its x(+1) + x(-1), rows j-1, j
  T e3 = 0, e2 = 0, e1 = 0;                         // its Laplacian, rows j-3 .. j-1
  T es2 = 0, es1 = 0;                               // x(+1) + x(-1) of that, rows j-2, j-1
  T dd3 = 0, dd2 = 0;                               // del^4 damping term, rows j-3, j-2
  T w3 = 0, w2 = 0, w1 = 0;                         // vorticity, rows j-3 .. j-1
  T ws2 = 0, ws1 = 0;                               // its x(+1) + x(-1), rows j-2, j-1
  YLine<T, CON> lt;                                 // inner x sweep of the vorticity along y (newest row j-1)
  T fw1 = 0, fw0 = 0;                               // the vorticity's piecewise-constant y flux at interfaces j-3, j-2
  T ke3 = 0, ke2 = 0;                               // kinetic energy, rows j-3, j-2
  T lp4 = 0, lp3 = 0, lp2 = 0;                      // Laplacian of the vorticity, rows j-4 .. j-2
  T cu3 = 0, cu2 = T(uL[row_of(g, oy - 5) + xi]), cu1 = T(uL[row_of(g, oy - 4) + xi]);  // layer-nlay uc, rows j-3 .. j-1
  T cv3 = 0, cv2 = T(vL[row_of(g, oy - 5) + xi]);  // layer-nlay vc, rows j-3, j-2
  double pb0y = 0, pb1y = 0, gb0y = 0, gb1y = 0;    // pkapb, gzb at k, k+1, row j-3
  bool bad = false;
  const int jend = min(oy + tys, g.ny) + 3;
  enum { F_U, F_V, F_CU, F_CV, F_P0, F_P1, F_G0, F_G1, F_UC, F_VC, F_UO, F_VO };
  Feed<RO, DMOM_NF<SAME>, 0> feed(sm);
  auto early = [&](int j) {
    const unsigned r = row_of(g, j) + xi;
    feed.early(j, F_U, uk + r);
    feed.early(j, F_V, vk + r);
    feed.early(j, F_CU, uL + (row_of(g, j - 1) + xi));
    feed.early(j, F_CV, vL + (row_of(g, j - 2) + xi));
  };
  auto late = [&](int j) {  // the pressure terms of row j-2, the winds of row y = j-3
    const unsigned r = row_of(g, j - 2) + xi, oi = row_of(g, j - 3) + xi;
    feed.late(j, F_P0, pba + r);
    feed.late(j, F_P1, pbb + r);
    feed.late(j, F_G0, gba + r);
    feed.late(j, F_G1, gbb + r);
    feed.late(j, F_UC, ucK + oi);
    feed.late(j, F_VC, vcK + oi);
    if constexpr (!SAME) {
      feed.late(j, F_UO, uk + oi);
      feed.late(j, F_VO, vk + oi);
    }
  };
  feed.start(early, late, oy - 2);
#pragma unroll MarchL<T, MK_DMOM>::unroll
  for (int j = oy - 2; j < jend; ++j) {
    const int y = j - 3;
    const unsigned oi = row_of(g, y) + xi;
    feed.next(early, late, j, jend);
    // ---- row j inputs; vorticity of row j-1 (:659-663), divergence of row j (:682-685)
    const T sn = T(feed.template get<S>(j, F_U)), vn = T(feed.template get<S>(j, F_V));
    const C cu_c = feed.template get<C>(j, F_CU), cv_c = feed.template get<C>(j, F_CV);
    const T vorn = fmadd(shfl_dn(v0, 1) - v0, rdx, fmadd(-(sn - s0), rdy, f));
    const T dvn = fmadd(rdy, vn - v0, rdx * (sn - shfl_up(sn, 1)));
    s3 = s2; s2 = s1; s1 = s0; s0 = sn;
    v3 = lv.q2;
    v0 = vn;
    w3 = w2; w2 = w1; w1 = vorn;
    q2 = q1; q1 = q0; q0 = dvn;
    qs1 = qs0; qs0 = shfl_dn(dvn, 1) + shfl_up(dvn, 1);
    cu3 = cu2; cu2 = cu1; cu1 = T(cu_c);
    cv3 = cv2; cv2 = T(cv_c);
    // vd's slope at row j-1, its edges at row j-2 (:870-911)
    lv.push(vn);
    // del^2 of the divergence at row j-1 (:688-692), del^4 at row j-2 (:695-702)
    e3 = e2; e2 = e1;
    e1 = fmadd(q0 + q2, rdy2, fmadd(qs1, rdx2, q1 * m2rdxy));
    es2 = es1; es1 = shfl_dn(e1, 1) + shfl_up(e1, 1);
    dd3 = dd2;
    dd2 = divdamp * (fmadd(e1 + e3, rdy2, fmadd(es2, rdx2, e2 * m2rdxy)));
    // inner x sweep of the vorticity at row j-1 with the layer-nlay Courant numbers (:708-722)
    {
      const T cR = shfl_dn(cu1, 1);
      const T den = T(1) / fmadd(-dtdx, cR - cu1, T(1));
      const T wl = shfl_up(w1, 1), wr = shfl_dn(w1, 1);  // every lane takes part in the shuffles
      ws2 = ws1; ws1 = wr + wl;
      lt.push(inner_e(w1, (dtdx * cu1 > T(0)) ? wl : w1, (dtdx * cR > T(0)) ? w1 : wr, den, rA));
    }
    // the vorticity's inner y sweep at the interface below row j-2, its Laplacian at row j-2
    fw1 = fw0;
    fw0 = (dtdx * cv2 > T(0)) ? w3 : w2;
    lp4 = lp3; lp3 = lp2;
    lp2 = fmadd(w1 + w3, rdy2, fmadd(ws2, rdx2, w2 * m2rdxy));
    // kinetic energy of row j-2 with PPM_CONSTRAINED (:639-657) and the
    // layer-nlay B-grid winds (:441-444)
    {
      const T ubL = T(.5) * (cu2 + cu3);
      const T vbL = T(.5) * (cv2 + shfl_up(cv2, 1));
      const T kv = vbL * lv.flux(dtdy * vbL);
      const T fx = xline_flux<T, CON>(s2, dtdx * ubL);
      ke3 = ke2;
      ke2 = T(.5) * fmadd(ubL, fx, kv);
    }
    if (y >= oy) {
      // ---- row y: inner y sweep of the vorticity (:744-753), its x sweep, the
      // updates of ud, vd (:724-738, 755-769) with the B-grid PGF
      const T den = T(1) / fmadd(-dtdy, cv2 - cv3, T(1));
      const T tv = inner_e(w3, fw1, fw0, den, rA);
      const T fx = xline_flux<T, CON>(tv, dtdx * cu3);
      const T fy = lt.flux(dtdx * cv3);
      const T ke_r = shfl_dn(ke3, 1), dd_r = shfl_dn(dd3, 1), lp_l = shfl_up(lp3, 1);
      const double pb0n = feed.template get<double>(j, F_P0), pb1n = feed.template get<double>(j, F_P1);
      const double gb0n = feed.template get<double>(j, F_G0), gb1n = feed.template get<double>(j, F_G1);
      const double pb0r = shfl_dn(pb0y, 1), pb1r = shfl_dn(pb1y, 1), gb0r = shfl_dn(gb0y, 1), gb1r = shfl_dn(gb1y, 1);
      if (out_lane && y < g.ny) {
        const double pgx = ((pb0r - pb1y) * (gb0y - gb1r) + (pb0y - pb1r) * (gb1y - gb0r)) / (pb0r - pb1y + pb0y - pb1r);
        const double pgy = ((pb0n - pb1y) * (gb0y - gb1n) + (pb0y - pb1n) * (gb1y - gb0n)) / (pb0n - pb1y + pb0y - pb1n);
        const T svc = T(feed.template get<C>(j, F_VC)), suc = T(feed.template get<C>(j, F_UC));
        S u, v;
        if constexpr (SAME) {  // the reference's operations, in order
          u = s3 + dt * (svc * fy + vdy * (lp3 - lp4)) - dtdx * (ke_r - ke3 - dd_r + dd3 - T(pgx));
          v = v3 - dt * (suc * fx + vdx * (lp3 - lp_l)) - dtdy * (ke2 - ke3 - dd2 + dd3 - T(pgy));
        } else {  // the tendency in the sweep type added to the state's type
          const T du = fmadd(-dtdx, ke_r - ke3 - dd_r + dd3 - T(pgx), dt * fmadd(vdy, lp3 - lp4, svc * fy));
          const T dv = fmadd(-dtdy, ke2 - ke3 - dd2 + dd3 - T(pgy), -dt * fmadd(vdx, lp3 - lp_l, suc * fx));
          u = feed.template get<S>(j, F_UO) + S(du);
          v = feed.template get<S>(j, F_VO) + S(dv);
        }
        udo[kS + oi] = u;
        vdo[kS + oi] = v;
        bad = bad || !(finite_(u) && finite_(v));
      }
    }
    if (y >= oy - 1) {
      pb0y = feed.template get<double>(j, F_P0);
      pb1y = feed.template get<double>(j, F_P1);
      gb0y = feed.template get<double>(j, F_G0);
      gb1y = feed.template get<double>(j, F_G1);
    }
  }
  flag_nonfinite(nonfinite, bad);
}

template <typename T, typename S, typename C>
__global__ void __launch_bounds__(MW * MWARPS, MarchL<T, MK_DMOM>::min_blocks) k_d_mom_m(Geom g, Consts c, const S* ud,
                                                          const S* vd, const C* uc,
                                                          const C* vc, const double* pkapb,
                                                          const double* gzb, S* udo,
                                                          S* vdo, int* nonfinite, int tys) {
  stream_order();
  extern __shared__ __align__(16) char feed_sm[];
  d_mom_strip<T, S, C>(g, c, ud, vd, uc, vc, pkapb, gzb, udo, vdo, nonfinite, strip_x(), blockIdx.y, blockIdx.z, tys,
                       feed_sm);
}

// ================================================================ corners ==
// interpolate_to_corners (src/mod_sw_dyn.f90:921-956; corner() of
// atm_kernels.cuh, in its order) of pkap at level l into pkapb and of gz at level
// l+1 into gzb on [0, nx] x [0, ny], l = blockIdx.z (PK = false: gz at level l
// alone).  A strip as the sweeps': each point is loaded once, its interpolation
// along x formed once and kept for four rows, that along y formed once and
// passed between lanes; 29 of the 32 columns are outputs.  A thread a corner
// loaded 32 values of L1 a corner: 0.67 ms at 1024x1024x64 -> 0.42 (251x187x27: 22 us -> 18), bound by the
// four fields' traffic.
constexpr int COUT = 29, CORN_WARPS_SM = 32;
template <bool PK> constexpr int CORN_SMEM = FEED_BYTES<PK ? 2 : 1, 0>;
struct CornerLine {
  double q3 = 0, q2 = 0, q1 = 0, q0 = 0, t3 = 0, t2 = 0, t1 = 0, t0 = 0;  // values, x interpolations of rows j-3 .. j
  __device__ __forceinline__ double push(double q) {  // the corner of row j-1
    q3 = q2; q2 = q1; q1 = q0; q0 = q;
    t3 = t2; t2 = t1; t1 = t0;
    t0 = C7_12 * (q + shfl_up(q, 1)) - C1_12 * (shfl_dn(q, 1) + shfl_up(q, 2));
    const double y = C7_12 * (q1 + q2) - C1_12 * (q0 + q3);
    double out = C9_32 * (t1 + t2) - C1_32 * (t0 + t3);
    out = out + C9_32 * (y + shfl_up(y, 1)) - C1_32 * (shfl_dn(y, 1) + shfl_up(y, 2));
    return out;
  }
};
template <bool PK>
__global__ void __launch_bounds__(MW * MWARPS, CORN_WARPS_SM / MWARPS) k_corners_m(Geom g, const double* pkap,
                                                                                 const double* gz,
                                                                                 double* pkapb,
                                                                                 double* gzb, int tys) {
  stream_order();
  extern __shared__ __align__(16) char feed_sm[];
  const int lane = threadIdx.x & (MW - 1);
  const int ox = strip_x() * COUT, oy = (int)blockIdx.y * tys;
  if (ox > g.nx) return;
  const int x = ox - 2 + lane, yend = min(oy + tys, g.ny + 1);
  const bool out = lane >= 2 && lane < 2 + COUT && x <= g.nx;
  const long long kS = (long long)blockIdx.z * g.S, zS = PK ? kS + g.S : kS;
  const unsigned xi = col_of(g, x);
  enum { F_GZ, F_PK };
  FeedRing<PK ? 2 : 1, 0> feed(feed_sm);
  auto copy = [&](int j) {
    const unsigned r = row_of(g, j) + xi;
    feed.early(j, F_GZ, gz + (zS + r));
    if constexpr (PK) feed.early(j, F_PK, pkap + (kS + r));
  };
  auto none = [](int) {};
  feed.start(copy, none, oy - 2);
  CornerLine lz, lp;
#pragma unroll 4
  for (int j = oy - 2; j <= yend; ++j) {
    feed.next(copy, none, j, yend + 1);
    const double z = lz.push(feed.template get<double>(j, F_GZ));
    double p = 0.;
    if constexpr (PK) p = lp.push(feed.template get<double>(j, F_PK));
    if (j > oy && out) {
      const unsigned r = row_of(g, j - 1) + xi;
      gzb[zS + r] = z;
      if constexpr (PK) pkapb[kS + r] = p;
    }
  }
}

}  // namespace atm
