// Shared device definitions of the B200 dynamical core: field geometry in
// HBM, physical constants, how kernels share rows, status words, and division by
// constants.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "atm_math.h"

namespace atm {

// Halo width of every stored field, src/mod_tiles.f90:12.
constexpr int H = 7;
// Leading pad of each row so that interior column i = 0 starts 64 bytes
// into a 256-byte-aligned row for FP64 (32 bytes for FP32).
constexpr int XOFF = 1;

// src/mod_constants.f90:8-14; R_dry is a default-real (FP32) literal.
constexpr double R_DRY = (double)287.052874f;
constexpr double CP_DRY = 1005.0;
constexpr double CV_DRY = CP_DRY - R_DRY;
constexpr double KAPPA = R_DRY / CP_DRY;
// Default-real constant expressions of src/mod_sw_dyn.f90:933-953 and
// src/mod_remap.f90:86-100,243.
constexpr double C7_12 = (double)(7.0f / 12.0f);
constexpr double C1_12 = (double)(1.0f / 12.0f);
constexpr double C9_32 = (double)(9.0f / 32.0f);
constexpr double C1_32 = (double)(1.0f / 32.0f);
constexpr double C2_3 = (double)(2.0f / 3.0f);

// Flux variants, src/mod_sw_dyn.f90:73-76.
enum { PC = 0, PPM_UNC = 1, PPM_CON = 2, PPM_NN = 3 };

// Layout of one field in HBM: nlev levels of (ny + 2H) rows of pitch P
// elements; element (i, j, k) of the reference's (is:ie, js:je, 1:K) array
// with i = isd + ii, j = jsd + jj lives at ((k-1)*NYP + jj + H)*P + ii + H + XOFF.
// ii, jj run over [-H, n + H).
struct Geom {
  int nx, ny, L;
  int P;       // row pitch, elements
  int NYP;     // rows per level = ny + 2H
  long long S; // level stride = P * NYP
  __host__ __device__ long long at(int i, int j) const { return (long long)(j + H) * P + (i + H + XOFF); }
  __host__ __device__ long long at(int i, int j, int k) const { return (long long)k * S + at(i, j); }
};

// Constants of init_sw_dyn (src/mod_sw_dyn.f90:961-1021) and the step.
struct Consts {
  double rdx, rdy, rdx2, rdy2, rdx2rdy2, rA;
  double vdx, vdy;        // vortdamp_xcoeff, vortdamp_ycoeff
  double divdamp;         // divdamp_coeff = (c_div dx dy)^2
  double coriolis, gravity;
  double ptop, pk_top;    // Ak(1) and Ak(1)**kappa
  double dt, dtdx, dtdy;  // per call: dtdx = dt*rdx, dtdy = dt*rdy
};

// How the kernels that pass over whole rows share them: groups of 1 << lg threads,
// each a row or one of its pieces of len points.  A group's threads fit the row
// (their last round is not mostly empty), and rows too few to fill the GPU are cut
// up.  With 64 threads a row whatever its width (256 in the finite check), four
// fields out of 16x2048x64 took 98 us, in 113 and the check 217, of 7x4096x20 46, 53
// and 79; so 45, 84, 30 and 15, 42, 9.
struct RowSplit {
  int lg, pieces, len;
};
inline RowSplit row_split(int width, int rows, int lg_most) {
  RowSplit r;
  r.lg = lg_most;
  while (r.lg > 3 && ((width - 1) >> r.lg << r.lg) + (1 << r.lg) > width + width / 2 + 2) --r.lg;
  const int lanes = 1 << r.lg;
  const int most = (width + 4 * lanes - 1) / (4 * lanes);  // four points a thread at least
  const int want = (148 * 2048 / lanes + rows - 1) / rows;  // a piece to every group the GPU holds
  r.pieces = want < most ? want : most;
  r.len = ((width + r.pieces - 1) / r.pieces + lanes - 1) / lanes * lanes;
  r.pieces = (width + r.len - 1) / r.len;
  return r;
}

// Blocks of 256 threads that pass over the rows: blockIdx.y the piece, the row's
// groups along x, at most `most` blocks.
inline dim3 row_grid(const RowSplit& r, int rows, int most) {
  const int per = 256 >> r.lg, nb = (rows + per - 1) / per, cap = most / r.pieces > 0 ? most / r.pieces : 1;
  return dim3(nb < cap ? nb : cap, r.pieces);
}

// f(the group's lg as a constant)
template <typename F>
inline cudaError_t with_lg(const RowSplit& r, F&& f) {
  if (r.lg <= 3) return f(std::integral_constant<int, 3>{});
  if (r.lg == 4) return f(std::integral_constant<int, 4>{});
  if (r.lg == 5) return f(std::integral_constant<int, 5>{});
  if (r.lg == 6) return f(std::integral_constant<int, 6>{});
  return f(std::integral_constant<int, 8>{});
}

// Status words shared by every kernel of a context.
struct Status {
  int nonfinite_step;   // a non-finite prognostic value left the D-grid step
  int nonfinite_remap;  // ... or the vertical remap
  int nonfinite_check;  // standalone stability check
  int fallback_pairs;   // columns whose remap used the all-pairs search
  int radiation_range;  // a radiation table lookup left its table
};

// Hybrid coordinate of the vertical remap (src/mod_remap.f90:57-71).
struct RemapArgs {
  const double* ak;  // device, nlay+1 entries (k = 1..nlay+1 at index k-1)
  const double* bk;
  double ptop, pk_top;
};

// std::min/std::max semantics (return the first argument on ties), so that
// signed zeros behave exactly as in the host restatement.
template <typename T> __device__ __forceinline__ T mn(T a, T b) { return (b < a) ? b : a; }
template <typename T> __device__ __forceinline__ T mx(T a, T b) { return (a < b) ? b : a; }
template <typename T> __device__ __forceinline__ T mn3(T a, T b, T c) { return mn(mn(a, b), c); }
template <typename T> __device__ __forceinline__ T mx3(T a, T b, T c) { return mx(mx(a, b), c); }
__device__ __forceinline__ double cpsign(double a, double b) { return copysign(a, b); }
__device__ __forceinline__ float cpsign(float a, float b) { return copysignf(a, b); }
__device__ __forceinline__ double fab(double a) { return fabs(a); }
__device__ __forceinline__ float fab(float a) { return fabsf(a); }

// Division by the constants 3 and 12 of the PPM formulas
// (src/mod_sw_dyn.f90:878-879,899) and by 6 of the remap's overlaps, correctly rounded like an IEEE
// division: q = x*RN(1/b) is within one ulp of x/b, the remainder
// r = x - q*b is exact in one FMA, and RN(q + r*RN(1/b)) is the correctly
// rounded quotient (P. Markstein, IBM J. Res. Dev. 34(1), 1990).  Zeros,
// infinities, NaN and magnitudes near the ends of the exponent range take
// the IEEE division.
static __device__ __noinline__ double div_ieee(double x, double b) { return x / b; }
template <int B> __device__ __forceinline__ double div_const(double x) {
  constexpr double r = 1.0 / B;  // RN(1/B)
  double a = fabs(x);
  if (!(a > 0x1p-960 && a < 0x1p1000)) return div_ieee(x, (double)B);
  double q = x * r;
  double e = __fma_rn(-q, (double)B, x);
  return __fma_rn(e, r, q);
}
// The mixed form's FP32 sweeps need no correctly rounded quotient: a
// multiplication by the rounded reciprocal.
template <int B> __device__ __forceinline__ float div_const(float x) { return x * (1.0f / B); }

}  // namespace atm
