// Launchers of the FP64 adjoint kernels (atm_adj_march.cuh, atm_adjoint.cuh).
// Compiled with --fmad=false like the FP64 form: the adjoint kernels recompute
// the forward's intermediates with the forward's exact operations, so every
// limiter and upwind branch is taken as in the forward step.
#include "atm_adj_march.cuh"
#include "atm_adjoint.cuh"
#include "atm_remap_adj.cuh"
#include "atm_ops.h"
#include "atm_strips.h"

namespace atm {
namespace {

// Whole fields copied or cleared, one launch for all of a stage's (blockIdx.y the
// field): the tape and the scratch of a step of a small domain took twenty
// copies and clears of a few microseconds each (gradient at 64x64x20: 2.68 -> 2.19 ms a pass).
template <bool COPY>
__global__ void __launch_bounds__(256) k_fields(FieldList f) {
  stream_order();
  double* d = f.d[blockIdx.y];
  const double* q = f.s[blockIdx.y];
  const long long n = f.n[blockIdx.y], t0 = blockIdx.x * 256LL + threadIdx.x, step = gridDim.x * 256LL;
  if ((((size_t)d | (COPY ? (size_t)q : 0)) & 15) == 0) {  // pairs (a tape is where the caller put it)
    double2* d2 = (double2*)d;
    const double2* q2 = (const double2*)q;
#pragma unroll 4
    for (long long i = t0; i < n / 2; i += step) d2[i] = COPY ? q2[i] : make_double2(0., 0.);
    if ((n & 1) && t0 == 0) d[n - 1] = COPY ? q[n - 1] : 0.;
  } else {
#pragma unroll 4
    for (long long i = t0; i < n; i += step) d[i] = COPY ? q[i] : 0.;
  }
}

// strips of a marching reverse over w x h points, `warm` rows beside the strip's own
inline StripPlan adj_strips(int w, int h, int layers, int out, int warm, int most = 128) {
  return plan_strips(w, h, layers, out, warm, 3 * MWARPS, most);
}

}  // namespace

static dim3 fields_grid(const FieldList& f) {
  long long n = 0;
  for (int i = 0; i < f.nf; ++i) n = f.n[i] > n ? f.n[i] : n;
  const long long b = (n + 2047) / 2048;  // eight elements a thread, up to four blocks an SM and field
  return dim3((unsigned)(b < 592 ? (b > 0 ? b : 1) : 592), f.nf);
}
cudaError_t fields_copy(const FieldList& f, cudaStream_t s) {
  size_t low = 0;
  for (int i = 0; i < f.nf; ++i) low |= (size_t)f.d[i] | (size_t)f.s[i];
  if (low & 7) {  // a tape that is not on a multiple of eight bytes
    for (int i = 0; i < f.nf; ++i) {
      const cudaError_t e = cudaMemcpyAsync(f.d[i], f.s[i], (size_t)f.n[i] * 8, cudaMemcpyDeviceToDevice, s);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  return f.nf ? launch(k_fields<true>, fields_grid(f), 256, 0, s, f) : cudaSuccess;
}
cudaError_t fields_zero(const FieldList& f, cudaStream_t s) {
  return f.nf ? launch(k_fields<false>, fields_grid(f), 256, 0, s, f) : cudaSuccess;
}

cudaError_t adj_mass(const Geom& g, const Consts& c, const double* dp, const double* pt, const double* u,
                     const double* v, const double* dpo, const double* pto, const double* lam_dpo,
                     const double* lam_pto, double* lam_dp, double* lam_pt, double* lam_u, double* lam_v, int lo,
                     int hi, bool cgrid, cudaStream_t s, int part) {
  const MassAdjArgs a{dp, pt, u, v, dpo, pto, lam_dpo, lam_pto, lam_dp, lam_pt, lam_u, lam_v};
  const int w = g.nx - lo + hi, h = g.ny - lo + hi;
  const bool xb = part == 1;
  // the x kernels take few rows beside a strip's own, and short strips spread their
  // adjoint sums, whose contention plan_strips does not know: heights of at most 20 rows
  // (C / D mass, us, against up to 128: 512x512x32 359 / 474, 375 / 513; 301x203x40 140 /
  // 170, 154 / 176; 1024x1024x8 338 / 441, 408 / 539; 700x600x20 338 / 465, 422 / 578;
  // 100x3000x10 158 / 252, 189 / 267; 512x512x64 686 / 910, 692 / 934; 192x160x48 105 / 113,
  // 101 / 113; the one loss of sixteen grids 90x90x100 70 / 72, 62 / 70).  14 or 32 rows
  // are within 5% of it on most.
  const StripPlan p = xb ? adj_strips(w, h, g.L, MOUT, 4, 20) : adj_strips(w, h, g.L, YOUT_MASS, 11);
  const int sm = p.threads / MW * mass_adj_smem(cgrid, xb);
  auto run = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               MWARPS * mass_adj_smem(cgrid, xb));
    if (e != cudaSuccess) return e;
    return launch(kernel, p.grid, p.threads, sm, s, g, c, a, lo, hi, p.rows);
  };
  if (xb) return cgrid ? run(k_mass_adj_x<true>) : run(k_mass_adj_x<false>);
  return cgrid ? run(k_mass_adj_y<true>) : run(k_mass_adj_y<false>);
}

// shared memory of a warp's row ring (at most 32 KB a block)
constexpr int ADJ_RING7 = RowRing<7, 4>::bytes, ADJ_RING8 = RowRing<8, 4>::bytes;

cudaError_t adj_c_mom(const Geom& g, const Consts& c, const double* ud, const double* vd, const double* lam_uc,
                      const double* lam_vc, double* lam_ud, double* lam_vd, double* lam_w, double* lam_uc1,
                      double* lam_vc1, double* lam_nlay, cudaStream_t s) {
  const CMomAdjArgs a{ud, vd, lam_uc, lam_vc, lam_ud, lam_vd, lam_w, lam_uc1, lam_vc1, lam_nlay, lam_nlay + g.S};
  FieldList z;
  z.add(lam_w, nullptr, g.S * g.L);
  z.add(lam_uc1, nullptr, g.S * g.L);
  z.add(lam_vc1, nullptr, g.S * g.L);
  z.add(lam_nlay, nullptr, g.S * 2);
  const cudaError_t e = fields_zero(z, s);
  if (e != cudaSuccess) return e;
  StripPlan p = adj_strips(g.nx, g.ny, g.L, MOUT, 3);
  launch(k_c_mom_adj_x, p.grid, p.threads, p.threads / MW * ADJ_RING7, s, g, c, a, p.rows);
  p = adj_strips(g.nx + 1, g.ny + 1, g.L, YOUT_CMOM, 10);
  launch(k_c_mom_adj_y, p.grid, p.threads, p.threads / MW * ADJ_RING7, s, g, c, a, p.rows);
  const int rows = g.ny + 8 < 65535 ? g.ny + 8 : 65535;
  launch(k_c_mom_adj_fin, dim3((g.nx + 8 + 127) / 128, rows, g.L), 128, 0, s, g, c, a);
  return cudaGetLastError();
}

cudaError_t adj_d_mom(const Geom& g, const Consts& c, const double* ud, const double* vd, const double* uc,
                      const double* vc, const double* lam_udo, const double* lam_vdo, double* lam_ud, double* lam_vd,
                      double* lam_uc, double* lam_vc, cudaStream_t s, int part) {
  const DMomAdjArgs a{ud, vd, uc, vc, lam_udo, lam_vdo, lam_ud, lam_vd, lam_uc, lam_vc};
  if (part == 1) {
    const StripPlan p = adj_strips(g.nx, g.ny, g.L, MOUT, 6);
    launch(k_d_mom_adj_x, p.grid, p.threads, p.threads / MW * ADJ_RING7, s, g, c, a, p.rows);
  } else {
    const StripPlan p = adj_strips(g.nx + 1, g.ny + 1, g.L, YOUT_DMOM, 11);
    launch(k_d_mom_adj_y, p.grid, p.threads, p.threads / MW * ADJ_RING8, s, g, c, a, p.rows);
  }
  return cudaGetLastError();
}

template <bool CGRID>
static cudaError_t column_adj(const Geom& g, const Consts& c, const double* dp, const double* pt, const double* pkap,
                              const double* gz, const double* lam_u, const double* lam_v, double* lam_dp,
                              double* lam_pt, cudaStream_t s) {
  const int n = (g.nx + 4) * (g.ny + 4);
  if (n > column_adj_few(g.L)) {
    auto run = [&](auto kernel) {
      return launch(kernel, (n + 127) / 128, 128, 0, s, g, c, dp, pt, pkap, gz, lam_u, lam_v, lam_dp, lam_pt);
    };
    if (g.L <= 32) return run(k_column_adj_columns<32, CGRID>);
    if (g.L <= 64) return run(k_column_adj_columns<64, CGRID>);
    return run(k_column_adj_columns<MAX_LAYERS, CGRID>);
  }
  const size_t sm = column_adj_smem(g.L);
  const cudaError_t e = remap_smem_attr(k_column_adj<CGRID>, column_adj_smem(MAX_LAYERS));
  if (e != cudaSuccess) return e;
  launch(k_column_adj<CGRID>, (n + 31) / 32, 32 * CADJ_WARPS, sm, s, g, c, dp, pt, pkap, gz, lam_u, lam_v, lam_dp, lam_pt);
  return cudaGetLastError();
}

cudaError_t adj_c_column(const Geom& g, const Consts& c, const double* dp, const double* pt, const double* pkap,
                         const double* gz, const double* lam_uc, const double* lam_vc, double* lam_dp, double* lam_pt,
                         cudaStream_t s) {
  return column_adj<true>(g, c, dp, pt, pkap, gz, lam_uc, lam_vc, lam_dp, lam_pt, s);
}

cudaError_t adj_d_column(const Geom& g, const Consts& c, const double* dp, const double* pt, const double* lam_pk,
                         const double* lam_gz, double* lam_dp, double* lam_pt, cudaStream_t s) {
  return column_adj<false>(g, c, dp, pt, nullptr, nullptr, lam_pk, lam_gz, lam_dp, lam_pt, s);
}

cudaError_t adj_pgf_corners(const Geom& g, const Consts& c, const double* pkapb, const double* gzb,
                            const double* lam_udo, const double* lam_vdo, double* lam_pkb, double* lam_gzb,
                            cudaStream_t s) {
  const int n = (g.nx + 1) * (g.ny + 1);
  launch(k_pgf_adj_corners, dim3((n + 127) / 128, (g.L + PGF_CHUNK - 1) / PGF_CHUNK), 128, 0, s, 
      g, c, pkapb, gzb, lam_udo, lam_vdo, lam_pkb, lam_gzb);
  return cudaGetLastError();
}

cudaError_t adj_corners(const Geom& g, const double* lam_pkb, const double* lam_gzb, double* lam_pk, double* lam_gz,
                        cudaStream_t s) {
  const StripPlan p = plan_strips(g.nx + 4, g.ny + 4, g.L, COUT, 3, CORN_WARPS_SM);
  return launch(k_corners_adj, p.grid, p.threads, p.threads / MW * CORN_SMEM<true>, s, g, lam_pkb, lam_gzb, lam_pk, lam_gz,
                p.rows);
}

cudaError_t adj_ring_fold(const Geom& g, double* const* f, int nf, int K, cudaStream_t s) {
  const int nring = 2 * H * (g.nx + 2 * H) + 2 * H * g.ny;
  double* d[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < nf; ++i) d[i] = f[i];
  launch(k_ring_fold, dim3((nring + 255) / 256, K, nf), 256, 0, s, g, d[0], d[1], d[2], d[3], K);
  return cudaGetLastError();
}

cudaError_t adj_ring_copy(const Geom& g, double* const* dst, double* const* src, int K, int band01, int band23,
                          cudaStream_t s) {
  const int nring = 2 * H * (g.nx + 2 * H) + 2 * H * g.ny;
  launch(k_ring_copy_adj, dim3((nring + 255) / 256, K, 4), 256, 0, s, g, dst[0], dst[1], dst[2], dst[3], src[0], src[1],
                                                                   src[2], src[3], K, band01, band23);
  return cudaGetLastError();
}

// Whether the reverse of a remap of n columns takes a thread a column (beyond 64
// layers always).  Of the energy: from 54 layers one block of the shared-level form
// fills an SM's shared memory, and few layers leave most of a block's warps without
// work, either of which loses on domains of many columns.  Measured on B200, both
// reverses of a remap (us, shared levels / a thread a column; columns in thousands):
// 3 layers 16 101/104, 37 180/165, 590 2630/1815; 8 layers 66 438/480, 147 964/844;
// 16 layers 147 1674/1578; 28 layers 262 4947/4891; 32 layers 147 3119/3023, 262 5401/5503;
// 40 layers 66 2108/2460, 147 4570/3914; 53 layers 66 2830/3283, 147 6184/5204;
// 54 layers 37 2164/2831, 66 3654/3346; 64 layers 262 16752/11369.
// Of the winds, whose blocks are smaller, only with few layers (energy by a thread a column):
// 3 layers 16 104/101, 37 165/147, 590 1815/1055; 6 layers 66 387/344; 8 layers 147 844/806;
// 11 layers 590 4628/4328; 12 layers 590 4749/4725; 16 layers 590 6021/6488.
template <int LM>
static bool remap_adj_columns(int n, int L) {
  if (LM > 64) return true;
  const bool one_block = 2 * (remap_smem(L, 8) + 3328) > 228 * 1024;
  return n > 148 * (L < 10 ? 64 * L : one_block ? 400 : 640);
}

template <int LM>
static cudaError_t remap_energy_adj_lm(const Geom& g, const RemapArgs& ra, const double* dp, const double* pt,
                                       const double* ud, const double* vd, const double* urem, const double* vrem,
                                       const double* gzs, const double* lam_dpo, const double* lam_pto,
                                       const double* lam_udo, const double* lam_vdo, double* lam_dp, double* lam_pt,
                                       double* lam_ud, double* lam_vd, double* lam_ur, double* lam_vr, cudaStream_t s) {
  const int n = g.nx * g.ny;
  if (remap_adj_columns<LM>(n, g.L) && (LM != 32 || g.L <= 28)) {
    launch(k_remap_energy_adj<LM>, (n + 63) / 64, 64, 0, s, g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto,
                                                        lam_udo, lam_vdo, lam_dp, lam_pt, lam_ud, lam_vd, lam_ur, lam_vr);
  } else if constexpr (LM <= 64) {
    const size_t sm = remap_smem(g.L, 8);
    const cudaError_t e = remap_smem_attr(k_remap_energy_adj_split<LM>, remap_smem(LM, 8));
    if (e != cudaSuccess) return e;
    launch(k_remap_energy_adj_split<LM>, (n + RM_LANES - 1) / RM_LANES, RM_LANES * RMA_WARPS, sm, s, 
        g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_udo, lam_vdo, lam_dp, lam_pt, lam_ud, lam_vd, lam_ur,
        lam_vr);
  }
  return cudaGetLastError();
}

template <int LM>
static cudaError_t remap_winds_adj_lm(const Geom& g, const RemapArgs& ra, const double* dp, const double* ud,
                                      const double* vd, const double* lam_ur, const double* lam_vr, double* lam_dp,
                                      double* lam_ud, double* lam_vd, cudaStream_t s) {
  const int n = (g.nx + 2) * (g.ny + 2);
  if (remap_adj_columns<LM>(g.nx * g.ny, g.L) && (LM > 64 || g.L < 12)) {
    launch(k_remap_winds_adj<LM>, dim3((n + 63) / 64, 2), 64, 0, s, g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud,
                                                                lam_vd);
  } else if constexpr (LM <= 64) {
    const size_t sm = remap_smem(g.L, 6);
    const cudaError_t e = remap_smem_attr(k_remap_winds_adj_split<LM>, remap_smem(LM, 6));
    if (e != cudaSuccess) return e;
    launch(k_remap_winds_adj_split<LM>, dim3((n + RM_LANES - 1) / RM_LANES, 2), RM_LANES * RMA_WARPS, sm, s, 
        g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud, lam_vd);
  }
  return cudaGetLastError();
}

cudaError_t adj_remap_energy(const Geom& g, const RemapArgs& ra, const double* dp, const double* pt, const double* ud,
                             const double* vd, const double* urem, const double* vrem, const double* gzs,
                             const double* lam_dpo, const double* lam_pto, const double* lam_udo,
                             const double* lam_vdo, double* lam_dp, double* lam_pt, double* lam_ud, double* lam_vd,
                             double* lam_ur, double* lam_vr, cudaStream_t s) {
  if (g.L <= 32)
    return remap_energy_adj_lm<32>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_udo, lam_vdo, lam_dp,
                                   lam_pt, lam_ud, lam_vd, lam_ur, lam_vr, s);
  if (g.L <= 64)
    return remap_energy_adj_lm<64>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_udo, lam_vdo, lam_dp,
                                   lam_pt, lam_ud, lam_vd, lam_ur, lam_vr, s);
  return remap_energy_adj_lm<MAX_LAYERS>(g, ra, dp, pt, ud, vd, urem, vrem, gzs, lam_dpo, lam_pto, lam_udo, lam_vdo,
                                         lam_dp, lam_pt, lam_ud, lam_vd, lam_ur, lam_vr, s);
}

cudaError_t adj_remap_winds(const Geom& g, const RemapArgs& ra, const double* dp, const double* ud, const double* vd,
                            const double* lam_ur, const double* lam_vr, double* lam_dp, double* lam_ud, double* lam_vd,
                            cudaStream_t s) {
  if (g.L <= 32) return remap_winds_adj_lm<32>(g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud, lam_vd, s);
  if (g.L <= 64) return remap_winds_adj_lm<64>(g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud, lam_vd, s);
  return remap_winds_adj_lm<MAX_LAYERS>(g, ra, dp, ud, vd, lam_ur, lam_vr, lam_dp, lam_ud, lam_vd, s);
}

}  // namespace atm
