// Launch wrappers of one form of the dynamical core (T = sweep type).
// Included once by atm_fp64.cu (T = double) and once by atm_mixed.cu
// (T = float), which each define ATM_FORM_T and ATM_OPS_NAME.
#pragma once

#include "atm_kernels.cuh"
#include "atm_march.cuh"
#include "atm_ops.h"
#include "atm_remap.cuh"
#include "atm_strips.h"

namespace atm {
namespace {

using T = ATM_FORM_T;  // sweep arithmetic
using S = double;      // prognostic state (dp, pt, ud, vd), both forms
using C = T;           // C-grid fields (dpc, ptc, uc, vc)
// strips of kernel K over [lo, n-1+hi]^2 (six rows fill the windows)
template <int K>
inline StripPlan strips(int lo, int hi, const Geom& g) {
  return plan_strips(g.nx - lo + hi, g.ny - lo + hi, g.L, MOUT, 6, MarchL<T, K>::min_blocks * MWARPS);
}

cudaError_t mass(const Geom& g, const Consts& c, const void* dp, const void* pt, const void* u, const void* v,
                 const double* heat, void* dpo, void* pto, int lo, int hi, int* nonfinite, bool cgrid, cudaStream_t s) {
  if (cgrid) {  // state in, C-grid fields out
    const StripPlan p = strips<MK_CMASS>(lo, hi, g);
    launch(k_mass_m<T, true, S, C>, p.grid, p.threads, p.threads / MW * MASS_SMEM<T, true, S> + FEED_PAD, s, 
        g, c, (const S*)dp, (const S*)pt, (const S*)u, (const S*)v, heat, (C*)dpo, (C*)pto, lo, hi, nonfinite, p.rows);
  } else {  // state and C-grid winds in, state out
    const StripPlan p = strips<MK_DMASS>(lo, hi, g);
    launch(k_mass_m<T, false, S, C>, p.grid, p.threads, p.threads / MW * MASS_SMEM<T, false, S> + FEED_PAD, s, 
        g, c, (const S*)dp, (const S*)pt, (const C*)u, (const C*)v, heat, (S*)dpo, (S*)pto, lo, hi, nonfinite, p.rows);
  }
  return cudaGetLastError();
}

cudaError_t column(const Geom& g, const Consts& c, const void* dpl, const void* ptl, int es, double* pkap, double* gz,
                   int lo, int hi, double* plev, cudaStream_t s) {
  const int n = (g.nx - lo + hi) * (g.ny - lo + hi);
  if (few_columns(n, g.L, es == 4)) {
    const int nb = (n + 31) / 32, nt = 32 * COL_WARPS;
    const size_t sm = (size_t)g.L * 32 * sizeof(double);  // at most 32 KB (128 layers)
    if (es == 8)
      launch(k_column_split<double, FormPow<T>>, nb, nt, sm, s, g, c, (const double*)dpl, (const double*)ptl, pkap, gz, lo,
                                                            hi, plev);
    else
      launch(k_column_split<float, FormPow<T>>, nb, nt, sm, s, g, c, (const float*)dpl, (const float*)ptl, pkap, gz, lo, hi,
                                                           plev);
    return cudaGetLastError();
  }
  if (es == 8)
    launch(k_column<double, FormPow<T>>, (n + 127) / 128, 128, 0, s, g, c, (const double*)dpl, (const double*)ptl, pkap, gz,
                                                                 lo, hi, plev);
  else
    launch(k_column<float, FormPow<T>>, (n + 127) / 128, 128, 0, s, g, c, (const float*)dpl, (const float*)ptl, pkap, gz, lo,
                                                                hi, plev);
  return cudaGetLastError();
}

cudaError_t heating(const Geom& g, const Consts& c, const void* dpl, int es, const double* nf, double* heat,
                    cudaStream_t s) {
  int n = (g.nx + 2 * H) * g.NYP;
  if (!heating_few(n, g.L)) {
    if (es == 8) return launch(k_heating_columns<double>, (n + 63) / 64, 64, 0, s, g, c, (const double*)dpl, nf, heat);
    return launch(k_heating_columns<float>, (n + 63) / 64, 64, 0, s, g, c, (const float*)dpl, nf, heat);
  }
  const int nb = (n + 31) / 32;
  const size_t sm = (size_t)2 * g.L * 32 * sizeof(double), most = (size_t)2 * MAX_LAYERS * 32 * sizeof(double);
  const cudaError_t e = es == 8 ? remap_smem_attr(k_heating<double>, most) : remap_smem_attr(k_heating<float>, most);
  if (e != cudaSuccess) return e;
  if (es == 8) return launch(k_heating<double>, nb, 32 * HEAT_WARPS, sm, s, g, c, (const double*)dpl, nf, heat);
  return launch(k_heating<float>, nb, 32 * HEAT_WARPS, sm, s, g, c, (const float*)dpl, nf, heat);
}

cudaError_t c_mom(const Geom& g, const Consts& c, const void* ud, const void* vd, const double* pkap, const double* gz,
                  void* uc, void* vc, cudaStream_t s) {
  const StripPlan p = strips<MK_CMOM>(0, 0, g);
  launch(k_c_mom_m<T, S, C>, p.grid, p.threads, p.threads / MW * FEED_BYTES<CMOM_NF, 0>, s, 
      g, c, (const S*)ud, (const S*)vd, pkap, gz, (C*)uc, (C*)vc, p.rows);
  return cudaGetLastError();
}

cudaError_t d_mom(const Geom& g, const Consts& c, const void* ud, const void* vd, const void* uc, const void* vc,
                  const double* pkapb, const double* gzb, void* udo, void* vdo, int* nonfinite, cudaStream_t s) {
  const StripPlan p = strips<MK_DMOM>(0, 0, g);
  launch(k_d_mom_m<T, S, C>, p.grid, p.threads, p.threads / MW * FEED_BYTES<DMOM_NF<std::is_same_v<S, T>>, 0>, s, 
      g, c, (const S*)ud, (const S*)vd, (const C*)uc, (const C*)vc, pkapb, gzb, (S*)udo, (S*)vdo, nonfinite, p.rows);
  return cudaGetLastError();
}

template <typename E>
cudaError_t ring_t(const Geom& g, void* const* f, const void* const* src, int nf, int K, bool copy,
                   const RingStatus& w, cudaStream_t s) {
  int nring = 2 * H * (g.nx + 2 * H) + 2 * H * g.ny;
  dim3 grid((nring + 255) / 256, K, nf);
  E* d[4] = {nullptr, nullptr, nullptr, nullptr};
  const E* q[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < nf; ++i) {
    d[i] = (E*)f[i];
    if (src) q[i] = (const E*)src[i];
  }
  if (copy)
    launch(k_ring<E, true>, grid, 256, 0, s, g, d[0], d[1], d[2], d[3], q[0], q[1], q[2], q[3], K, w);
  else
    launch(k_ring<E, false>, grid, 256, 0, s, g, d[0], d[1], d[2], d[3], q[0], q[1], q[2], q[3], K, w);
  return cudaGetLastError();
}

// halo passes of the state fields and of the C-grid fields
cudaError_t ring(const Geom& g, void* const* f, const void* const* src, int nf, int K, bool copy, cudaStream_t s) {
  return ring_t<S>(g, f, src, nf, K, copy, RingStatus{}, s);
}
// the four state fields' halo, with the status words to mapped host memory
cudaError_t ring_report(const Geom& g, void* const* f, int K, const Status* report, Status* host, cudaStream_t s) {
  RingStatus w;
  w.report = report;
  w.host = host;
  return ring_t<S>(g, f, nullptr, 4, K, false, w, s);
}
cudaError_t ring_cg(const Geom& g, void* const* f, int nf, int K, Status* clear, bool remap, cudaStream_t s) {
  RingStatus w;
  w.clear = clear;
  w.remap = remap;
  return ring_t<C>(g, f, nullptr, nf, K, false, w, s);
}

cudaError_t remap_winds(const Geom& g, const RemapArgs& ra, const void* dp, const void* ud, const void* vd, void* urem,
                        void* vrem, int* trace, Status* st, cudaStream_t s) {
  auto run = [&](auto lm) {
    return launch_remap_winds<S, decltype(lm)::value, T>(g, ra, (const S*)dp, (const S*)ud, (const S*)vd, (S*)urem,
                                                         (S*)vrem, trace, st, s);
  };
  if (g.L <= 32) return run(std::integral_constant<int, 32>{});
  if (g.L <= 64) return run(std::integral_constant<int, 64>{});
  return run(std::integral_constant<int, MAX_LAYERS>{});
}

cudaError_t remap_energy(const Geom& g, const RemapArgs& ra, const void* dp, const void* pt, const void* ud,
                         const void* vd, const void* urem, const void* vrem, const double* gzs, void* dpo, void* pto,
                         void* udo, void* vdo, int* trace, Status* st, cudaStream_t s) {
  auto run = [&](auto lm) {
    return launch_remap_energy<S, decltype(lm)::value, FormPow<T>>(
        g, ra, (const S*)dp, (const S*)pt, (const S*)ud, (const S*)vd, (const S*)urem, (const S*)vrem, gzs, (S*)dpo,
        (S*)pto, (S*)udo, (S*)vdo, trace, st, s);
  };
  if (g.L <= 32) return run(std::integral_constant<int, 32>{});
  if (g.L <= 64) return run(std::integral_constant<int, 64>{});
  return run(std::integral_constant<int, MAX_LAYERS>{});
}

cudaError_t check_finite(const Geom& g, const void* const* f, int* flag, cudaStream_t s) {
  RowSplit sp = row_split(g.nx, g.ny * g.L, 8);
  if (sp.lg == 7) sp = row_split(g.nx, g.ny * g.L, 6);
  return with_lg(sp, [&](auto lg) {
    k_check_finite<S, decltype(lg)::value><<<row_grid(sp, g.ny * g.L, 148 * 8), 256, 0, s>>>(g, (const S*)f[0], (const S*)f[1], (const S*)f[2],
                                                                   (const S*)f[3], flag, sp);
    return cudaGetLastError();
  });
}

cudaError_t mass_sum(const Geom& g, const void* dp, double* partial, int nblocks, double* out, cudaStream_t s) {
  k_mass_partial<S><<<nblocks, 256, 0, s>>>(g, (const S*)dp, partial);
  k_mass_final<<<1, 32, 0, s>>>(partial, nblocks, out);
  return cudaGetLastError();
}

cudaError_t to_double(const void* src, double* dst, long long n, cudaStream_t s) {
  k_convert<T, double><<<1184, 256, 0, s>>>((const T*)src, dst, n);
  return cudaGetLastError();
}
cudaError_t from_double(const double* src, void* dst, long long n, cudaStream_t s) {
  k_convert<double, T><<<1184, 256, 0, s>>>(src, (T*)dst, n);
  return cudaGetLastError();
}

}  // namespace

const Ops ATM_OPS_NAME = {(int)sizeof(S), (int)sizeof(C), mass,       column,
                          heating,        c_mom,          d_mom,        ring,       ring_report,   ring_cg,
                          remap_winds,    remap_energy,   check_finite, mass_sum,   to_double,
                          from_double};

}  // namespace atm
