// Precision-independent table of the device operations of one form of the
// dynamical core.  atm_fp64.cu fills it for the FP64 form (compiled without
// fused multiply-add so that it matches the FP64 restatement bit for bit),
// atm_mixed.cu for the FP32-sweep form.  Buffers are passed as void* and
// hold the form's sweep type; pressure, pkap and geopotential are double.
#pragma once

#include <cuda_runtime.h>
#include "atm_common.cuh"

namespace atm {

struct Ops {
  int elem;     // bytes of an element of the prognostic state (dp, pt, ud, vd)
  int cg_elem;  // bytes of an element of the C-grid fields (dpc, ptc, uc, vc)
  // C- or D-grid mass/potential-temperature sweep of every layer
  cudaError_t (*mass)(const Geom&, const Consts&, const void* dp, const void* pt, const void* u, const void* v,
                      const double* heat, void* dpo, void* pto, int lo, int hi, int* nonfinite, bool cgrid,
                      cudaStream_t);
  // plev/pkap/gz columns over [lo, n-1+hi]^2 from dp, pt of element size es
  cudaError_t (*column)(const Geom&, const Consts&, const void* dpl, const void* ptl, int es, double* pkap,
                        double* gz, int lo, int hi, double* plev, cudaStream_t);
  cudaError_t (*heating)(const Geom&, const Consts&, const void* dpl, int es, const double* net_flux, double* heat,
                         cudaStream_t);
  cudaError_t (*c_mom)(const Geom&, const Consts&, const void* ud, const void* vd, const double* pkap,
                       const double* gz, void* uc, void* vc, cudaStream_t);
  cudaError_t (*d_mom)(const Geom&, const Consts&, const void* ud, const void* vd, const void* uc, const void* vc,
                       const double* pkapb, const double* gzb, void* udo, void* vdo, int* nonfinite,
                       cudaStream_t);
  // periodic halo fill (copy = false) or ring copy src -> f (copy = true) of
  // nf state fields (ring), the four with the status words to the mapped memory
  // host (ring_report), or C-grid fields (ring_cg, which clears the step's words of
  // clear, and the remap's, where it is not null)
  cudaError_t (*ring)(const Geom&, void* const* f, const void* const* src, int nf, int K, bool copy, cudaStream_t);
  cudaError_t (*ring_report)(const Geom&, void* const* f, int K, const Status* report, Status* host, cudaStream_t);
  cudaError_t (*ring_cg)(const Geom&, void* const* f, int nf, int K, Status* clear, bool remap, cudaStream_t);
  cudaError_t (*remap_winds)(const Geom&, const RemapArgs&, const void* dp, const void* ud, const void* vd,
                             void* urem, void* vrem, int* trace, Status*, cudaStream_t);
  cudaError_t (*remap_energy)(const Geom&, const RemapArgs&, const void* dp, const void* pt, const void* ud,
                              const void* vd, const void* urem, const void* vrem, const double* gzs, void* dpo,
                              void* pto, void* udo, void* vdo, int* trace, Status*, cudaStream_t);
  cudaError_t (*check_finite)(const Geom&, const void* const* f, int* flag, cudaStream_t);
  cudaError_t (*mass_sum)(const Geom&, const void* dp, double* partial, int nblocks, double* out, cudaStream_t);
  // C-grid-type <-> double conversion of whole padded fields
  cudaError_t (*to_double)(const void* src, double* dst, long long n, cudaStream_t);
  cudaError_t (*from_double)(const double* src, void* dst, long long n, cudaStream_t);
};

extern const Ops ops_fp64;
extern const Ops ops_mixed;

// interpolate_to_corners of pkap/gz (double in both forms)
cudaError_t corners(const Geom&, const double* pkap, const double* gz, double* pkapb, double* gzb, cudaStream_t);
cudaError_t corners_gz0(const Geom&, const double* gz, double* gzb, cudaStream_t);  // level 0 of gzb

// x**y and log(x) of the portable math on the device (tests)
cudaError_t device_pow_log(const double* x, double y, double* p, double* l, int n, cudaStream_t);
// p**kappa as the mixed form evaluates it (atm_mixed.cu)
cudaError_t device_kappa_pow(const double* x, double* out, int n, cudaStream_t);

// count of arguments where div_const<3>, <6>, <12> or third differs from IEEE division (tests)
cudaError_t device_div_check(unsigned long long n, unsigned long long seed, unsigned long long* bad, cudaStream_t);
// a bounded mbarrier wait on a barrier nothing completes: *flag = 1 when it gave up
cudaError_t device_wait_timeout(int max_polls, int* flag, cudaStream_t);

// ---- FP64 adjoint (atm_adjoint.cu); lam_* are adjoint fields laid out like
// the fields they belong to, accumulated with +=
// dpo, pto: the new dp and pt the forward sweep wrote; part: 1 the x branch,
// 2 the y branch
cudaError_t adj_mass(const Geom&, const Consts&, const double* dp, const double* pt, const double* u, const double* v,
                     const double* dpo, const double* pto, const double* lam_dpo, const double* lam_pto, double* lam_dp,
                     double* lam_pt, double* lam_u, double* lam_v, int lo, int hi, bool cgrid, cudaStream_t, int part);
// lam_w, lam_uc1, lam_vc1 (nlay levels), lam_nlay (2 levels): scratch
cudaError_t adj_c_mom(const Geom&, const Consts&, const double* ud, const double* vd, const double* lam_uc,
                      const double* lam_vc, double* lam_ud, double* lam_vd, double* lam_w, double* lam_uc1,
                      double* lam_vc1, double* lam_nlay, cudaStream_t);
// without the pressure-gradient force; part: 1 the x branch, 2 the y branch
cudaError_t adj_d_mom(const Geom&, const Consts&, const double* ud, const double* vd, const double* uc,
                      const double* vc, const double* lam_udo, const double* lam_vdo, double* lam_ud, double* lam_vd,
                      double* lam_uc, double* lam_vc, cudaStream_t, int part);
// lam_pkb (levels 1..nlay), lam_gzb = the D grid's pressure-gradient force reversed
cudaError_t adj_pgf_corners(const Geom&, const Consts&, const double* pkapb, const double* gzb, const double* lam_udo,
                            const double* lam_vdo, double* lam_pkb, double* lam_gzb, cudaStream_t);
// columns over [-2, n+1]^2, on the C grid with the pressure-gradient force
cudaError_t adj_c_column(const Geom&, const Consts&, const double* dp, const double* pt, const double* pkap,
                         const double* gz, const double* lam_uc, const double* lam_vc, double* lam_dp,
                         double* lam_pt, cudaStream_t);
cudaError_t adj_d_column(const Geom&, const Consts&, const double* dp, const double* pt, const double* lam_pk,
                         const double* lam_gz, double* lam_dp, double* lam_pt, cudaStream_t);
// lam_pk (levels 1..nlay), lam_gz (2..nlay+1) = the corner interpolation reversed
cudaError_t adj_corners(const Geom&, const double* lam_pkb, const double* lam_gzb, double* lam_pk, double* lam_gz,
                        cudaStream_t);
cudaError_t adj_ring_fold(const Geom&, double* const* f, int nf, int K, cudaStream_t);
cudaError_t adj_ring_copy(const Geom&, double* const* dst, double* const* src, int K, int band01, int band23,
                          cudaStream_t);
cudaError_t adj_remap_energy(const Geom&, const RemapArgs&, const double* dp, const double* pt, const double* ud,
                             const double* vd, const double* urem, const double* vrem, const double* gzs,
                             const double* lam_dpo, const double* lam_pto, const double* lam_udo,
                             const double* lam_vdo, double* lam_dp, double* lam_pt, double* lam_ud, double* lam_vd,
                             double* lam_ur, double* lam_vr, cudaStream_t);
cudaError_t adj_remap_winds(const Geom&, const RemapArgs&, const double* dp, const double* ud, const double* vd,
                            const double* lam_ur, const double* lam_vr, double* lam_dp, double* lam_ud, double* lam_vd,
                            cudaStream_t);

// the persistent ensemble kernel of the mixed form (atm_ensemble.cuh): its
// largest cooperative grid on the current device, and one launch of a plan
struct EnsPlan;
int ensemble_max_blocks();
cudaError_t ensemble_launch(const EnsPlan& plan, int blocks, cudaStream_t);

// whether n columns of L layers leave a column pass of one thread a column with so
// few blocks of 128 a multiprocessor that levels are better shared.  Measured on B200
// (us, shared levels / a thread a column; columns in thousands): FP64 fields 3 layers 31
// 8/10, 66 13/10, 32 layers 31 23/35, 66 40/39, 160 78/68; 64 layers 66 76/74; 128 layers
// 31 96/112, 66 155/141; 301x203x40 44/50.  FP32 fields (single) 20 layers 66 20/21, 96 25/23; 64 layers
// 66 43/47, 96 63/56; 128 layers 31 66/72, 66 112/93.
inline bool few_columns(long long n, int L, bool single) {
  return n <= 148LL * (L > 96 ? 400 : single && L > 8 ? 512 : 448);
}

// whole fields: destinations, sources (copies), elements
struct FieldList {
  double* d[10];
  const double* s[10];
  long long n[10];
  int nf = 0;
  void add(double* dst, const double* src, long long elems) {
    d[nf] = dst;
    s[nf] = src;
    n[nf++] = elems;
  }
};
cudaError_t fields_copy(const FieldList&, cudaStream_t);
cudaError_t fields_zero(const FieldList&, cudaStream_t);

// largest number of layers the vertical remap supports
constexpr int MAX_LAYERS = 128;

}  // namespace atm
