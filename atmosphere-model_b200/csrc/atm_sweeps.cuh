// Tile building blocks of the adjoint sweep kernels (atm_adjoint.cuh), which
// recompute the forward sweeps of a TX x TY tile of one layer in shared
// memory: the PPM stages -- monotone slopes dqi_mono
// (src/mod_sw_dyn.f90:870-875), edge values (:877-911), fluxes (:802-838) --
// the region loops and the TMA box layouts of each sweep's inputs.
#pragma once

#include <type_traits>

#include "atm_kernels.cuh"
#include "atm_tma.cuh"

namespace atm {

// Edge anomalies of a cell from precomputed monotone slopes.  q points at
// the cell (cell spacing sq), mono at its monotone slope (spacing sm).  The
// raw slope dqi of the cell is recomputed from q exactly as slopes() forms it.
template <typename T, int V>
__device__ __forceinline__ void edges_pre(const T* q, int sq, const T* mono, int sm, T& eL, T& eR) {
  const T q0 = q[0];
  eL = (q[-sq] - q0) * T(0.5) + div_const<3>(mono[-sm] - mono[0]);
  eR = (q[sq] - q0) * T(0.5) + div_const<3>(mono[0] - mono[sm]);
  if (V == PPM_CON || V == PPM_NN) {
    const T d0 = (q[sq] - q[-sq]) * T(0.25);
    const T lim = T(2) * fab(d0);
    eL = -cpsign(mn(lim, fab(eL)), d0);
    eR = +cpsign(mn(lim, fab(eR)), d0);
    if (V == PPM_NN) {
      eL = mx(eL, -q0);
      eR = mx(eR, -q0);
      T a = eR - eL;
      T b = T(-3) * (eR + eL);
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
  }
}

// Flux at the interface between cells i-1 and i with slopes precomputed
// (PPM_UNCONSTRAINED / PPM_NONNEGATIVE): only the upwind cell's edges.
// q and mono point at cell i.
template <typename T, int V>
__device__ __forceinline__ T flux_pre(const T* q, int sq, const T* mono, int sm, T c) {
  T sa = fab(c);
  T k1 = (T(1) - T(2) * sa) * (T(1) - sa);
  T k2 = sa * (sa - T(1));
  T eL, eR;
  if (c > T(0)) {
    edges_pre<T, V>(q - sq, sq, mono - sm, sm, eL, eR);
    return q[-sq] + k1 * eR + k2 * eL;
  }
  edges_pre<T, V>(q, sq, mono, sm, eL, eR);
  return q[0] + k1 * eL + k2 * eR;
}

// Flux with precomputed edges (PPM_CONSTRAINED): q points at cell i
// (spacing sq), eL and eR at its edges (spacing se).
template <typename T>
__device__ __forceinline__ T flux_con_pre(const T* q, int sq, const T* eL, const T* eR, int se, T c) {
  const T eLm = eL[-se], eRm = eR[-se], eL0 = eL[0], eR0 = eR[0];
  if ((T(3) * fab(eL0 + eR0) > fab(eL0 - eR0)) && (T(3) * fab(eLm + eRm) > fab(eLm - eRm)))
    return (c > T(0)) ? q[-sq] : q[0];
  T sa = fab(c);
  T k1 = (T(1) - T(2) * sa) * (T(1) - sa);
  T k2 = sa * (sa - T(1));
  if (c > T(0)) return q[-sq] + k1 * eRm + k2 * eLm;
  return q[0] + k1 * eL0 + k2 * eR0;
}

// Monotone slope of one cell from its neighbours along s.
template <typename T>
__device__ __forceinline__ T slope_at(const T* q, int s) {
  T mono, dqi;
  slopes(q[-s], q[0], q[s], dqi, mono);
  return mono;
}

// 128-byte aligned start of the dynamic shared memory (TMA destinations)
__device__ __forceinline__ unsigned char* smem_base(unsigned char* raw) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 127) & ~uintptr_t(127));
}

// Region loop: body(x, y) for every point of [x0, x0+W) x [y0, y0+Hh).
template <int W, int Hh, typename F>
__device__ __forceinline__ void region(int x0, int y0, F&& body) {
  for (int idx = threadIdx.x; idx < W * Hh; idx += NT) {
    const int y = idx / W;
    const int x = idx - y * W;
    body(x0 + x, y0 + y);
  }
}

// One stage's independent region loops as a single index space: the block's
// threads share the whole stage evenly, where separate region() loops of
// W*H a little above NT points each leave most threads idle in a last
// partial pass.  regions(reg<W1, H1>(x1, y1, body1), reg<W2, H2>(...), ...).
template <int W, int Hh, typename F>
struct Reg {
  static constexpr int N = W * Hh;
  int x0, y0;
  F body;
  __device__ __forceinline__ void at(int idx) const {
    const int y = idx / W;
    body(x0 + idx - y * W, y0 + y);
  }
};
template <int W, int Hh, typename F>
__device__ __forceinline__ Reg<W, Hh, F> reg(int x0, int y0, F body) {
  return Reg<W, Hh, F>{x0, y0, body};
}
template <typename R0, typename... Rs>
__device__ __forceinline__ void reg_dispatch(int idx, const R0& r0, const Rs&... rs) {
  if (idx < R0::N) r0.at(idx);
  else if constexpr (sizeof...(Rs) > 0) reg_dispatch(idx - R0::N, rs...);
}
template <typename... Rs>
__device__ __forceinline__ void regions(const Rs&... rs) {
  constexpr int N = (Rs::N + ...);
  for (int idx = threadIdx.x; idx < N; idx += NT) reg_dispatch(idx, rs...);
}

// Start of a TMA box whose first wanted column is i0, rounded down to a
// 16-byte boundary of the tensor row.
template <typename T>
__device__ __forceinline__ int tma_x0(int i0) {
  constexpr int q = tma_q<T>();
  return ((i0 + H + XOFF) / q) * q - H - XOFF;
}

// ---------------------------------------------------------------- mass ----
// S: element type of the prognostic state (dp, pt, ud, vd), C: of the
// C-grid fields (dpc, ptc, uc, vc), T: the sweep arithmetic.  The FP64 form
// has S = C = T = double; the mixed form keeps the state in double, the
// C-grid fields in float and sweeps in float.
template <typename T, int TX, int TY, bool CGRID, typename S = T, typename C = T>
struct MassL {
  // TMA boxes: dp and pt (state), and the u, v boxes (D winds on the C grid
  // step, C winds on the D grid step)
  using UB = std::conditional_t<CGRID, S, C>;
  static_assert(CGRID || std::is_same_v<C, T>, "the D-grid step sweeps with the C-grid winds' type");
  static constexpr int WD = tma_width<S>(TX + 6), HD = TY + 6;
  static constexpr int WU = tma_width<UB>(CGRID ? TX + 2 : TX + 1), HU = CGRID ? TY + 7 : TY + 6;
  static constexpr int WV = tma_width<UB>(CGRID ? TX + 7 : TX + 6), HV = CGRID ? TY + 2 : TY + 1;
  static constexpr uint32_t tx_bytes =
      (uint32_t)(2 * WD * HD * sizeof(S) + (WU * HU + WV * HV) * sizeof(UB));
  static constexpr size_t boxes = 2 * tma_box_bytes(WD, HD, sizeof(S)) + tma_box_bytes(WU, HU, sizeof(UB)) +
                                  tma_box_bytes(WV, HV, sizeof(UB));
  static constexpr bool NN = !CGRID;
  static constexpr size_t work =
      (CGRID ? box_bytes<T>(TX + 1, TY + 6) + box_bytes<T>(TX + 6, TY + 1) : 0) +  // uc, vc (C grid)
      2 * box_bytes<T>(TX + 6, TY) + 2 * box_bytes<T>(TX, TY + 6) +               // inner sweeps
      2 * box_bytes<T>(TX + 2, TY + 2) +                                         // Laplacians
      2 * box_bytes<T>(TX + 4, TY) + 2 * box_bytes<T>(TX, TY + 4) +               // slopes
      2 * box_bytes<T>(TX + 1, TY) + 2 * box_bytes<T>(TX, TY + 1);                // fluxes
  static constexpr size_t bytes = boxes + work + 128;
};

// ======================================================== C-grid momentum ==
template <typename T, int TX, int TY, typename S = T>
struct CMomL {
  static constexpr int WU = tma_width<S>(TX + 7), HU = TY + 7;   // ud box x in [ox-4, ox+TX+2]
  static constexpr int WV = tma_width<S>(TX + 7), HV = TY + 7;   // vd box x in [ox-3, ox+TX+3]
  static constexpr int WL = tma_width<S>(TX + 3), HL = TY + 3;   // layer-nlay ud, vd
  static constexpr int WP = tma_width<double>(TX + 1), HP = TY + 1;  // pkap, gz at k and k+1
  // all eight input boxes at once (the adjoint kernel's layout)
  static constexpr uint32_t tx_bytes =
      (uint32_t)((WU * HU + WV * HV + 2 * WL * HL) * sizeof(S) + 4 * WP * HP * sizeof(double));
  static constexpr size_t boxes = tma_box_bytes(WU, HU, sizeof(S)) + tma_box_bytes(WV, HV, sizeof(S)) +
                                  2 * tma_box_bytes(WL, HL, sizeof(S)) + 4 * tma_box_bytes(WP, HP, 8);
};

// The layer-nlay A-grid winds at (x, y) from the layer-nlay D-grid winds
// (src/mod_sw_dyn.f90:110-125 at k = nlay), recomputed where they are read.
template <typename T, typename A>
__device__ __forceinline__ void al_winds(const A& udL, const A& vdL, int x, int y, T& ua, T& va) {
  T ub = T(.5) * (udL(x, y) + udL(x - 1, y));
  T ucl = T(.5) * (ub + T(.5) * (udL(x, y + 1) + udL(x - 1, y + 1)));
  ua = T(.5) * (ucl + T(.25) * (udL(x + 1, y) + udL(x, y) + udL(x + 1, y + 1) + udL(x, y + 1)));
  T vb = T(.5) * (vdL(x, y) + vdL(x, y - 1));
  T vcl = T(.5) * (vb + T(.5) * (vdL(x + 1, y) + vdL(x + 1, y - 1)));
  va = T(.5) * (vcl + T(.25) * (vdL(x, y + 1) + vdL(x, y) + vdL(x + 1, y + 1) + vdL(x + 1, y)));
}

// ======================================================== D-grid momentum ==
template <typename T, int TX, int TY, typename S = T, typename C = T>
struct DMomL {
  static_assert(std::is_same_v<C, T>, "the D-grid step sweeps with the C-grid winds' type");
  static constexpr int WU = tma_width<S>(TX + 6), HU = TY + 6;       // ud, vd: [ox-3, ox+TX+2]^2
  static constexpr int WUL = tma_width<T>(TX + 1), HUL = TY + 5;     // uc layer nlay: x [ox, ox+TX], y [oy-3, oy+TY+1]
  static constexpr int WVL = tma_width<T>(TX + 5), HVL = TY + 1;     // vc layer nlay: x [ox-3, ox+TX+1], y [oy, oy+TY]
  static constexpr int WC = tma_width<T>(TX), HC = TY;               // uc, vc of the layer at the outputs
  static constexpr int WP = tma_width<double>(TX + 1), HP = TY + 1;  // pkapb, gzb
  // all ten input boxes at once (the adjoint kernels' layouts)
  static constexpr uint32_t tx_bytes = (uint32_t)(2 * WU * HU * sizeof(S) +
                                                   (WUL * HUL + WVL * HVL + 2 * WC * HC) * sizeof(T) +
                                                   4 * WP * HP * sizeof(double));
  static constexpr size_t boxes = 2 * tma_box_bytes(WU, HU, sizeof(S)) + tma_box_bytes(WUL, HUL, sizeof(T)) +
                                  tma_box_bytes(WVL, HVL, sizeof(T)) + 2 * tma_box_bytes(WC, HC, sizeof(T)) +
                                  4 * tma_box_bytes(WP, HP, 8);
  // slopes of the KE sweeps, later of the vorticity-flux sweeps (one buffer)
  static constexpr size_t slopes_ke = box_bytes<T>(TX + 1, TY + 4) + box_bytes<T>(TX + 4, TY + 1);
  static constexpr size_t slopes_vf = box_bytes<T>(TX, TY + 3) + box_bytes<T>(TX + 3, TY);
  static constexpr size_t slopes = slopes_ke > slopes_vf ? slopes_ke : slopes_vf;
  // edges of the KE sweeps, later of the vorticity-flux sweeps (one buffer)
  static constexpr size_t edges_ke = 2 * box_bytes<T>(TX + 1, TY + 2) + 2 * box_bytes<T>(TX + 2, TY + 1);
  static constexpr size_t edges_vf = 2 * box_bytes<T>(TX, TY + 1) + 2 * box_bytes<T>(TX + 1, TY);
  static constexpr size_t edges = edges_ke > edges_vf ? edges_ke : edges_vf;
};

}  // namespace atm
