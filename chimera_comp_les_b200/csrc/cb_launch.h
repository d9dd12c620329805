// Host-side launch interface of the stage kernels (single block and batched)
// and of the mixed form's set-up kernel.
#pragma once
#include <cuda_runtime.h>

#include "cb_common.cuh"
#include "cb_stage.cuh"

namespace cb {

// Grid of a stage-kernel launch: (tile columns in i, in j, k-chunks) for
// kchunk > 0; `slots` CTAs (the resident ones) for the balanced segments of
// kchunk == 0.  by: the tile height of the variant (StageGeo::BY).
inline dim3 stage_grid(const DevCfg &c, int kchunk, int slots, int by = SBY) {
  if (kchunk <= 0) return dim3((unsigned)slots);
  return dim3((c.mx - 2 + SBX - 1) / SBX, (c.my - 2 + by - 1) / by, (c.mz - 2 + kchunk - 1) / kchunk);
}
// k-chunk of a block's stage launches before any autotuning (cb_autotune
// refines it by measurement): `cols` tile columns of nk planes on 1 (FP64) or
// 2 (mixed) resident CTAs per SM.  A chunk's prologue costs about one plane,
// so kc planes cost whole waves x (kc + 1); small blocks take chunks down to
// one plane (32^3 FP64: 44.2 us per stage at k-chunk 4, 30.2 at 2; mixed 30.7
// at 4, 21.0 at 1).  k-chunk 0 (balanced segments) costs an equal share of all
// planes + 2.  FP64, one CTA per SM: taken when that is no more (128^3 MUSCL
// 611 -> 586 us per stage, 64x63x96 238 -> 226; where the model is near
// equal the two are within 1-2 %).  Mixed: two CTAs share an SM and even out
// their own ends, so segments win only by a margin of 12 % in the model
// (128^3 MUSCL 271 -> 261; 160^3 461 -> 484 stays chunked), and not at all
// with WENO5-JS or with both fluxes of the blend on every face (192^3
// WENO5-JS 2180 -> 2480, 128^3 blend 485 -> 503).  Nor with an immersed body
// (masked): its planes cost more, and a segment cannot give them to another
// CTA (sphere 96x96x128 FP64: segments 1698, k-chunk 13 1135).
inline int default_kchunk(int cols, int nk, int sms, bool mixed, int fl, bool les, bool masked) {
  const long long slots = (long long)sms * (mixed ? 2 : 1);
  double best = 1e300;
  int bkc = nk;
  for (int kc = 1; kc <= nk; kc++) {
    const long long blocks = (long long)cols * ((nk + kc - 1) / kc);
    const double cost = (double)((blocks + slots - 1) / slots) * (kc + 1.0);
    if (cost < best) { best = cost; bkc = kc; }
  }
  const bool heavy = (fl & FLUX_W5) || (les && !(fl & (FLUX_SIGMA0 | FLUX_SIGMA1)));
  const double seg = (double)((cols * (long long)nk + slots - 1) / slots) + 2.0;
  if (!masked && (mixed ? (!heavy && 1.12 * seg <= best) : seg <= best)) bkc = 0;
  return bkc;
}
inline int stage_tile_rows(int fl) { return (fl & FLUX_W5) ? SBY_W5 : SBY; }

// Launchers of the stage kernels, defined in cb_stage_parts.cu.  That file is
// compiled once per (form, LES) pair -- the FP64 parity form without FMA
// contraction, the mixed form with it -- and once more for the batched work
// queue, so the many template variants build in parallel.
//
// fl: FLUX bits; nv0: nvert is zero everywhere, the variant without any nvert test
// (time step only); slots: CTAs of the balanced-segment shape (kchunk 0).
template <typename R, bool MIX, bool LES>
struct StageLaunch {
  static cudaError_t attrs();  // shared-memory opt-in of every variant
  static cudaError_t launch(const DevCfg &c, const DevFields &F, int istage, double alfa, double beta, double adt,
                            int kchunk, bool visc, bool rhs_mode, int fl, bool nv0, int slots, cudaStream_t s);
};
// The persistent multi-block work-queue launch (ctas CTAs).
template <typename R, bool MIX, bool LES>
struct BatchLaunch {
  static cudaError_t attrs();
  static cudaError_t launch(const BatchBlock *tab, const int2 *items, int nitems, unsigned *counter, int istage,
                            double alfa, double beta, double adt, bool visc, int fl, bool nv0, int ctas,
                            cudaStream_t s);
};

// Each (form, LES) instantiation is defined in exactly one object, the part
// built with that form's floating-point flags.  Without these declarations a
// part would also instantiate the other parts' launchers (the inline
// dispatchers below name all of them) and compile their kernels with its own
// flags: an FP64 kernel built with FMA contraction, registered beside the
// right one under the same host symbol.
extern template struct StageLaunch<double, false, false>;
extern template struct StageLaunch<double, false, true>;
extern template struct StageLaunch<float, true, false>;
extern template struct StageLaunch<float, true, true>;
extern template struct BatchLaunch<double, false, false>;
extern template struct BatchLaunch<double, false, true>;
extern template struct BatchLaunch<float, true, false>;
extern template struct BatchLaunch<float, true, true>;

inline cudaError_t stage_attrs_all(bool mix) {
  cudaError_t e = mix ? StageLaunch<float, true, true>::attrs() : StageLaunch<double, false, true>::attrs();
  if (e == cudaSuccess) e = mix ? StageLaunch<float, true, false>::attrs() : StageLaunch<double, false, false>::attrs();
  return e;
}
inline cudaError_t launch_stage_any(bool mix, bool les, const DevCfg &c, const DevFields &F, int istage, double alfa,
                                    double beta, double adt, int kchunk, bool visc, bool rhs_mode, int fl, bool nv0,
                                    int slots, cudaStream_t s) {
  if (mix)
    return les ? StageLaunch<float, true, true>::launch(c, F, istage, alfa, beta, adt, kchunk, visc, rhs_mode, fl, nv0, slots, s)
               : StageLaunch<float, true, false>::launch(c, F, istage, alfa, beta, adt, kchunk, visc, rhs_mode, fl, nv0, slots, s);
  return les ? StageLaunch<double, false, true>::launch(c, F, istage, alfa, beta, adt, kchunk, visc, rhs_mode, fl, nv0, slots, s)
             : StageLaunch<double, false, false>::launch(c, F, istage, alfa, beta, adt, kchunk, visc, rhs_mode, fl, nv0, slots, s);
}
inline cudaError_t batch_attrs_all(bool mix) {
  cudaError_t e = mix ? BatchLaunch<float, true, true>::attrs() : BatchLaunch<double, false, true>::attrs();
  if (e == cudaSuccess) e = mix ? BatchLaunch<float, true, false>::attrs() : BatchLaunch<double, false, false>::attrs();
  return e;
}
inline cudaError_t launch_batched_any(bool mix, bool les, const BatchBlock *tab, const int2 *items, int nitems,
                                      unsigned *counter, int istage, double alfa, double beta, double adt, bool visc,
                                      int fl, bool nv0, int ctas, cudaStream_t s) {
  if (mix)
    return les ? BatchLaunch<float, true, true>::launch(tab, items, nitems, counter, istage, alfa, beta, adt, visc, fl, nv0, ctas, s)
               : BatchLaunch<float, true, false>::launch(tab, items, nitems, counter, istage, alfa, beta, adt, visc, fl, nv0, ctas, s);
  return les ? BatchLaunch<double, false, true>::launch(tab, items, nitems, counter, istage, alfa, beta, adt, visc, fl, nv0, ctas, s)
             : BatchLaunch<double, false, false>::launch(tab, items, nitems, counter, istage, alfa, beta, adt, visc, fl, nv0, ctas, s);
}

// FP32 metric vectors (w: filter width, aj, 0) and the FP64 metric divergence
// (sum over directions of h(+1/2) - h(-1/2)) for the mixed form.
cudaError_t launch_mixed_prep(const DevCfg &c, const double *const *met, const double *delta2, const double *aj,
                              float4 *const *met4, double *const *gcl, int grid, cudaStream_t s);
// Compute_eddy_viscosity_LES with constant CS for the mixed form: FP32
// velocity gradients and |S| from the FP32 metric vectors, nu_t into the FP64
// plane nut (interior nodes); qu: the recorded state (nullptr: zero velocity);
// nvert nullptr: no immersed body.  Defined in cb_mixed.cu.
cudaError_t launch_eddy_mixed(const DevCfg &c, const double *const *qu, const float4 *const *met4, const double *nvert,
                              double *nut, int sms, cudaStream_t s);

}  // namespace cb
