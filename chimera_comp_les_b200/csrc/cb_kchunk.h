// Default launch shape of the single-block stage kernels.
#pragma once
#include "cb_stage.cuh"

namespace cb {

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
// CTA (sphere 96x96x128 FP64: segments 1698, k-chunk 13 1135).  For the same
// reason one long wave is worse than several short ones there: 0.7 of a chunk
// is added for the tail (sphere mixed: k-chunk 26, one wave, 596; 9, 442).
inline int default_kchunk(int cols, int nk, int sms, bool mixed, int fl, bool les, bool masked) {
  const long long slots = (long long)sms * (mixed ? 2 : 1);
  double best = 1e300;
  int bkc = nk;
  for (int kc = 1; kc <= nk; kc++) {
    const long long blocks = (long long)cols * ((nk + kc - 1) / kc);
    const double cost = ((double)((blocks + slots - 1) / slots) + (masked ? 0.7 : 0.0)) * (kc + 1.0);
    if (cost < best) { best = cost; bkc = kc; }
  }
  const bool heavy = (fl & FLUX_W5) || (les && !(fl & (FLUX_SIGMA0 | FLUX_SIGMA1)));
  const double seg = (double)((cols * (long long)nk + slots - 1) / slots) + 2.0;
  if (!masked && (mixed ? (!heavy && 1.12 * seg <= best) : seg <= best)) bkc = 0;
  return bkc;
}

}  // namespace cb
