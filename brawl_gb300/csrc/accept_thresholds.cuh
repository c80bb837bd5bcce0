// accept_thresholds.cuh -- the uphill decision as two integer compares.
#pragma once

#include <climits>

#include "chain_engine.cuh"

namespace brawl {

// Log-domain acceptance thresholds: the uphill decision as two integer
// compares of the fixed-point energy change against bounds taken from the
// acceptance word (no exponential of the change).  The reference accepts an uphill move iff u < exp(-beta dE_ref)
// (src/metropolis.F90:802), i.e. iff t > beta dE_ref log2(e) with
// t = -log2(u) = 32 - log2(w) for u = w 2^-32.  With k = beta 2^-S log2(e)
// and the fixed-point dE within band quanta of dE_ref 2^S, the move is
// certainly accepted when dE < (t - e)/k - band and certainly rejected when
// dE > (t + e)/k + band, where e = 1e-4 bounds the error of t as computed
// here (float conversion of w, lg2.approx, the subtraction: together below
// 2e-5 on [0, 32]) with room to spare.  The float products carry a further
// relative 1e-6 and the thresholds are rounded towards the undecided side.
// Between the two, and for w = 0, the exact tier decides.  For beta >= 0 only: with
// any other the band holds every change (set_beta, capi.cu) and these decide none.
struct AcceptThresholds {
  int acc_below;  // dE < acc_below: accepted
  int rej_above;  // dE > rej_above: rejected
};

__device__ __forceinline__ AcceptThresholds accept_thresholds(uint32_t w, float inv_k, float band_f) {
  AcceptThresholds T;
  float lw;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lw) : "f"(__uint2float_rn(w)));
  const float t = 32.0f - lw;
  const float a = __fmul_rn(__fmul_rn(t - 1e-4f, inv_k), 1.0f - 1e-6f) - band_f - 1.0f;
  const float r = __fmul_rn(__fmul_rn(t + 1e-4f, inv_k), 1.0f + 1e-6f) + band_f + 1.0f;
  // fixed-point changes stay within +-2^30: clamp before converting
  T.acc_below = w == 0u ? INT_MIN : __float2int_rd(fminf(a, 1073741824.0f));
  T.rej_above = w == 0u ? INT_MAX : __float2int_ru(fminf(r, 2147483520.0f));
  return T;
}

}  // namespace brawl
