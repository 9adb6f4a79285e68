// nrscan.cuh -- bounds in FP32 on the convergence measure of the Newton exit
// time (EXPONENTIAL advection).
//
// The solve first scans seven times, 1e-7 to 1e-1 of the step, for one at
// which the measure g = |f0 f2 / f1^2| is at most one (pr_SetInitialGuess,
// TrackSubCell.F90:2162-2448); nearly every scan runs to the end, and each
// point is an exponential, a root and four quotients in FP64.  What a skipped
// point contributes is only that g is above one there and, should no point be
// below one, which point's g is the least: bounds decide both, and a point
// they do not decide is evaluated.
//
// f0 = adv + divD t + dB sqrt(t) - dI, f1 and f2 its derivatives.  Each term is
// a product of at most eight rounded factors (the exponential's argument is at
// most one, so neither it nor e^x - 1 magnifies its error), below 2e-6 of the term;
// kTerm of the terms' sum bounds a sum's error five times over.
// The FP64 evaluation's e^x - 1 is a difference that keeps 2^-53 of one, a
// bound of its own.  Values out of the plain FP32 range have no bounds.
#pragma once
#include <cmath>

#include "fpbits.cuh"

namespace mprw {

struct NrScan {
  float v, dvdx, length, dI, divD, dB;  // length: v / dvdx
  bool grad;                            // |dvdx| > 1e-10: the exponential form
};

MPRW_FB NrScan nr_scan_setup(double v, double dvdx, double dI, double divD, double dB, bool grad) {
  NrScan q;
  q.v = (float)v;
  q.dvdx = (float)dvdx;
  q.length = grad ? (float)v / (float)dvdx : 0.0f;
  q.dI = (float)dI;
  q.divD = (float)divD;
  q.dB = (float)dB;
  q.grad = grad;
  return q;
}

MPRW_FB bool nr_plain(float x) { return x >= 1e-18f && x <= 1e18f; }

// lo <= g <= hi at time t (the FP64 evaluation's g), or false
MPRW_FB bool nr_scan_bounds(const NrScan &q, float t, float &lo, float &hi) {
  const float kTerm = 1e-5f;
  const float w = q.dvdx * t;
  if (!(t >= 1e-18f && t <= 1e18f && fabsf(w) <= 1.0f)) return false;
  const float em1 = expm1f(w), s = sqrtf(t), r = 1.0f / s;
  const float adv = q.grad ? q.length * em1 : q.v * t;
  const float a1 = q.divD * t, a2 = q.dB * s;
  const float f0 = fabsf(adv + a1 + a2 - q.dI);
  const float e0 = kTerm * (fabsf(adv) + fabsf(a1) + fabsf(a2) + fabsf(q.dI)) + 4e-16f * fabsf(q.length);
  const float b = q.dB * r, ve = q.v * (em1 + 1.0f);
  const float f1 = fabsf(ve + q.divD + 0.5f * b);
  const float e1 = kTerm * (fabsf(ve) + fabsf(q.divD) + 0.5f * fabsf(b));
  const float c2 = q.dvdx * ve, d2 = 0.25f * b * r * r;
  const float f2 = fabsf(c2 - d2), e2 = kTerm * (fabsf(c2) + fabsf(d2));
  if (!(nr_plain(f0) && nr_plain(f1) && nr_plain(f2) && f0 > e0 && f1 > e1 && f2 > e2)) return false;
  const float il = 1.0f / (f1 + e1), ih = 1.0f / (f1 - e1);
  lo = (f2 - e2) * il * ((f0 - e0) * il) * (1.0f - kTerm);
  hi = (f2 + e2) * ih * ((f0 + e0) * ih) * (1.0f + kTerm);
  return true;
}

}  // namespace mprw
