// Host check of nr_scan_bounds (modpath-rw_gb300/csrc/nrscan.cuh): the measure
// |f0 f2 / f1^2| evaluated in FP64 as the solve evaluates it lies within the
// bounds wherever there are bounds -- over random velocities, gradients,
// drifts, dispersion terms, distances and times of many magnitudes, among
// them residuals and derivatives that nearly cancel, gradients on both sides
// of the exponential form's threshold, and values past the FP32 range.
// Prints "ok <with bounds> <tried>"; exit status 1 on a violation.
#include <cstdio>
#include <random>

#include "nrscan.cuh"

using namespace mprw;

int main() {
  std::mt19937_64 g(12345);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  auto mag = [&](double lo, double hi) { return std::pow(10.0, lo + (hi - lo) * U(g)) * (U(g) < 0.5 ? -1.0 : 1.0); };
  long long with = 0, tried = 0, bad = 0;
  for (int i = 0; i < 4000000; ++i) {
    const int kind = i % 8;
    double v = mag(-4, 2), dvdx = mag(-6, 1), divD = mag(-6, 0), dB = mag(-4, 1), dI = mag(-6, 1);
    const double t = std::fabs(mag(kind == 1 ? -12 : -9, kind == 2 ? 3 : 0));
    if (kind == 3) dvdx = mag(-13, -8);
    if (kind == 4) { v = mag(-30, 30); dB = mag(-30, 30); dvdx = mag(-30, 3); dI = mag(-30, 30); }
    const double s = std::sqrt(t);
    const bool grad = std::fabs(dvdx) > 1.0e-10;
    const double e = std::exp(dvdx * t), adv = grad ? v * (e - 1.0) / dvdx : v * t;
    if (kind == 5) dI = (adv + divD * t + dB * s) * (1.0 + mag(-9, -3));  // near the root
    if (kind == 6) divD = -(v * e + 0.5 * dB / s) * (1.0 + mag(-9, -3));  // a flat residual
    if (kind == 7) dB = dvdx * v * e * 4.0 * t * s * (1.0 + mag(-9, -3)); // no curvature
    const double q = dB / s, f0 = adv + divD * t + dB * s - dI, f1 = v * e + divD + 0.5 * q;
    const double f2 = dvdx * v * e - 0.25 * (q / t), m = std::fabs(f2 * f0 / (f1 * f1));
    float lo, hi;
    ++tried;
    if (!nr_scan_bounds(nr_scan_setup(v, dvdx, dI, divD, dB, grad), (float)t, lo, hi)) continue;
    ++with;
    if (!((double)lo <= m && m <= (double)hi) && bad++ < 20)
      std::printf("OUTSIDE %d v %a dvdx %a dI %a divD %a dB %a t %a: %a not in [%a, %a]\n", kind, v, dvdx, dI, divD, dB,
                  t, m, (double)lo, (double)hi);
  }
  if (bad) return 1;
  std::printf("ok %lld %lld\n", with, tried);
  return 0;
}
