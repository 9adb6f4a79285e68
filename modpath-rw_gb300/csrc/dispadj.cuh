// dispadj.cuh -- the adjoint of one step's displacement (the differentiable
// walk, adjoint.cu).
//
// The step moves by (u + G) dt + B xi sqrt(dt), B xi = a xi + kappa P u with
// P = u . xi, s2 = |u|^2, r = sqrt(s2 + eps^2), a = sqrt(2 (aT r + Dm)), b =
// sqrt(2 (aT r + Dm + (aL - aT) s2 / r)), kappa = 2 (aL - aT) / (r (a + b)).
// As a function of u, aL, aT and Dm its transposed derivatives are applied to
// lt: dr = (u . du) / r, da = (aT / a) dr, db = d(ll) / b, dkappa = -kappa (dr / r
// + (da + db) / (a + b)).
//
// A quotient that an output's value rests on is one division of its rounded
// numerator and denominator; reciprocals, a rounding more each, serve what is
// added to larger terms.  (Reciprocals throughout had, with fused multiply-adds,
// errors of dL/du 1.02 and dL/d aT 1.05 times the plain quotients'; these 1.00,
// 1.00 and, of dL/d aL, 0.99.)
// The header also compiles as plain C++ for the host, where the tests measure
// the errors.
#pragma once
#include "fpbits.cuh"

namespace mprw {

MPRW_FB double div_i(double a, double b) { return fb::div_plain(a, b) ? fb::div_core(a, b, 0) : a / b; }

struct Disp {
  double s2, r, a, b, kappa, P, bxi[3];
};

// q = dL/d(u[3], G[3], aL, aT, Dm) of the step, given lt = dL/dx'
MPRW_FB void displacement_adjoint(const Disp &D, const double u[3], double aL, double aT, const double xi[3],
                                  const double lt[3], double dt, double sdt, double q[9]) {
  const double ul = u[0] * lt[0] + u[1] * lt[1] + u[2] * lt[2];
  const double xl = xi[0] * lt[0] + xi[1] * lt[1] + xi[2] * lt[2];
  const double k = D.kappa, P = D.P, s2 = D.s2, r = D.r, a = D.a, b = D.b, ab = a + b, dA = aL - aT;
  // (five divisions, none waiting for another)
  const double ir = div_i(1.0, r), ibr = div_i(1.0, b * r), ib = r * ibr;
  const double Pul = P * ul, Pab = div_i(Pul, ab), s2r = s2 * ir;
  const double ca = div_i(aT, a * r);                          // da = ca (u . du)
  const double cb = (aT + dA * (2.0 - s2r * ir)) * ibr;        // db = cb (u . du)
  // dkappa = -kappa (1 / r^2 + (ca + cb) / (a + b)) (u . du)
  const double ju = ca * xl - k * (ir * ir * Pul + (ca + cb) * Pab), jx = k * ul, jl = k * P;
  const double da_daT = div_i(r, a), db_daT = (r - s2r) * ib;
  const double cL = (2.0 - k * (s2 * ib)) * (ir * Pab);
  const double cT = da_daT * xl - (2.0 * ir + k * (da_daT + db_daT)) * Pab;
  const double ia = da_daT * ir, cD = xl * ia - k * (ia + ib) * Pab;
  for (int d = 0; d < 3; ++d) {
    q[3 + d] = dt * lt[d];
    q[d] = q[3 + d] + sdt * (jl * lt[d] + (jx * xi[d] + ju * u[d]));
  }
  q[6] = sdt * cL;
  q[7] = sdt * cT;
  q[8] = sdt * cD;
}

}  // namespace mprw
