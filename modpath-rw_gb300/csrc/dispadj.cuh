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
// Every output is a quotient of one rounded numerator and one denominator where
// its value rests on it; reciprocals, a rounding more each, serve what is added
// to larger terms.  (Reciprocals throughout had, with fused multiply-adds,
// errors of dL/du 1.02 and dL/d aT 1.05 times the plain quotients'; these 1.00,
// 1.00 and, of dL/d aL, 0.89.)
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
  const double ir = div_i(1.0, r), s2r = s2 * ir;
  const double ca = div_i(aT, a * r);                                // da = ca (u . du)
  const double cb = div_i(aT + dA * (2.0 - s2r * ir), b * r);        // db = cb (u . du)
  const double ck = -k * (ir * ir + div_i(ca + cb, ab));             // dkappa = ck (u . du)
  const double Pul = P * ul, ju = ca * xl + ck * Pul, jx = k * ul, jl = k * P;
  const double da_daT = div_i(r, a), db_daT = div_i(r - s2r, b);
  const double cL = div_i(2.0 - k * div_i(s2, b), r * ab) * Pul;
  const double cT = da_daT * xl - div_i(2.0 * ir + k * (da_daT + db_daT), ab) * Pul;
  const double ia = div_i(1.0, a), ib = div_i(1.0, b);
  const double cD = xl * ia - div_i(k * (ia + ib), ab) * Pul;
  for (int d = 0; d < 3; ++d) {
    q[3 + d] = dt * lt[d];
    q[d] = q[3 + d] + sdt * (jl * lt[d] + (jx * xi[d] + ju * u[d]));
  }
  q[6] = sdt * cL;
  q[7] = sdt * cT;
  q[8] = sdt * cD;
}

}  // namespace mprw
