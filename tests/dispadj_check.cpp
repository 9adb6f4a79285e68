// Host measurement of displacement_adjoint's rounding errors
// (modpath-rw_gb300/csrc/dispadj.cuh): root mean squares over random steps,
// against the same formulas in long double, beside those of the formulas with
// every quotient written out in double.  Prints one ratio per output; exit
// status 1 when an output of either is off by more than rounding.
#include <cstdio>
#include <random>

#include "dispadj.cuh"

using namespace mprw;

template <typename T>
struct Step {
  T u[3], xi[3], lt[3], aL, aT, dm, dt, sdt, eps2;
};

template <typename T>
static Disp disp(const Step<T> &n, T &s2, T &r, T &a, T &b, T &k, T &P) {
  s2 = n.u[0] * n.u[0] + n.u[1] * n.u[1] + n.u[2] * n.u[2];
  r = std::sqrt(s2 + n.eps2);
  const T lt = n.aT * r + n.dm, ll = lt + (n.aL - n.aT) * s2 / r;
  a = std::sqrt(T(2) * lt);
  b = std::sqrt(T(2) * ll);
  k = T(2) * (n.aL - n.aT) / (r * (a + b));
  P = n.u[0] * n.xi[0] + n.u[1] * n.xi[1] + n.u[2] * n.xi[2];
  return Disp{(double)s2, (double)r, (double)a, (double)b, (double)k, (double)P, {0, 0, 0}};
}

// the derivatives with their quotients written out
template <typename T>
static void quotients(const Step<T> &n, T q[9]) {
  T s2, r, a, b, k, P;
  disp(n, s2, r, a, b, k, P);
  const T ul = n.u[0] * n.lt[0] + n.u[1] * n.lt[1] + n.u[2] * n.lt[2];
  const T xl = n.xi[0] * n.lt[0] + n.xi[1] * n.lt[1] + n.xi[2] * n.lt[2];
  const T ab = a + b, dA = n.aL - n.aT;
  const T ca = (n.aT / a) / r, cb = (n.aT / r + dA * (T(2) / r - s2 / (r * r * r))) / b;
  const T ck = -k * (T(1) / (r * r) + (ca + cb) / ab);
  const T kL = T(2) / (r * ab) - k * (s2 / (r * b)) / ab;
  const T aT_ = r / a, bT = (r - s2 / r) / b, kT = -T(2) / (r * ab) - k * (aT_ + bT) / ab;
  const T kD = -k * (T(1) / a + T(1) / b) / ab;
  for (int d = 0; d < 3; ++d) {
    const T jv = ca * xl * n.u[d] + ck * P * ul * n.u[d] + k * ul * n.xi[d] + k * P * n.lt[d];
    q[3 + d] = n.dt * n.lt[d];
    q[d] = q[3 + d] + n.sdt * jv;
  }
  q[6] = n.sdt * (kL * P * ul);
  q[7] = n.sdt * (aT_ * xl + kT * P * ul);
  q[8] = n.sdt * (xl / a + kD * P * ul);
}

int main() {
  std::mt19937_64 g(7);
  std::normal_distribution<double> N;
  std::uniform_real_distribution<double> U(0.0, 1.0);
  const int n = 400000;
  double e[2][9] = {{0.0}}, scale[9] = {0.0};
  for (int i = 0; i < n; ++i) {
    Step<double> s;
    const double v = 0.2 * std::exp(0.5 * N(g));
    for (int d = 0; d < 3; ++d) {
      s.u[d] = (d ? 0.3 * v * N(g) : v * (1.0 + 0.2 * N(g)));
      s.xi[d] = N(g);
      s.lt[d] = N(g);
    }
    s.aL = 0.5 * (0.9 + 0.2 * U(g));
    s.aT = 0.05 * (0.9 + 0.2 * U(g));
    s.dm = 4e-4;
    s.dt = 0.05;
    s.sdt = std::sqrt(s.dt);
    s.eps2 = 1e-4;
    Step<long double> l;
    for (int d = 0; d < 3; ++d) {
      l.u[d] = s.u[d];
      l.xi[d] = s.xi[d];
      l.lt[d] = s.lt[d];
    }
    l.aL = s.aL, l.aT = s.aT, l.dm = s.dm, l.dt = s.dt, l.sdt = s.sdt, l.eps2 = s.eps2;
    double s2, r, a, b, k, P, q[9], p[9];
    long double want[9];
    const Disp D = disp(s, s2, r, a, b, k, P);
    displacement_adjoint(D, s.u, s.aL, s.aT, s.xi, s.lt, s.dt, s.sdt, q);
    quotients(s, p);
    quotients(l, want);
    for (int j = 0; j < 9; ++j) {
      const double eq = (double)((long double)q[j] - want[j]), ep = (double)((long double)p[j] - want[j]);
      e[0][j] += eq * eq;
      e[1][j] += ep * ep;
      scale[j] += (double)(want[j] * want[j]);
    }
  }
  for (int j = 0; j < 9; ++j) {
    if (!(std::sqrt(e[0][j] / scale[j]) < 1e-15 && std::sqrt(e[1][j] / scale[j]) < 1e-15)) return 1;
    std::printf("%.4f ", std::sqrt(e[0][j] / e[1][j]));
  }
  std::printf("\n");
  return 0;
}
