// step.cu -- the random-walk particle-tracking step kernel.
//
// One persistent kernel advances every particle to the end of the tracking
// interval.  Each lane runs a flat state machine, one time-loop pass per
// iteration of its main loop:
//   fetch particle -> release checks -> enter cell (stage the cell record in
//   shared memory, entry checks) -> time-loop passes -> exit / stop / store
// so lanes of a warp stay on the common step body no matter which particle,
// cell or phase each one is in.  Particles are taken from an atomic queue in
// cell-sorted order (perm[]), which keeps the records a warp reads in cache.
//
// Per-pass logic restates pr_ExecuteRandomWalkParticleTracking
// (TrackSubCell.F90:812-1373) with the quadratic exit-face solver of the
// EULERIAN advection model (TrackSubCell.F90:1576-1892); the cell-to-cell
// logic restates pr_RWPTrackPath (ParticleTrackingEngine.f90:1051-1254),
// TrackCell (TrackCell.f90:375-669) and ConvertFromNeighbor
// (RectangularGridDisMf6.f90:50-108).  Interpolants are evaluated from the
// monomial coefficients the prep kernel stores, with fused multiply-adds.
#include <cstddef>

#include "mprw_common.cuh"
#include "mprw_kernels.cuh"
#include "nrscan.cuh"

namespace mprw {

// Shared-memory view of one lane's record: field f at sm[f].
enum : int {
  F_V1 = 0, F_DV = 3, F_D = 6, F_INVD = 9, F_DIV = 12, F_VB = 33,
  F_AL = 57, F_AT = 58, F_DM = 59, F_2R = 60, F_V2 = 61, F_ALV = 64, F_ATV = 65, NFIELDS = 66
};

template <typename R>
struct Lane {
  R *p;
  int stride;  // threads of the block
  __device__ __forceinline__ R operator()(int f) const { return p[f]; }
};

// Tests against the constants 0, 1/2 and 1 and the time compares: native in
// the FP32 kernel, from the IEEE-754 bit patterns in the FP64 kernel (the
// same decisions for every input; fpbits.cuh).  Where a site reads
// `sizeof(R) == 8 ? <bit-pattern form> : <compare>`, the FP32 kernel keeps
// its compare written as before: it is latency-bound at 80 registers, and
// every reshaping of its compares measured slower.
template <typename R>
__device__ __forceinline__ bool above1(R v) { return v > R(1); }
template <>
__device__ __forceinline__ bool above1<double>(double v) { return fb::above1(v); }
template <typename R>
__device__ __forceinline__ bool below0(R v) { return v < R(0); }
template <>
__device__ __forceinline__ bool below0<double>(double v) { return fb::below0(v); }
template <typename R>
__device__ __forceinline__ bool above0(R v) { return v > R(0); }
template <>
__device__ __forceinline__ bool above0<double>(double v) { return fb::above0(v); }
template <typename R>
__device__ __forceinline__ bool is0(R v) { return v == R(0); }
template <>
__device__ __forceinline__ bool is0<double>(double v) { return fb::is0(v); }
template <typename R>
__device__ __forceinline__ bool nonneg(R v) { return v >= R(0); }
template <>
__device__ __forceinline__ bool nonneg<double>(double v) { return fb::nonneg(v); }
template <typename R>
__device__ __forceinline__ bool abs_above_half(R v) { return fabs(v) > R(0.5); }
template <>
__device__ __forceinline__ bool abs_above_half<double>(double v) { return fb::abs_above_half(v); }
// |a b| > 1/2: in the FP64 kernel without the product (the jump limiter's test
// of every pass; 54.7 -> 52.3 ms on the same workload, with the exit steps
// formed on two axes 51.8)
template <typename R>
__device__ __forceinline__ bool over_half(R a, R b) { return fabs(a * b) > R(0.5); }
template <>
__device__ __forceinline__ bool over_half<double>(double a, double b) { return fb::prod_above_half(a, b); }
template <typename R>
__device__ __forceinline__ bool out01(R v) { return v > R(1) || v < R(0); }
template <>
__device__ __forceinline__ bool out01<double>(double v) { return fb::out01(v); }
template <typename R>
__device__ __forceinline__ bool is1(R v) { return v == R(1); }
template <>
__device__ __forceinline__ bool is1<double>(double v) { return fb::is1(v); }
// a < b for a, b > 0 (not NaN)
template <typename R>
__device__ __forceinline__ bool pos_lt(R a, R b) { return a < b; }
template <>
__device__ __forceinline__ bool pos_lt<double>(double a, double b) { return fb::pos_lt(a, b); }
// Square root and quotient of the FP64 kernels: on the integer pipe (the same
// bits; the operator, out of line, outside the plain normal range).  A pass
// takes about six roots and four quotients per warp, eight FP64 instructions
// each, on the pipe that bounds the kernel (78 % active before).  The first
// 10-day interval of 200,000 particles in the lognormal slab: 6.80 -> 6.20 ms,
// FP64 pipe 70 %; with the exit solves' operands in shared memory 5.62 ms, 75 %.
__device__ __noinline__ double sqrt_op(double x) { return sqrt(x); }
__device__ __noinline__ double div_op(double a, double b) { return a / b; }
template <typename R>
__device__ __forceinline__ R sqrt_r(R x) { return sqrt(x); }
// (out of line: the FP64 kernels are longer than the instruction caches and
// wait for them in one slot of four; 1,000,000 particles, three 10-day
// intervals 50.8 -> 50.0 ms, EXPONENTIAL 31.3 -> 30.0)
template <>
__device__ __noinline__ double sqrt_r<double>(double x) {
  return fb::sqrt_plain(x) ? fb::sqrt_core(x) : sqrt_op(x);
}
__device__ __forceinline__ double div_r(double a, double b) {
  return fb::div_plain(a, b) ? fb::div_core(a, b, 0) : div_op(a, b);
}
using fb::eq_any;
using fb::lt_any;
using fb::past_end;

// A lane's record in shared memory: the cell record's first NFIELDS values as
// they are (and, in FP32, two more words), kRecBytes apart -- an odd number of
// 16-byte units, so that 16-byte reads of one field pair by all lanes meet no
// bank twice.
static_assert(NFIELDS == 66, "the record's leading fields");
template <typename R>
constexpr int kRecUnits = sizeof(R) == 8 ? 33 : 17;
template <typename R>
constexpr int kRecStride = kRecUnits<R> * 16 / (int)sizeof(R);
// The copies take the record's bytes as they lie, so the fields' numbers are
// its layout.
template <typename R>
constexpr bool layout_is_the_records() {
  using C = CellRec<R>;
  constexpr size_t r = sizeof(R);
  return offsetof(C, v1) == F_V1 * r && offsetof(C, dv) == F_DV * r && offsetof(C, d) == F_D * r &&
         offsetof(C, inv_d) == F_INVD * r && offsetof(C, div) == F_DIV * r && offsetof(C, vb) == F_VB * r &&
         offsetof(C, aL) == F_AL * r && offsetof(C, aT) == F_AT * r && offsetof(C, dm) == F_DM * r &&
         offsetof(C, two_over_r) == F_2R * r && offsetof(C, v2) == F_V2 * r && offsetof(C, aLV) == F_ALV * r &&
         offsetof(C, aTV) == F_ATV * r && sizeof(C) % 16 == 0 && alignof(C) >= 16 &&
         sizeof(C) >= 16 * kRecUnits<R> && NFIELDS * r <= 16 * kRecUnits<R>;
}
static_assert(layout_is_the_records<double>() && layout_is_the_records<float>(), "CellRec moved: renumber the fields");

// Asynchronous copies, all in flight at once and without a register each;
// stage_wait before the first read.  Every warp waits here for its entering
// lanes in nine iterations of ten: loads and stores of one field column per
// lane (17 or 33 loads, 66 stores, in batches), after the entry checks, held
// MIXED at 12.5 ms and FP64 at 50.9 ms over three 10-day intervals of 1,000,000
// particles in the lognormal slab; these, issued before the checks, 10.7 and
// 50.5.
template <typename R>
__device__ __forceinline__ void stage_record(const CellRec<R> *__restrict__ recs, int32_t c, R *sm) {
  const char *src = reinterpret_cast<const char *>(recs + c);
  const unsigned dst = (unsigned)__cvta_generic_to_shared(sm);
#pragma unroll
  for (int q = 0; q < kRecUnits<R>; ++q)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * q), "l"(src + 16 * q) : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// N consecutive fields from a 16-byte boundary-aligned window (fields before
// base in the first unit and after the last are dropped)
template <typename R, int BASE, int N>
__device__ __forceinline__ void fields(const Lane<R> &F, R (&v)[N]) {
  constexpr int K = 16 / (int)sizeof(R), U0 = BASE / K, U1 = (BASE + N + K - 1) / K;
#pragma unroll
  for (int u = U0; u < U1; ++u) {
    if constexpr (sizeof(R) == 8) {
      const double2 q = reinterpret_cast<const double2 *>(F.p)[u];
      const double t[2] = {q.x, q.y};
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (u * K + k >= BASE && u * K + k < BASE + N) v[u * K + k - BASE] = t[k];
    } else {
      const float4 q = reinterpret_cast<const float4 *>(F.p)[u];
      const float t[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (u * K + k >= BASE && u * K + k < BASE + N) v[u * K + k - BASE] = t[k];
    }
  }
}

template <typename R>
__device__ __forceinline__ R tril(const R *c, R x, R y, R z, R xy, R xz, R yz, R xyz) {
  R a = c[0];
  a = fma(c[1], x, a);
  a = fma(c[2], y, a);
  a = fma(c[3], z, a);
  a = fma(c[4], xy, a);
  a = fma(c[5], xz, a);
  a = fma(c[6], yz, a);
  a = fma(c[7], xyz, a);
  return a;
}

template <typename R>
__device__ __forceinline__ R divc(const R *c, R x, R y, R z, R xy, R xz, R yz) {
  R a = c[0];
  a = fma(c[1], x, a);
  a = fma(c[2], y, a);
  a = fma(c[3], z, a);
  a = fma(c[4], xy, a);
  a = fma(c[5], xz, a);
  a = fma(c[6], yz, a);
  return a;
}

// The step's standard normals, the reference's Irwin-Hall(12) distribution
// in both paths, from the same 3 Philox blocks per normal: FP64 exact, MIXED
// rounded to FP32 (the two precisions share their random numbers).
template <typename R>
struct Normals;
template <>
struct Normals<double> {
  __device__ __forceinline__ static void draw(int ndim, uint64_t seed, uint64_t id, uint64_t &ctr, double &r0,
                                              double &r1, double &r2) {
    r0 = normal_ih12(seed, id, ctr);
    r1 = (ndim > 1) ? normal_ih12(seed, id, ctr) : 0.0;
    r2 = (ndim > 2) ? normal_ih12(seed, id, ctr) : 0.0;
  }
};
template <>
struct Normals<float> {
  __device__ __forceinline__ static void draw(int ndim, uint64_t seed, uint64_t id, uint64_t &ctr, float &r0,
                                              float &r1, float &r2) {
    r0 = normal_ih12_f32(seed, id, ctr);
    r1 = (ndim > 1) ? normal_ih12_f32(seed, id, ctr) : 0.0f;
    r2 = (ndim > 2) ? normal_ih12_f32(seed, id, ctr) : 0.0f;
  }
};

// pr_DisplacementRandomDischarge (3-D :2821-2928, 2-D :2931-3028, 1-D :3031-3113).
// AXI (linear axisymmetric model): alphaL, alphaT are blended with the
// particle's velocity (vpx, vpy, vpz) as pr_RWPTDisplacementsAxisymmetric
// does (:750-806, cosinesq = vz**2/|v| as written), and the horizontal
// transverse terms use alphaTH (pr_DisplacementRandomDischargeAxisymmetric
// {,2D,1D}, :3306-3604).
template <typename R, bool AXI>
__device__ __forceinline__ void random_displacement(const Lane<R> &F, int ndim, int d1, int d2, R x, R y,
                                                    R z, R vpx, R vpy, R vpz, uint64_t seed, uint64_t id,
                                                    uint64_t &ctr, R &bx, R &by, R &bz) {
  const R zero = R(0);
  R xy = x * y, xz = x * z, yz = y * z, xyz = xy * z;
  R aL = F(F_AL), aT = F(F_AT), dm = F(F_DM), tr = F(F_2R);
  R aTH = aT;
  if constexpr (AXI) {
    const R vnorm = sqrt_r(vpx * vpx + vpy * vpy + vpz * vpz);
    R cosinesq = zero;
    if (vnorm > zero) cosinesq = vpz * vpz / vnorm;
    aL = aL + cosinesq * (F(F_ALV) - aL);
    aT = F(F_ATV) + cosinesq * (aTH - F(F_ATV));
  }
  if (ndim == 3) {
    R cv[24];
    fields<R, F_VB, 24>(F, cv);
    R vx = tril(cv, x, y, z, xy, xz, yz, xyz);
    R vy = tril(cv + 8, x, y, z, xy, xz, yz, xyz);
    R vz = tril(cv + 16, x, y, z, xy, xz, yz, xyz);
    R nxy2 = fma(vx, vx, vy * vy);
    R n2 = fma(vz, vz, nxy2);
    R B11 = zero, B12 = zero, B13 = zero, B21 = zero, B22 = zero, B23 = zero, B31 = zero, B32 = zero;
    if (sizeof(R) == 8 ? above0(n2) : n2 > zero) {
      R inv = rsqrt(n2);
      R nrm = n2 * inv;
      R sL = sqrt_r(tr * fma(aL, nrm, dm));
      R sT = sqrt_r(tr * fma(aT, nrm, dm));
      R sTH = AXI ? sqrt_r(tr * fma(aTH, nrm, dm)) : sT;
      R sLi = sL * inv;
      B11 = vx * sLi;
      B21 = vy * sLi;
      B31 = vz * sLi;
      if (sizeof(R) == 8 ? above0(nxy2) : nxy2 > zero) {
        R invxy = rsqrt(nxy2);
        R nxy = nxy2 * invxy;
        R sTi = sT * inv;
        B32 = nxy * sTi;
        R sTixy = sTi * invxy;
        B12 = -(vx * vz) * sTixy;
        B22 = -(vy * vz) * sTixy;
        R sTxy = sTH * invxy;
        B13 = -vy * sTxy;
        B23 = vx * sTxy;
      }
    }
    R rx, ry, rz;
    Normals<R>::draw(3, seed, id, ctr, rx, ry, rz);
    bx = fma(B13, rz, fma(B12, ry, B11 * rx));
    by = fma(B23, rz, fma(B22, ry, B21 * rx));
    bz = fma(B32, ry, B31 * rx);
  } else if (ndim == 2) {
    R v1 = tril(F.p + F_VB + 8 * d1, x, y, z, xy, xz, yz, xyz);
    R v2 = tril(F.p + F_VB + 8 * d2, x, y, z, xy, xz, yz, xyz);
    R n2 = fma(v1, v1, v2 * v2);
    R B11 = zero, B12 = zero, B21 = zero, B22 = zero;
    if (n2 > zero) {
      R inv = rsqrt(n2);
      R nrm = n2 * inv;
      R sLi = sqrt_r(tr * fma(aL, nrm, dm)) * inv;
      R sTi = sqrt_r(tr * fma(aTH, nrm, dm)) * inv;
      B11 = v1 * sLi;
      B21 = v2 * sLi;
      B12 = -v2 * sTi;
      B22 = v1 * sTi;
    }
    R r1, r2, r3;
    Normals<R>::draw(2, seed, id, ctr, r1, r2, r3);
    R o1 = fma(B12, r2, B11 * r1), o2 = fma(B22, r2, B21 * r1);
    bx = zero; by = zero; bz = zero;
    if (d1 == 0) bx = o1; else if (d1 == 1) by = o1; else bz = o1;
    if (d2 == 0) bx = o2; else if (d2 == 1) by = o2; else bz = o2;
  } else {
    R v1 = tril(F.p + F_VB + 8 * d1, x, y, z, xy, xz, yz, xyz);
    R nrm = fabs(v1);
    R B11 = zero;
    if (nrm > zero) B11 = sqrt_r(tr * fma(aL, nrm, dm));
    R r1, r2, r3;
    Normals<R>::draw(1, seed, id, ctr, r1, r2, r3);
    bx = zero; by = zero; bz = zero;
    R o1 = B11 * r1;
    if (d1 == 0) bx = o1; else if (d1 == 1) by = o1; else bz = o1;
  }
}

// One axis of pr_DetectExitFaceAndUpdateTimeStepQuadratic (:1622-1710).
// Returns true when the routine must return at once (exitFace, dt set).
// The step length dt comes in the type T of its comparison: FP64 compares in
// double as the reference; MIXED passes the FP32 copy of dt (no FP64 op).
template <typename R, typename T>
__device__ __forceinline__ bool quad_axis(R npos, R pos, R d, R v, R divD, R dB, int faceLo, int faceHi,
                                          T dt, R &dtaxis, int &exitAxis, int &exitFace,
                                          double &dtout) {
  const R zero = R(0), one = R(1);
  R dI;
  if (npos > one) {
    dI = d * (one - pos);
    exitAxis = faceHi;
  } else {
    dI = -d * pos;
    exitAxis = faceLo;
  }
  if (dI == zero) {
    exitFace = exitAxis;
    dtout = 0.0;
    return true;
  }
  R A = v + divD, B = dB;
  R arg = B * B + R(4) * dI * A;
  if ((arg >= zero) && (A != zero)) {
    R zs = sqrt(arg);
    R z1, z2;
    if constexpr (sizeof(R) == 4) {
      // the same two roots without cancellation: q = -(B + sign(B) sqrt(arg))/2,
      // roots q/A and -dI/q
      R q = (B >= zero) ? -(B + zs) * R(0.5) : (zs - B) * R(0.5);
      z1 = q / A;
      z2 = (q != zero) ? -dI / q : zero;
    } else {
      z1 = (-B + zs) / (R(2) * A);
      z2 = (-B - zs) / (R(2) * A);
    }
    if (z1 > zero || z2 > zero) {
      R zm = (z1 > zero && z2 > zero) ? (z1 < z2 ? z1 : z2) : (z1 > zero ? z1 : z2);
      dtaxis = zm * zm;
      if (dtaxis == zero) {
        exitFace = exitAxis;
        dtout = 0.0;
        return true;
      }
    } else if (z1 == zero || z2 == zero) {
      exitFace = exitAxis;
      dtout = 0.0;
      return true;
    }
  } else if (A == zero) {
    if (B != zero) {
      R q = dI / B;
      dtaxis = q * q;
      if (dtaxis == zero) {
        exitFace = exitAxis;
        dtout = 0.0;
        return true;
      }
    }
  }
  if ((T)dtaxis > dt) dtaxis = zero;
  return false;
}

// quad_axis in FP64 with its tests against 0 and 1 and its step compare on
// the integer pipe (the same decisions, see above).
// `high`: the step leaves through the axis's upper face.
__device__ __forceinline__ bool quad_axis_f64(bool high, double pos, double d, double v, double divD, double dB,
                                              int faceLo, int faceHi, double dt, double &dtaxis, int &exitAxis,
                                              int &exitFace, double &dtout) {
  using R = double;
  const R zero = R(0), one = R(1);
  R dI;
  if (high) {
    dI = d * (one - pos);
    exitAxis = faceHi;
  } else {
    dI = -d * pos;
    exitAxis = faceLo;
  }
  if (is0(dI)) {
    exitFace = exitAxis;
    dtout = 0.0;
    return true;
  }
  R A = v + divD, B = dB;
  R arg = B * B + R(4) * dI * A;
  if (nonneg(arg) && !is0(A)) {
    const R zs = sqrt_r(arg);
    // roots z1 = n1 / (2A), z2 = n2 / (2A), n1 >= n2: the smaller positive
    // one is n2's for A > 0 and n1's for A < 0 when that is positive, else the
    // other; one division instead of two
    const R n1 = -B + zs, n2 = -B - zs;
    const bool pa = above0(A);
    const R na = pa ? n2 : n1, nb = pa ? n1 : n2;
    const bool fa = pa ? above0(na) : below0(na), fbk = pa ? above0(nb) : below0(nb);
    const R nm = fa ? na : nb;
    if ((fa || fbk) && fb::div_plain(nm, A)) {
      const R zm = fb::div_core(nm, A, 1);
      dtaxis = zm * zm;
      if (is0(dtaxis)) {
        exitFace = exitAxis;
        dtout = 0.0;
        return true;
      }
    } else {
      // no positive numerator, or a quotient outside the plain range: both
      // roots as written
      const R z1 = div_op(n1, R(2) * A), z2 = div_op(n2, R(2) * A);
      const bool p1 = above0(z1), p2 = above0(z2);
      if (p1 || p2) {
        R zm = (p1 && p2) ? (pos_lt(z1, z2) ? z1 : z2) : (p1 ? z1 : z2);
        dtaxis = zm * zm;
        if (is0(dtaxis)) {
          exitFace = exitAxis;
          dtout = 0.0;
          return true;
        }
      } else if (is0(z1) || is0(z2)) {
        exitFace = exitAxis;
        dtout = 0.0;
        return true;
      }
    }
  } else if (is0(A)) {
    if (!is0(B)) {
      R q = div_r(dI, B);
      dtaxis = q * q;
      if (is0(dtaxis)) {
        exitFace = exitAxis;
        dtout = 0.0;
        return true;
      }
    }
  }
  if (lt_any(dt, dtaxis)) dtaxis = zero;
  return false;
}

// ---- EXPONENTIAL advection (TrackSubCell.F90:1487-1538) and its exit time by
// Newton-Raphson (:1895-2554).  Both run in FP64 whatever the particle
// precision: the displacement v (e^{dv dt} - 1)/dv and the exit-time solve
// lose their digits to cancellation at small velocity gradients.
// Their quotients and displacements are calls: inlined at some thirty sites the
// integer divisions made the kernel's code longer than the instruction caches
// hold, and with the few warps that this kernel runs a third of the time went
// into fetching it (40,001 particles of a 61x37x7 field, two 5-day intervals,
// 57 -> 43 ms; 200,001, one interval: 99 -> 64).
__device__ __noinline__ double div_n(double a, double b) { return div_r(a, b); }
// em1 = e^{dvdx dt} - 1
__device__ __forceinline__ double adv_exponential(double v, double dvdx, double dt, double em1) {
  const double dvtol = 1.0e-10;
  return lt_any(dvtol, fabs(dvdx)) ? div_n(v * em1, dvdx) : v * dt;
}

__device__ __noinline__ double exp_displacement(double v, double dvdx, double dt) {
  return adv_exponential(v, dvdx, dt, exp(dvdx * dt) - 1.0);
}

__device__ __forceinline__ double nr_conv_g(double f0, double f1, double f2) { return fabs(div_n(f2 * f0, f1 * f1)); }
__device__ __forceinline__ double nr_conv_gder(double f0, double f1, double f2, double f3) {
  const double gna = div_n(f2 * f0, f1 * f1);
  const double gpp = div_n(-2.0 * (f0 * (f2 * f2)), f1 * f1 * f1) + div_n(f1 * f2 + f0 * f3, f1 * f1);
  return div_n(gna, fabs(gna)) * gpp;
}
// |x| < 1, 1/2 for x = |..| (NaN: false, as the compare)
__device__ __forceinline__ bool mag_below(double x, double c) { return fb::bits(x) < fb::bits(c); }
__constant__ double kP10[8] = {1e-8, 1e-7, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 1e-1};

// NewtonRaphsonTimeStepExponentialAdvection (:2451-2554, at most 50
// iterations) from pr_SetInitialGuess (:2162-2448; loops of 7, 50 and 8
// passes) as one loop around one evaluation of
// pr_NewtonRaphsonVariablesExponentialAdvection (:2082-2120): the displacement
// residual f0 at time `at` and its derivatives f1, f2, f3.  The lanes of a
// warp solve different faces and sit in different phases; with one evaluation
// site they run it together, and its instruction count is what the solve
// costs (the evaluation is FP64-pipe work).  An evaluation the reference
// repeats at a time it has just used is taken from the one before: one per
// pass of the 50-pass loop instead of three.  The convergence measure is only
// ever compared, so there the -3/2 power of the time in f2 is a quotient by
// its square root and itself, on the integer pipe; the measure's derivative,
// whose last bits the 50-pass loop carries into the guess, keeps pow (84 FP64
// instructions each) and is formed only when that loop goes on.
// Together with the solves dealt out over the warp (below) and the velocity
// gradients and exponentials held for a cell visit: 40,001 particles of a
// 61x37x7 field, two 5-day intervals, 145 -> 69 ms in FP64 and 143 -> 64 ms in
// MIXED at the same launch shape, every particle's state the same to the bit.
__device__ __noinline__ double nr_time_step(double dt, double v, double dvdx, double dI, double divD, double dB) {
  enum { SCAN, START, FIRST, ITER, SCAN2, NEWTON };
  const double gdtol = (double)1e-6f, nrtol = (double)1e-6f;
  const int maxter = 50, maxIter = 50;
  if (is0(dt)) return 0.0;
  double f0 = 0, f1 = 0, f2 = 0, ve = 0.0, fat = 0.0;
  double dtnew = 0.0, dtold = 0.0, gprimder = 0.0, gprimdernew = 0.0, gprimnew = 10.0;
  double gprim = (double)1e10f, gprimmin = (double)1e10f, mindtfrac = 0.0, nrerror = 1e6;
  int counter = 0, ccount = 0, bcount = 0, zcount = 0, rcount = 0, gcount = 1;
  double dtfraction = kP10[1], at = dt * dtfraction;
  int phase = SCAN;
  // The scan's first points by bounds (nrscan.cuh), as far as these put the
  // measure above one: the least of them, and the lower bound of the others.
  // Nearly every scan runs through all seven points (mean 6.7); bounds for one
  // are a tenth of its evaluation's instructions.  40,001 particles of a
  // 61x37x7 field, two 5-day intervals: 34.9 -> 31.2 ms (FP64), one in MIXED
  // 17.5 -> 14.6; 200,001, FP64: 54.4 -> 49.0.
  int jmin = 0;
  float lomin = INFINITY, himin = INFINITY, lorest = INFINITY;
  {
    const NrScan q = nr_scan_setup(v, dvdx, dI, divD, dB, lt_any(1.0e-10, fabs(dvdx)));
    for (; gcount < 7; ++gcount) {
      float lo, hi;
      if (!nr_scan_bounds(q, (float)dt * (float)kP10[gcount], lo, hi) || !(lo > 1.0f)) break;
      if (lo > 1.1e10f) continue;  // never the least: the search starts at 1e10
      if (hi > 0.9e10f) break;
      if (hi < himin) {
        lorest = fminf(lorest, lomin);
        jmin = gcount;
        lomin = lo;
        himin = hi;
      } else {
        lorest = fminf(lorest, lo);
      }
    }
    dtfraction = kP10[gcount];
    at = dt * dtfraction;
  }
  for (;;) {
    if (!is0(at) || phase == NEWTON) {
      const double e = exp(dvdx * at), s = sqrt_r(at);
      f0 = adv_exponential(v, dvdx, at, e - 1.0) + divD * at + dB * s - dI;
      const double q = div_n(dB, s);
      f1 = v * e + divD + 0.5 * q;
      if (phase != NEWTON) {
        ve = e;
        fat = at;
        f2 = dvdx * v * e - 0.25 * div_n(q, at);
      }
    }
    bool guess = false;  // the initial guess is dtnew: go on to Newton
    bool derive = false;   // the guess goes on: a pass of its 50-pass loop
    if (phase == NEWTON) {
      nrerror = div_n(-f0, f1);
      dtnew = dtnew + nrerror;
      if (below0(dtnew)) dtnew = -(double)0.9f * dtnew;
      ++counter;
    } else {
      const double g = nr_conv_g(f0, f1, f2);
      if (phase == SCAN || phase == SCAN2) {
        gprim = g;
        if (mag_below(gprim, gprimmin)) {
          gprimmin = gprim;
          mindtfrac = dtfraction;
        }
        if (above1(gprim) && (gcount < (phase == SCAN ? 7 : 9))) {
          ++gcount;
          dtfraction = (phase == SCAN) ? kP10[gcount] : (double)(0.1f * (float)gcount);
          at = dt * dtfraction;
          continue;
        }
        if (phase == SCAN2) {
          if (mag_below(gprimmin, 1.0)) dtnew = dt * mindtfrac;
          if ((below0(dtnew) || is0(dtnew)) && above0(fabs(v))) dtnew = fabs(div_n(dI, v));
          guess = true;
        } else {
          double dtoldfraction;
          const bool below = mag_below(gprim, 1.0);
          if (!below && jmin) {
            // no point is below one: the least of all seven, where the bounds
            // leave it open from the evaluations
            if (lorest > himin && pos_lt((double)himin, gprimmin)) {
              mindtfrac = kP10[jmin];
            } else if (!pos_lt(gprimmin, (double)fminf(lomin, lorest))) {
              jmin = 0;
              gcount = 1;
              gprim = gprimmin = (double)1e10f;
              mindtfrac = 0.0;
              at = dt * kP10[1];
              dtfraction = kP10[1];
              continue;
            }
          }
          if (below) {
            dtoldfraction = kP10[gcount - 1];
          } else {
            dtfraction = mindtfrac;
            dtoldfraction = div_n(0.5 * dtfraction, 10.0);
          }
          dtnew = dtfraction * dt;
          dtold = dtoldfraction * dt;
          phase = START;
          if (!below) {
            at = dtnew;
            continue;
          }
        }
      }
      if (phase == START) {
        gprim = g;
        if (mag_below(gprim, 0.5)) {
          guess = true;
        } else {
          derive = true;
        }
      } else if (phase == FIRST) {
        // at dtold; the values at dtnew are the starting ones
        derive = true;
      } else if (phase == ITER) {
        gprimnew = g;
        bool out = false;
        if (mag_below(gprimnew, 1.0) && above0(dtnew) && mag_below(div_n(dtnew, dt), 1.0)) {
          rcount = rcount + 1;
          guess = rcount > 1;
        } else {
          rcount = 0;
        }
        if (!guess && mag_below(gprim, 1.0) && lt_any(gprim, gprimnew)) {
          dtnew = dtold;
          guess = true;
        }
        if (!guess) {
          const bool still = mag_below(fabs(div_n(dtold - dtnew, dtold)), gdtol);
          if (still && mag_below(gprim, 1.0)) {
            ccount = ccount + 1;
            guess = ccount > 1;
          } else {
            ccount = 0;
          }
          if (!guess) {
            if (still && above1(gprim)) {
              bcount = bcount + 1;
              out = bcount > 1;
            } else {
              bcount = 0;
            }
          }
        }
        if (!guess) {
          if (out || counter >= maxter) {
            guess = mag_below(gprim, 1.0);
            if (!guess) phase = SCAN2;
          } else {
            derive = true;
          }
        }
      }
      if (derive) {
        // the derivative of the measure at the evaluated time (at zero time
        // the values stay those of the evaluation before)
        double p2 = 0.0, p3 = 0.0;
        if (!is0(fat)) {
          p2 = dvdx * v * ve - 0.25 * dB * pow(fat, -1.5);
          p3 = dvdx * dvdx * v * ve + 0.375 * dB * pow(fat, -2.5);
        }
        const double gd = nr_conv_gder(f0, f1, p2, p3);
        if (phase == START) {
          gprimdernew = gd;
          at = dtold;
          phase = FIRST;
          continue;
        }
        if (phase == FIRST) {
          gprimder = gd;
          if (is0(dtnew)) {
            gprimdernew = gd;
            gprim = g;
          }
        } else {
          // the next pass: dtold's values are those dtnew had before it
          gprimder = is0(dtold) ? gd : gprimdernew;
          gprimdernew = gd;
          gprim = g;
        }
        counter = counter + 1;
        const double dg = gprimdernew - gprimder;
        const double gamman = above0(dg) ? div_n(fabs((dtnew - dtold) * dg), dg * dg) : 0.0;
        dtold = dtnew;
        dtnew = dtnew - gamman * gprimdernew;
        bool out = false;
        if (fb::isnan_bits(dtnew)) {
          dtnew = 0.0;
          out = true;
        } else {
          const bool past = above1(div_n(dtnew, dt));
          if (mag_below(gprim, 1.0) && past) {
            dtnew = dtold;
            guess = true;
          } else if (past) {
            dtnew = (double)0.99f * dt;
          }
          if (!guess) {
            if (mag_below(gprim, 1.0) && below0(dtnew) && above0(dtold)) {
              dtnew = dtold;
              guess = true;
            } else if (below0(dtnew)) {
              dtnew = (double)1e-8f * dt;
              zcount = zcount + 1;
              if (zcount > 1) {
                dtnew = 0.0;
                out = true;
              }
            }
          }
        }
        if (!guess && out) {
          guess = mag_below(gprim, 1.0);
          if (!guess) phase = SCAN2;
        } else if (!guess) {
          at = dtnew;
          phase = ITER;
          continue;
        }
      }
      if (!guess) {  // the second scan begins
        gprim = gprimmin = (double)1e10f;
        mindtfrac = 0.0;
        gcount = 2;
        dtfraction = (double)(0.1f * (float)gcount);
        at = dt * dtfraction;
        continue;
      }
      if (is0(dtnew)) return 0.0;
      phase = NEWTON;
      counter = 0;
    }
    if (!(lt_any(nrtol, fabs(div_n(nrerror, dtnew))) && (counter < maxIter))) break;
    at = dtnew;
  }
  if (lt_any(dt, dtnew)) return dt;
  if ((counter == maxIter) && lt_any(nrtol, fabs(div_n(nrerror, dtnew)))) return 0.0;
  return dtnew;
}

// One axis of pr_DetectExitFaceAndUpdateTimeStepNewton (:1895-2079).
// Returns true when the routine must return at once (exitFace, dt set); `high`:
// the step leaves through the axis's upper face.
__device__ __forceinline__ bool newton_axis(bool high, double pos, double d, double v, double dvdx, double divD, double dB,
                            int faceLo, int faceHi, double dt, double &dtaxis, int &exitAxis, int &exitFace,
                            double &dtout) {
  double dI;
  if (high) {
    dI = d * (1.0 - pos);
    exitAxis = faceHi;
  } else {
    dI = -d * pos;
    exitAxis = faceLo;
  }
  if (is0(dI)) {
    exitFace = exitAxis;
    dtout = 0.0;
    return true;
  }
  dtaxis = nr_time_step(dt, v, dvdx, dI, divD, dB);
  if (lt_any(dt, dtaxis)) dtaxis = 0.0;
  return false;
}

template <typename R>
struct Visit {
  R x, y, z;     // current local position (TrackSubCell x,y,z)
  R ix, iy, iz;  // cell-entry location (initialLocation)
  double t, tinit, dtcell;
  R sqrt_dtcell, rdt_cell;
  int exitFace, posRestart;
  bool reachedMax;
  int waits;  // passes a leaving lane has waited (EXPONENTIAL)
  int64_t passes;
};

enum : int { PASS_CONTINUE = 0, PASS_MAXTIME = 1, PASS_EXIT = 2, PASS_UNDEFINED = 3, PASS_WAIT = 4 };

// component k (0, 1, 2) of three values, by selects (no local-memory array)
template <typename T>
__device__ __forceinline__ T pick3(int k, T a, T b, T c) {
  return (k == 0) ? a : ((k == 1) ? b : c);
}

// bit k set when component k of the proposed position is outside [0, 1]
template <typename R>
__device__ __forceinline__ unsigned axes_outside(R nx, R ny, R nz) {
  if constexpr (sizeof(R) == 8) {
    return (out01(nx) ? 1u : 0u) | (out01(ny) ? 2u : 0u) | (out01(nz) ? 4u : 0u);
  } else {
    const R zero = R(0), one = R(1);
    return ((nx > one || nx < zero) ? 1u : 0u) | ((ny > one || ny < zero) ? 2u : 0u) |
           ((nz > one || nz < zero) ? 4u : 0u);
  }
}

template <typename R>
__device__ __forceinline__ bool outside3(R a, R b, R c) {
  if constexpr (sizeof(R) == 8) {
    return out01(a) | out01(b) | out01(c);
  } else {
    const R zero = R(0), one = R(1);
    return (a > one) || (a < zero) || (b > one) || (b < zero) || (c > one) || (c < zero);
  }
}
#define MPRW_OUTSIDE(a, b, c) outside3(a, b, c)

// Exchange slots of a block in shared memory, kExitSlot doubles per thread,
// field k of a slot at p[k * stride + slot]; and the EXPONENTIAL kernel's
// per-lane values of a cell visit: the velocity gradients (V2 - V1)/D and
// e^{gradient dtcell} - 1 per axis.
constexpr int kLeaveEighths = 5, kMaxWaits = 16;
constexpr int kExitSlot = 7;
constexpr int kExpFields = 6;

// The first interface iteration's exit-face solves of the leaving lanes of
// `grp`, dealt out to every lane of `grp` (FP64, and the Newton solves of
// EXPONENTIAL advection, whose dv is the velocity gradient).  Each (leaving lane,
// leaving axis) pair is a task; tasks in axis-major order go to the group's
// lanes by rank (a second round only past one task per lane), every lane
// solves one with its owner's values (quad_axis is a pure function of them),
// and each owner gets back, per leaving axis, whether the solve returned at
// once (bit k of rbits), its exit face and its time.  Without this, a warp
// solves its lanes' first leaving axes together and then their second axes
// (corner crossings) in a second round of one or two lanes.  Every lane of
// grp calls it together, and no other lane of the warp.  The operands travel through the warp's exchange
// slots in shared memory: the owner of task t writes slot t, the lane of that
// rank reads it and writes the result back, so nobody searches for an owner.
template <typename R, bool EXP>
__device__ __forceinline__ void warp_exit_solves(unsigned grp, unsigned need, const Lane<R> &F, double *slots,
                                                 R nx, R ny, R nz, R x, R y, R z,
                                                 R vx, R vy, R vz, R ddx, R ddy,
                                                 R ddz, R bx, R by, R bz, double dvx,
                                                 double dvy, double dvz, double dt, unsigned &rbits,
                                                 double &tx, double &ty, double &tz, int &fx, int &fy,
                                                 int &fz) {
  const int lane = threadIdx.x & 31, stride = F.stride;
  const unsigned below = (1u << lane) - 1u;
  const unsigned m0 = __ballot_sync(grp, need & 1u), m1 = __ballot_sync(grp, need & 2u);
  const unsigned m2 = __ballot_sync(grp, need & 4u);
  const int c0 = __popc(m0), c1 = __popc(m1), total = c0 + c1 + __popc(m2);
  const int nw = __popc(grp), rank = __popc(grp & below);
  // this lane's own tasks, one per leaving axis
  const int t0 = __popc(m0 & below), t1 = c0 + __popc(m1 & below), t2 = c0 + c1 + __popc(m2 & below);
  double *slot = slots + (threadIdx.x & ~31);  // the warp's slots
  const R *rec = F.p - lane * kRecStride<R>;   // the warp's records
  rbits = 0u;
  tx = ty = tz = 0.0;
  fx = fy = fz = 0;
  for (int base = 0; base < total; base += nw) {
    auto put = [&](int a, int t, R npos, R pos, R v, R dd, R b, double dv) {
      const int k = t - base;
      if (!((need >> a) & 1u) || k < 0 || k >= nw) return;
      slot[k] = (double)pos;
      slot[stride + k] = (double)v;
      slot[2 * stride + k] = (double)dd;
      slot[3 * stride + k] = (double)b;
      slot[4 * stride + k] = dt;
      if (EXP) slot[6 * stride + k] = dv;
      reinterpret_cast<int *>(slot + 5 * stride + k)[0] = lane | (a << 5) | (above1(npos) ? 128 : 0);
    };
    put(0, t0, nx, x, vx, ddx, bx, dvx);
    put(1, t1, ny, y, vy, ddy, by, dvy);
    put(2, t2, nz, z, vz, ddz, bz, dvz);
    __syncwarp(grp);
    if (base + rank < total) {
      const int meta = reinterpret_cast<const int *>(slot + 5 * stride + rank)[0];
      const int a = (meta >> 5) & 3;
      int efa = 0, ef_unused = 0;
      double dta = 0.0, dt_unused = 0.0;
      const double d = (double)rec[(meta & 31) * kRecStride<R> + F_D + a];
      bool r;
      if constexpr (EXP)
        r = newton_axis((meta & 128) != 0, slot[rank], d, slot[stride + rank], slot[6 * stride + rank],
                        slot[2 * stride + rank], slot[3 * stride + rank], 2 * a + 1, 2 * a + 2,
                        slot[4 * stride + rank], dta, efa, ef_unused, dt_unused);
      else
        r = quad_axis_f64((meta & 128) != 0, slot[rank], d, slot[stride + rank], slot[2 * stride + rank],
                          slot[3 * stride + rank], 2 * a + 1, 2 * a + 2, slot[4 * stride + rank], dta, efa,
                          ef_unused, dt_unused);
      slot[rank] = dta;
      reinterpret_cast<int *>(slot + 5 * stride + rank)[0] = (r ? 8 : 0) | efa;
    }
    __syncwarp(grp);
    auto get = [&](int a, int t, double &ta, int &fa) {
      const int k = t - base;
      if (!((need >> a) & 1u) || k < 0 || k >= nw) return;
      ta = slot[k];
      const int pk = reinterpret_cast<const int *>(slot + 5 * stride + k)[0];
      fa = pk & 7;
      if (pk & 8) rbits |= 1u << a;
    };
    get(0, t0, tx, fx);
    get(1, t1, ty, fy);
    get(2, t2, tz, fz);
    __syncwarp(grp);
  }
}

// One pass of the `do while (continueTimeLoop)` body, TrackSubCell.F90:956-1368.
// On PASS_MAXTIME / PASS_EXIT the final location is (ox,oy,oz,V.t); on
// PASS_UNDEFINED the caller uses the last recorded point; PASS_WAIT: the pass
// has not been made.  `grp` (FP64, EXPONENTIAL): the lanes of the warp that
// call this together.
template <typename R, bool EXP, bool AXI>
__device__ int rw_pass(unsigned grp, Visit<R> &V, const Lane<R> &F, double *slots, uint32_t massb, double maxTime, int ndim, int d1, int d2,
                       uint64_t seed, uint64_t id, uint64_t &ctr, R &ox, R &oy, R &oz) {
  const R zero = R(0), one = R(1), half = R(0.5);
  const double t_in = V.t;        // (EXPONENTIAL)
  const uint64_t ctr_in = ctr;
  const double dtRed = (double)0.1f;  // dtReductionFactor, a single-precision literal (:850)
  double dt = V.dtcell;
  R rdt = V.rdt_cell, sdt = V.sqrt_dtcell;  // FP32 copies: no conversion on the common pass
  V.t = V.t + dt;
  if (sizeof(R) == 8 ? past_end(maxTime, V.t) : maxTime < V.t) {
    V.t = V.t - dt;
    dt = fmax(maxTime - V.t, 0.0);
    V.t = maxTime;
    V.reachedMax = true;
    rdt = (R)dt;
    sdt = sqrt_r(rdt);
  }
  R x = V.x, y = V.y, z = V.z;
  R head[12];  // V1, DV, D, 1/D
  fields<R, 0, 12>(F, head);
  R dX = head[F_D + 0], dY = head[F_D + 1], dZ = head[F_D + 2];
  R iX = head[F_INVD + 0], iY = head[F_INVD + 1], iZ = head[F_INVD + 2];
  // pr_RWPTDisplacementsLinear (:673-706)
  R vx = fma(x, head[F_DV + 0], head[F_V1 + 0]);
  R vy = fma(y, head[F_DV + 1], head[F_V1 + 1]);
  R vz = fma(z, head[F_DV + 2], head[F_V1 + 2]);
  R xy = x * y, xz = x * z, yz = y * z;
  R cd[21];
  fields<R, F_DIV, 21>(F, cd);
  R ddx = divc(cd, x, y, z, xy, xz, yz);
  R ddy = divc(cd + 7, x, y, z, xy, xz, yz);
  R ddz = divc(cd + 14, x, y, z, xy, xz, yz);
  R bx, by, bz;
  random_displacement<R, AXI>(F, ndim, d1, d2, x, y, z, vx, vy, vz, seed, id, ctr, bx, by, bz);
  // advection displacement: EULERIAN v dt, EXPONENTIAL (FP64) v (e^{dv dt}-1)/dv
  // with dv = (V2 - V1)/D of the cell (pr_AdvectionDisplacement*, :1487-1573)
  // (dv, and the exponentials of the whole cell step, held for the visit)
  double dvx = 0.0, dvy = 0.0, dvz = 0.0;
  const double *xf = slots + kExitSlot * F.stride + threadIdx.x;
  if constexpr (EXP) {
    dvx = xf[0];
    dvy = xf[F.stride];
    dvz = xf[2 * F.stride];
  }
  R ax, ay, az;
  auto advect = [&]() {
    if constexpr (EXP) {
      ax = (R)exp_displacement((double)vx, dvx, dt);
      ay = (R)exp_displacement((double)vy, dvy, dt);
      az = (R)exp_displacement((double)vz, dvz, dt);
    } else {
      ax = vx * rdt;
      ay = vy * rdt;
      az = vz * rdt;
    }
  };
  if (EXP && eq_any(dt, V.dtcell)) {
    ax = (R)adv_exponential((double)vx, dvx, dt, xf[3 * F.stride]);
    ay = (R)adv_exponential((double)vy, dvy, dt, xf[4 * F.stride]);
    az = (R)adv_exponential((double)vz, dvz, dt, xf[5 * F.stride]);
  } else {
    advect();
  }
  R dxrw = ax + ddx * rdt + bx * sdt;
  R dyrw = ay + ddy * rdt + by * sdt;
  R dzrw = az + ddz * rdt + bz * sdt;
  // jump limiter (:989-1013)
  if constexpr (sizeof(R) == 4 && !EXP) {
    // MIXED: the cut step stays in FP32 (rdt = 0.1 rdt) and the simulation
    // time is corrected once after the loop.  The loop runs with a few
    // lanes, and every FP64 operation in it would cost a whole warp
    // instruction on the narrow FP64 pipe.
    const double dt0 = dt;
    bool cut = false;
    while ((fabs(dxrw * iX) > half) || (fabs(dyrw * iY) > half) || (fabs(dzrw * iZ) > half)) {
      rdt = R(0.1f) * rdt;
      sdt = sqrt_r(rdt);
      advect();
      dxrw = ax + ddx * rdt + bx * sdt;
      dyrw = ay + ddy * rdt + by * sdt;
      dzrw = az + ddz * rdt + bz * sdt;
      cut = true;
    }
    if (cut) {
      dt = (double)rdt;
      V.t = (V.t - dt0) + dt;
      V.reachedMax = false;
    }
  } else
  while (sizeof(R) == 8 ? over_half(dxrw, iX) | over_half(dyrw, iY) | over_half(dzrw, iZ)
                        : (fabs(dxrw * iX) > half) || (fabs(dyrw * iY) > half) || (fabs(dzrw * iZ) > half)) {
    V.t = V.t - dt;
    dt = dtRed * dt;
    rdt = (R)dt;
    sdt = sqrt_r(rdt);
    advect();
    dxrw = ax + ddx * rdt + bx * sdt;
    dyrw = ay + ddy * rdt + by * sdt;
    dzrw = az + ddz * rdt + bz * sdt;
    V.t = V.t + dt;
    V.reachedMax = false;
  }
  R nx = x + dxrw * iX, ny = y + dyrw * iY, nz = z + dzrw * iZ;
  // EXPONENTIAL: leaving lanes wait until they are five of eight.  A Newton
  // solve takes some ten passes' time and a warp runs it with the lanes that
  // have one, so a lane that would leave stays where it was before the pass
  // and repeats it -- the same draws, the same step; the other lanes' passes
  // pay for it -- until enough lanes of the warp, or all, would leave, or
  // one has waited for 16 passes (particles that seldom leave).  40,001
  // particles of a 61x37x7 field, two 5-day intervals: 43.3 -> 34.6 ms (three of
  // eight 38.6, four 36.5, six 35.9); 200,001, one interval: 64 -> 54.  In the
  // EULERIAN kernels, whose solves are short, the waiting costs what it gives
  // (FP64 50.6 -> 51.4 ms at two of eight, MIXED 10.7 -> 11.7).
  if constexpr (EXP) {
    __syncwarp(grp);
    const bool leaves = MPRW_OUTSIDE(nx, ny, nz);
    const unsigned lm = __ballot_sync(grp, leaves);
    if (lm != grp && 8 * __popc(lm) < kLeaveEighths * __popc(grp) &&
        !__any_sync(grp, leaves && V.waits >= kMaxWaits)) {
      if (leaves) {
        ++V.waits;
        V.t = t_in;
        V.reachedMax = false;
        ctr = ctr_in;
        return PASS_WAIT;
      }
      grp &= ~lm;
    }
    V.waits = 0;
  }
  // FP64 and EXPONENTIAL: the first interface iteration's exit-face solves of
  // the leaving lanes, spread over every lane of the pass
  unsigned pre_r = 0u;
  double pre_tx = 0.0, pre_ty = 0.0, pre_tz = 0.0;
  int pre_fx = 0, pre_fy = 0, pre_fz = 0;
  if constexpr (sizeof(R) == 8 || EXP) {
    __syncwarp(grp);
    warp_exit_solves<R, EXP>(grp, axes_outside(nx, ny, nz), F, slots, nx, ny, nz, x, y, z, vx, vy, vz, ddx, ddy,
                             ddz, bx, by, bz, dvx, dvy, dvz, dt, pre_r, pre_tx, pre_ty, pre_tz, pre_fx, pre_fy, pre_fz);
  }
  // particleLeavingCell (:1025-1316)
  int intLoop = 0;
  while (MPRW_OUTSIDE(nx, ny, nz)) {
    ++intLoop;
    if constexpr (EXP) {
      // ExitFaceAndUpdateTimeStep (Newton, :1895-2079), FP64
      double dtx = 0.0, dty = 0.0, dtz = 0.0;
      int efx = 0, efy = 0, efz = 0;
      bool ret = false;
      V.t = V.t - dt;
      // the axes the step leaves through, x then y then z, solved in one
      // shared block: the first axis of every leaving lane together, then
      // the second (a warp's leaving lanes mostly leave through different
      // axes; three per-axis branches would each run with a few lanes)
      unsigned need = axes_outside(nx, ny, nz);
      if (intLoop == 1) {
        // the warp-wide solves (the same inputs: nothing has moved yet)
        while (!ret && need) {
          const int k = __ffs(need) - 1;
          need &= need - 1;
          if ((pre_r >> k) & 1u) {
            V.exitFace = pick3(k, pre_fx, pre_fy, pre_fz);
            dt = 0.0;
            ret = true;
          } else if (k == 0) { dtx = pre_tx; efx = pre_fx; }
          else if (k == 1) { dty = pre_ty; efy = pre_fy; }
          else { dtz = pre_tz; efz = pre_fz; }
        }
      }
      while (!ret && need) {
        const int k = __ffs(need) - 1;
        need &= need - 1;
        double dta = 0.0;
        int efa = 0;
        ret = newton_axis(above1(pick3(k, nx, ny, nz)), (double)pick3(k, x, y, z), (double)pick3(k, dX, dY, dZ),
                          (double)pick3(k, vx, vy, vz), pick3(k, dvx, dvy, dvz), (double)pick3(k, ddx, ddy, ddz),
                          (double)pick3(k, bx, by, bz), 2 * k + 1, 2 * k + 2, dt, dta, efa, V.exitFace, dt);
        if (k == 0) { dtx = dta; efx = efa; }
        else if (k == 1) { dty = dta; efy = efa; }
        else { dtz = dta; efz = efa; }
      }
      if (!ret) {
        if (dtx == 0.0 && dty == 0.0 && dtz == 0.0) {
          V.t = V.t + dt;
        } else {
          int im = -1;
          double best = 0.0;
          if (dtx > 0.0) { im = 0; best = dtx; }
          if (dty > 0.0 && (im < 0 || dty < best)) { im = 1; best = dty; }
          if (dtz > 0.0 && (im < 0 || dtz < best)) { im = 2; best = dtz; }
          dt = best;
          V.exitFace = (im == 0) ? efx : (im == 1 ? efy : efz);
          V.t = V.t + dt;
        }
      }
    } else {
      R dtx = zero, dty = zero, dtz = zero;
      // ExitFaceAndUpdateTimeStep (quadratic, :1576-1892)
      int efx = 0, efy = 0, efz = 0;
      bool ret = false;
      // MIXED takes the time back only when the step changes (below)
      const double dt_in = dt;
      if constexpr (sizeof(R) == 8) V.t = V.t - dt;
      if constexpr (sizeof(R) == 8) {
        // FP64: the first iteration takes the warp-wide solves (the same
        // inputs: nothing has moved yet); later ones solve the leaving axes
        // in one shared block (as for EXPONENTIAL).  The FP32 solve is cheap
        // enough that the extra registers of either cost more than the
        // divergence.
        unsigned need = axes_outside(nx, ny, nz);
        if (intLoop == 1) {
          while (!ret && need) {
            const int k = __ffs(need) - 1;
            need &= need - 1;
            if ((pre_r >> k) & 1u) {
              V.exitFace = pick3(k, pre_fx, pre_fy, pre_fz);
              dt = 0.0;
              ret = true;
            } else if (k == 0) { dtx = pre_tx; efx = pre_fx; }
            else if (k == 1) { dty = pre_ty; efy = pre_fy; }
            else { dtz = pre_tz; efz = pre_fz; }
          }
        }
        while (!ret && need) {
          const int k = __ffs(need) - 1;
          need &= need - 1;
          R dta = zero;
          int efa = 0;
          ret = quad_axis_f64(above1(pick3(k, nx, ny, nz)), pick3(k, x, y, z), pick3(k, dX, dY, dZ), pick3(k, vx, vy, vz),
                          pick3(k, ddx, ddy, ddz), pick3(k, bx, by, bz), 2 * k + 1, 2 * k + 2, dt, dta, efa,
                          V.exitFace, dt);
          if (k == 0) { dtx = dta; efx = efa; }
          else if (k == 1) { dty = dta; efy = efa; }
          else { dtz = dta; efz = efa; }
        }
      } else {
        if (!ret && ((nx > one) || (nx < zero)))
          ret = quad_axis(nx, x, dX, vx, ddx, bx, 1, 2, rdt, dtx, efx, V.exitFace, dt);
        if (!ret && ((ny > one) || (ny < zero)))
          ret = quad_axis(ny, y, dY, vy, ddy, by, 3, 4, rdt, dty, efy, V.exitFace, dt);
        if (!ret && ((nz > one) || (nz < zero)))
          ret = quad_axis(nz, z, dZ, vz, ddz, bz, 5, 6, rdt, dtz, efz, V.exitFace, dt);
      }
      if (!ret) {
        if (sizeof(R) == 8 ? is0(dtx) && is0(dty) && is0(dtz) : dtx == zero && dty == zero && dtz == zero) {
          if constexpr (sizeof(R) == 8) V.t = V.t + dt;
        } else {
          int im = -1;
          R best = zero;
          if constexpr (sizeof(R) == 8) {
            // (best > 0 once im >= 0)
            if (above0(dtx)) { im = 0; best = dtx; }
            if (above0(dty) && (im < 0 || pos_lt(dty, best))) { im = 1; best = dty; }
            if (above0(dtz) && (im < 0 || pos_lt(dtz, best))) { im = 2; best = dtz; }
          } else {
            if (dtx > zero) { im = 0; best = dtx; }
            if (dty > zero && (im < 0 || dty < best)) { im = 1; best = dty; }
            if (dtz > zero && (im < 0 || dtz < best)) { im = 2; best = dtz; }
          }
          dt = (double)best;
          V.exitFace = (im == 0) ? efx : (im == 1 ? efy : efz);
          if constexpr (sizeof(R) == 8) {
            V.t = V.t + dt;
          } else {
            V.t = (V.t - dt_in) + dt;
            rdt = best;
          }
        }
      } else if constexpr (sizeof(R) == 4) {
        V.t = V.t - dt_in;
        rdt = zero;
      }
    }
    if (intLoop > 5) {
      nx = V.ix; ny = V.iy; nz = V.iz;
      V.t = V.tinit;
      dt = V.dtcell;
      if (++V.posRestart > 10) {
        V.x = x; V.y = y; V.z = z;
        return PASS_UNDEFINED;
      }
      break;
    }
    if constexpr (sizeof(R) == 8 || EXP) rdt = (R)dt;  // MIXED EULERIAN: rdt set above
    sdt = sqrt_r(rdt);
    if constexpr (sizeof(R) == 4) advect();
    V.reachedMax = false;
    int ef = V.exitFace;
    if (ef >= 1 && ef <= 6 && sizeof(R) == 8) {
      // FP64: the exit axis pinned to its face, the step of the truncated
      // time on the two others (p and q, one shared block)
      const int fa = (ef - 1) >> 1;
      const bool p0 = fa != 0, q2 = fa != 2;  // p: x, or y when x is pinned; q: z, or y
      const R pin = (ef & 1) ? zero : one;
      const double dvp = p0 ? dvx : dvy, dvq = q2 ? dvz : dvy;
      const R vp = p0 ? vx : vy, vq = q2 ? vz : vy;
      R ap, aq;
      if constexpr (EXP) {
        ap = (R)exp_displacement((double)vp, dvp, dt);
        aq = (R)exp_displacement((double)vq, dvq, dt);
      } else {
        ap = vp * rdt;
        aq = vq * rdt;
      }
      const R dp = ap + (p0 ? ddx : ddy) * rdt + (p0 ? bx : by) * sdt;
      const R dq = aq + (q2 ? ddz : ddy) * rdt + (q2 ? bz : by) * sdt;
      const R np = (p0 ? x : y) + dp * (p0 ? iX : iY), nq = (q2 ? z : y) + dq * (q2 ? iZ : iY);
      if (fa == 0) { nx = pin; dyrw = dp; ny = np; dzrw = dq; nz = nq; }
      else if (fa == 1) { dxrw = dp; nx = np; ny = pin; dzrw = dq; nz = nq; }
      else { dxrw = dp; nx = np; dyrw = dq; ny = nq; nz = pin; }
    } else if (ef == 1 || ef == 2) {
      nx = (ef == 1) ? zero : one;
      dyrw = ay + ddy * rdt + by * sdt;
      ny = y + dyrw * iY;
      dzrw = az + ddz * rdt + bz * sdt;
      nz = z + dzrw * iZ;
    } else if (ef == 3 || ef == 4) {
      dxrw = ax + ddx * rdt + bx * sdt;
      nx = x + dxrw * iX;
      ny = (ef == 3) ? zero : one;
      dzrw = az + ddz * rdt + bz * sdt;
      nz = z + dzrw * iZ;
    } else if (ef == 5 || ef == 6) {
      dxrw = ax + ddx * rdt + bx * sdt;
      nx = x + dxrw * iX;
      dyrw = ay + ddy * rdt + by * sdt;
      ny = y + dyrw * iY;
      nz = (ef == 5) ? zero : one;
    } else {
      nx = V.ix; ny = V.iy; nz = V.iz;
      V.t = V.tinit;
      dt = V.dtcell;
      if (++V.posRestart > 10) {
        V.x = x; V.y = y; V.z = z;
        return PASS_UNDEFINED;
      }
      break;
    }
    if (MPRW_OUTSIDE(nx, ny, nz)) continue;
    // elasticRebound (:1157-1312)
    int rebound = 0;
    while (V.exitFace > 0) {
      if (!((massb >> (V.exitFace - 1)) & 1u)) break;
      if (++rebound > 10) {
        V.x = x; V.y = y; V.z = z;
        return PASS_UNDEFINED;
      }
      R xi = nx, yi = ny, zi = nz;
      if (sizeof(R) == 8 ? is0(dt) : dt == 0.0) {
        nx = V.ix; ny = V.iy; nz = V.iz;
        V.t = V.t - dt;
        dt = V.dtcell;
        V.exitFace = 0;
        ++V.posRestart;
        break;
      }
      V.t = V.t + dt;
      if (sizeof(R) == 8 ? past_end(maxTime, V.t) : maxTime < V.t) {
        V.t = V.t - dt;
        dt = fmax(maxTime - V.t, 0.0);
        V.t = maxTime;
        V.reachedMax = true;
        rdt = (R)dt;
        sdt = sqrt_r(rdt);
        advect();
        dxrw = ax + ddx * rdt + bx * sdt;
        dyrw = ay + ddy * rdt + by * sdt;
        dzrw = az + ddz * rdt + bz * sdt;
      }
      ef = V.exitFace;
      if (ef == 1 || ef == 2) {
        nx = nx - dxrw * iX; ny = ny + dyrw * iY; nz = nz + dzrw * iZ;
      } else if (ef == 3 || ef == 4) {
        nx = nx + dxrw * iX; ny = ny - dyrw * iY; nz = nz + dzrw * iZ;
      } else {
        nx = nx + dxrw * iX; ny = ny + dyrw * iY; nz = nz - dzrw * iZ;
      }
      if (MPRW_OUTSIDE(nx, ny, nz)) {
        x = xi; y = yi; z = zi;
        if (ef == 1 || ef == 2) { vx = -vx; ddx = -ddx; bx = -bx; }
        else if (ef == 3 || ef == 4) { vy = -vy; ddy = -ddy; by = -by; }
        else { vz = -vz; ddz = -ddz; bz = -bz; }
        V.exitFace = 0;
      } else {
        dt = V.dtcell;
        V.exitFace = 0;
        if constexpr (sizeof(R) == 8) {
          if (is0(nx)) V.exitFace = 1;
          if (is1(nx)) V.exitFace = 2;
          if (is0(ny)) V.exitFace = 3;
          if (is1(ny)) V.exitFace = 4;
          if (is0(nz)) V.exitFace = 5;
          if (is1(nz)) V.exitFace = 6;
        } else {
          if (nx == zero) V.exitFace = 1;
          if (nx == one) V.exitFace = 2;
          if (ny == zero) V.exitFace = 3;
          if (ny == one) V.exitFace = 4;
          if (nz == zero) V.exitFace = 5;
          if (nz == one) V.exitFace = 6;
        }
      }
    }
  }
  if (V.reachedMax) {
    ox = nx; oy = ny; oz = nz;
    return PASS_MAXTIME;
  }
  if (V.exitFace > 0) {
    ox = nx; oy = ny; oz = nz;
    return PASS_EXIT;
  }
  V.x = nx; V.y = ny; V.z = nz;
  return PASS_CONTINUE;
}

// Persistent kernel: every lane owns one particle at a time.  Each iteration of
// the main loop (a) refills lanes without a particle from the atomic queue
// (one atomic per warp), (b) runs the cell-entry phase for lanes that changed
// cell, (c) runs one time-loop pass for every tracking lane.  All phases are
// structured and the loop head re-converges the warp, so the common pass body
// runs with every tracking lane active; the loop ends when no lane of the warp
// has work.
template <typename R, bool EXP, bool AXI>
__global__ void __launch_bounds__(step_threads(sizeof(R) == 8, EXP), (sizeof(R) == 4 && !EXP) ? 3 : 1) rwpt_advance_kernel(AdvanceArgs<R> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  R *sm = reinterpret_cast<R *>(smraw) + threadIdx.x * kRecStride<R>;
  const int stride = blockDim.x;
  Lane<R> F{sm, stride};
  // the exchange slots (FP64 or EXPONENTIAL) follow the records
  double *slots = reinterpret_cast<double *>(reinterpret_cast<R *>(smraw) + kRecStride<R> * stride);
  const R zero = R(0), one = R(1);
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;

  int64_t my_passes = 0;
  int64_t p = -1;        // particle being tracked (index into the state arrays)
  bool open = lane < a.lanes;  // the queue may still have particles for this lane
  int32_t c = 0;         // current cell (0-based)
  bool need_cell = false;
  uint64_t id = 0, ctr = 0;
  // last point of the pathline (cell, local coords, time)
  int32_t lc = 0;
  R lx = zero, ly = zero, lz = zero;
  double lt = 0.0;
  // location at cell entry
  R ex = zero, ey = zero, ez = zero;
  double et = 0.0;
  Visit<R> V;
  V.x = V.y = V.z = V.ix = V.iy = V.iz = zero;
  V.t = V.tinit = V.dtcell = 0.0;
  V.sqrt_dtcell = zero;
  V.rdt_cell = zero;
  V.exitFace = V.posRestart = 0;
  V.reachedMax = false;
  V.passes = 0;
  V.waits = 0;
  uint32_t massb = 0;
  // cell exits of the current particle in this launch (bits 0-19) and how
  // many of the last ones took no time (bits 20-30): one register for both caps
  static_assert(kMaxVisitsPerAdvance < (1 << 20) - 1 && kMaxZeroTimeExits < (1 << 11) - 1, "exit counter bits");
  uint32_t exits = 0;

  unsigned iter = 0;
  for (;;) {
    __syncwarp(FULL);
    // cancel: the host set the flag (timeout or mprw_cancel).  Each lane keeps
    // its particle where it is -- the start of the cell it is entering, or the
    // last completed pass of its visit -- as ACTIVE, and the queue is not
    // drained further, so every particle holds a valid location.
    if (a.abort && (++iter % kAbortPoll) == 0) {
      int ab = (lane == 0) ? *a.abort : 0;
      ab = __shfl_sync(FULL, ab, 0);
      if (ab) {
        if (p >= 0) {
          a.cell[p] = c;
          if (need_cell) {
            a.x[p] = ex; a.y[p] = ey; a.z[p] = ez; a.t[p] = et;
          } else {
            a.x[p] = V.x; a.y[p] = V.y; a.z[p] = V.z; a.t[p] = V.t;
          }
          a.status[p] = ST_ACTIVE;
          a.ctr[p] = ctr;
        }
        break;
      }
    }
    // (a) refill
    const bool want = (p < 0) && open;
    const unsigned m = __ballot_sync(FULL, want);
    if (m) {
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader)
        base = atomicAdd(reinterpret_cast<unsigned long long *>(a.queue), (unsigned long long)__popc(m));
      base = __shfl_sync(FULL, base, leader);
      if (want) {
        const int64_t q = (int64_t)base + __popc(m & ((1u << lane) - 1u));
        if (q >= a.n) {
          open = false;
        } else {
          p = a.perm ? (int64_t)a.perm[q] : q;
          int32_t status = a.status[p];
          c = a.cell[p];
          ex = a.x[p]; ey = a.y[p]; ez = a.z[p];
          et = a.t[p];
          // release checks, MPathRW.F90:1256-1302
          if (status == ST_PENDING) {
            if (et < a.t_begin) status = ST_UNRELEASED;
            else if (et <= a.t_end) {
              status = ST_ACTIVE;
              if (a.iboundts[c] == 0) status = ST_INACTIVE;
            }
          }
          if (status == ST_INACTIVE && (a.cellflags[c] & 2u)) status = ST_ACTIVE;  // partially dry
          if (status != ST_ACTIVE) {
            a.status[p] = status;
            p = -1;
          } else {
            id = a.id ? a.id[p] : (uint64_t)p;
            ctr = a.ctr[p];
            lc = c; lx = ex; ly = ey; lz = ez; lt = et;
            need_cell = true;
            exits = 0;
          }
        }
      }
    }
    if (!__any_sync(FULL, (p >= 0) || open)) break;

    // (b) cell entry (TrackCell checks + sub-cell set-up)
    if (p >= 0 && need_cell) {
      need_cell = false;
      int32_t fin = 0;  // 0 track, else final status
      bool use_last = false;
      if (sizeof(R) == 8 ? outside3(ex, ey, ez)
                         : ex < zero || ex > one || ey < zero || ey > one || ez < zero || ez > one) {
        fin = ST_UNDEFINED;  // InvalidLocation (TrackCell.f90:410-413)
        use_last = true;
      } else {
        // the record is on its way while the entry checks are read
        const CellRec<R> *rec = a.recs + c;
        stage_record(a.recs, c, sm);
        const int32_t es = rec->entry_status;
        const double dtc = rec->dtcell, sdtc = rec->sqrt_dtcell;
        massb = rec->massb;
        stage_wait();
        if (es != 0) {
          fin = es;
          use_last = (es == ST_UNDEFINED);
        } else {
          if constexpr (EXP) {
            double *xf = slots + kExitSlot * stride + threadIdx.x;
            for (int d = 0; d < 3; ++d) {
              const double g = div_r((double)F(F_DV + d), (double)F(F_D + d));
              xf[d * stride] = g;
              xf[(3 + d) * stride] = exp(g * dtc) - 1.0;
            }
          }
          V.x = ex; V.y = ey; V.z = ez;
          V.ix = ex; V.iy = ey; V.iz = ez;
          V.t = et; V.tinit = et;
          V.dtcell = dtc;
          V.sqrt_dtcell = (R)sdtc;
          V.rdt_cell = (R)dtc;
          V.exitFace = 0;
          V.posRestart = 0;
          V.reachedMax = false;
          V.passes = 0;
        }
      }
      if (fin != 0) {
        if (use_last) {
          a.cell[p] = lc; a.x[p] = lx; a.y[p] = ly; a.z[p] = lz; a.t[p] = lt;
        } else {
          a.cell[p] = c; a.x[p] = ex; a.y[p] = ey; a.z[p] = ez; a.t[p] = et;
        }
        a.status[p] = fin;
        a.ctr[p] = ctr;
        p = -1;
      }
    }

    // (c) one time-loop pass (with the per-visit safety cap).  Its lanes are
    // settled by a vote of the whole warp: cell entry has just divided it, and
    // the exit solves' exchange slots are the warp's, so two parts of it in
    // the pass at once would overwrite each other's operands.  (FP32 EULERIAN
    // exchanges nothing.)
    const bool tracks = p >= 0 && !need_cell;
    unsigned grp = 0u;
    if constexpr (sizeof(R) == 8 || EXP) grp = __ballot_sync(FULL, tracks && V.passes < kMaxStepsPerVisit);
    if (tracks) {
      R ox = zero, oy = zero, oz = zero;
      int r;
      if (++V.passes > kMaxStepsPerVisit) {
        r = PASS_UNDEFINED;
      } else {
        r = rw_pass<R, EXP, AXI>(grp, V, F, slots, massb, a.t_end, a.ndim, a.d1, a.d2, a.seed, id, ctr, ox, oy, oz);
        if (EXP && r == PASS_WAIT) --V.passes;
        else ++my_passes;
      }
      if (r == PASS_MAXTIME) {
        a.cell[p] = c; a.x[p] = ox; a.y[p] = oy; a.z[p] = oz; a.t[p] = V.t;
        a.status[p] = ST_ACTIVE;
        a.ctr[p] = ctr;
        p = -1;
      } else if (r == PASS_UNDEFINED) {
        a.cell[p] = lc; a.x[p] = lx; a.y[p] = ly; a.z[p] = lz; a.t[p] = lt;
        a.status[p] = ST_UNDEFINED;
        a.ctr[p] = ctr;
        p = -1;
      } else if (r == PASS_EXIT &&
                 ((exits = ((exits & 0xFFFFFu) + 1u) | ((sizeof(R) == 8 ? eq_any(V.t, V.tinit) : V.t == V.tinit) ? ((exits >> 20) + 1u) << 20 : 0u)) >> 20 >
                      (uint32_t)kMaxZeroTimeExits ||
                  (exits & 0xFFFFFu) > (uint32_t)kMaxVisitsPerAdvance)) {
        a.cell[p] = lc; a.x[p] = lx; a.y[p] = ly; a.z[p] = lz; a.t[p] = lt;
        a.status[p] = ST_UNDEFINED;
        a.ctr[p] = ctr;
        p = -1;
      } else if (r == PASS_EXIT) {
        // the exit point becomes the last pathline point
        const int face = V.exitFace;
        lc = c; lx = ox; ly = oy; lz = oz; lt = V.t;
        // the neighbour through the exit face, read from the cell's record
        // (not held in registers through the visit)
        const int32_t nc = __ldg(&a.recs[c].conn[face - 1]);
        // ConvertFromNeighbor: the exit coordinate must sit exactly on the face
        const bool bad = sizeof(R) == 8
                             ? (face == 2 && !is1(ox)) || (face == 1 && !is0(ox)) || (face == 4 && !is1(oy)) ||
                                   (face == 3 && !is0(oy)) || (face == 6 && !is1(oz)) || (face == 5 && !is0(oz))
                             : (face == 2 && ox != one) || (face == 1 && ox != zero) || (face == 4 && oy != one) ||
                                   (face == 3 && oy != zero) || (face == 6 && oz != one) || (face == 5 && oz != zero);
        if (nc < 0 || bad) {
          a.cell[p] = lc; a.x[p] = lx; a.y[p] = ly; a.z[p] = lz; a.t[p] = lt;
          a.status[p] = (nc < 0) ? ST_BOUNDARY : ST_UNDEFINED;
          a.ctr[p] = ctr;
          p = -1;
        } else {
          ex = ox; ey = oy; ez = oz; et = V.t;
          if (face == 2) ex = zero;
          if (face == 1) ex = one;
          if (face == 4) ey = zero;
          if (face == 3) ey = one;
          if (face == 6) ez = zero;
          if (face == 5) ez = one;
          c = nc;
          need_cell = true;
        }
      }
    }
  }
  // block-level sum of passes, one atomic per block
  __shared__ unsigned long long blk;
  if (threadIdx.x == 0) blk = 0;
  __syncthreads();
  atomicAdd(&blk, (unsigned long long)my_passes);
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(reinterpret_cast<unsigned long long *>(a.steps), blk);
}

// the lanes' records, the exchange slots (FP64 or EXPONENTIAL; EULERIAN leaves
// their last field out) and the EXPONENTIAL kernel's visit values
template <typename R>
static size_t advance_smem_bytes(int threads, int exp_adv) {
  const int extra = exp_adv ? kExitSlot + kExpFields : (sizeof(R) == 8 ? kExitSlot - 1 : 0);
  return (kRecUnits<R> * 16 + extra * sizeof(double)) * threads;
}

// A kernel's shared-memory limit is the process's, so it is the same at every
// launch, whatever the block: a launch of few threads that lowered it to its
// own size would have another host thread's launch of many refused.
template <typename R, typename Kern>
static cudaError_t raise_smem_limit(Kern kern, int exp_adv) {
  const size_t most = advance_smem_bytes<R>(step_threads(sizeof(R) == 8, exp_adv != 0), exp_adv);
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

template <typename R>
cudaError_t launch_advance(const AdvanceArgs<R> &a, int blocks, int threads, cudaStream_t s) {
  size_t smem = advance_smem_bytes<R>(threads, a.exp_adv);
  auto kern = a.exp_adv ? (a.axi ? rwpt_advance_kernel<R, true, true> : rwpt_advance_kernel<R, true, false>)
                        : (a.axi ? rwpt_advance_kernel<R, false, true> : rwpt_advance_kernel<R, false, false>);
  cudaError_t e = raise_smem_limit<R>(kern, a.exp_adv);
  if (e != cudaSuccess) return e;
  kern<<<blocks, threads, smem, s>>>(a);
  return cudaGetLastError();
}

template <typename R>
cudaError_t advance_occupancy(int exp_adv, int axi, int threads, int *blocks_per_sm) {
  size_t smem = advance_smem_bytes<R>(threads, exp_adv);
  auto kern = exp_adv ? (axi ? rwpt_advance_kernel<R, true, true> : rwpt_advance_kernel<R, true, false>)
                      : (axi ? rwpt_advance_kernel<R, false, true> : rwpt_advance_kernel<R, false, false>);
  cudaError_t e = raise_smem_limit<R>(kern, exp_adv);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kern, threads, smem);
}

template cudaError_t launch_advance<double>(const AdvanceArgs<double> &, int, int, cudaStream_t);
template cudaError_t advance_occupancy<double>(int, int, int, int *);
template cudaError_t advance_occupancy<float>(int, int, int, int *);
template cudaError_t launch_advance<float>(const AdvanceArgs<float> &, int, int, cudaStream_t);

}  // namespace mprw
