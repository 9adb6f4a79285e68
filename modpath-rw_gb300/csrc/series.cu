// series.cu -- the 1-D GPKDE of observation time series (breakthrough curves).
//
// The observation post-process (MPathRW.F90:1759-2840) reconstructs every
// observation's breakthrough curve from the record times of its particles
// with a one-dimensional GridProjectedKDE whose kernel database is off
// (databaseOptimization = .false.): every bin's kernels are set up from its
// exact smoothing (prSetKernelBrute / prSetKernelSigmaBrute /
// prSetKernelSD1DBrute, GridProjectedKDE.F90:6224-6317) instead of being
// looked up.  The time grid is small (10^2..10^5 bins), so the kernels are
// evaluated on the fly: one warp per active bin computes its taps (erf
// differences for W, the Gaussian-derivative differences for the second
// derivative), folds them at the grid ends exactly as prKernelReflection
// does, and gathers from or scatters into the grid.  Reductions run in one
// block in a fixed order; the host takes the per-loop convergence decision
// from a few scalars, as for the spatial reconstruction.
//
// Host-side scalar arithmetic (bin sizes, grid sizes, the initial smoothing,
// effective masses) is done in double precision on the host from sums and
// order statistics the device computes, in the reference's order of
// operations (Histogram.F90:603-720, GridProjectedKDE.F90:3794-4110).
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "../../include/mprw_gpu.h"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRed = 1024;                   // single-block reductions
// Time grids of at most 2^20 bins: a loop costs up to (active bins) x
// (kernel width) tap evaluations, and kernels may grow to 0.9 of the grid.
constexpr int64_t kMaxSeriesBins = 1 << 20;
constexpr double kBorderFraction = 0.05;     // defaultBorderFraction
constexpr double kDefaultInitialFactor = 2.0;
constexpr double kSqrt2 = 1.4142135623730951;

enum {
  S_SUMX, S_MINX, S_MAXX, S_SUMW, S_SUMW2, S_BAD, S_SUMDX2,
  S_MAXD, S_MAXD_OLD, S_ERRD, S_ERRS, S_ALMISE, S_NETMAX, S_MAXSCALE, S_NA, S_SUMABSW,
  S_ORDER,  // four order statistics
  S_COUNT = S_ORDER + 4
};

// Constants of one reconstruction (1-D, nd = 1).
struct SerParams {
  int G;             // bins of the grid
  double b;          // bin size (= bin volume = bin distance in 1-D)
  double max_k, min_k, max_sd, min_sd;
  double support_c, alpha_c, beta_c, one_over_nd4, minus_one_over_nd6, one_plus_nd_quarter;
  double sqrt8pi, fourpi_half, max_sigma_growth, npts2;
  double shape_term; // (1/(nd+4) * 5)^(-1/(nd+6)): the curvature bandwidth's shape factor at shape 1
  double sd_c0;      // 2^(nd - 1/2) * sqrt(pi)
};

struct SerBins {
  int na;
  const int *act;    // 0-based grid index of each active bin, ascending
  double *cnt, *wcnt, *ks, *scale, *scale_old, *support, *nest, *netr, *cb, *darr, *darr_old;
};

// ---------------------------------------------------------------------------
// kernel taps
// ---------------------------------------------------------------------------
// W taps of bandwidth h (range 3): zp(k) = 0.5 (erf((k+1/2)/(hd sqrt2)) -
// erf((k-1/2)/(hd sqrt2))), unfolded to 2m+1 entries and divided by their sum
// (KernelMultiGaussian.f90:549-590, 720-790).
struct WTap {
  int m;
  double hs2;   // hd * sqrt(2)
  double sum;
  __device__ double zp(int k) const { return 0.5 * (erf((k + 0.5) / hs2) - erf((k - 0.5) / hs2)); }
};

// Second-derivative taps of bandwidth h (range 4) along the only dimension:
// zp(k) = c ((k+1/2) e^{-(k+1/2)^2/(2 hd^2)} - (k-1/2) e^{-(k-1/2)^2/(2 hd^2)}),
// c = -1/(2^(1/2) sqrt(pi) hd^3); never rescaled (KernelMultiGaussian.f90:794-887).
struct SdTap {
  int m;
  double hd, c;
  __device__ double zp(int k) const {
    const double a = k + 0.5, d = k - 0.5;
    return c * (a * exp(-1.0 * (a * a) / (2.0 * (hd * hd))) - d * exp(-1.0 * (d * d) / (2.0 * (hd * hd))));
  }
};

// The value at grid position p (1-based) of the unfolded kernel centred on
// g, zero outside [g-m, g+m].
template <typename Tap>
__device__ inline double tap_at(const Tap &t, int p, int g, double norm) {
  const int j = p - g;
  if (j < -t.m || j > t.m) return 0.0;
  const double v = t.zp(j < 0 ? -j : j);
  return norm != 0.0 ? v / norm : v;
}

// prKernelReflection in 1-D: taps below position 1 are added onto 1-p
// (low fold first), then taps above G (including folded ones) onto 2G+1-p.
// Every fold target lies inside the (2m+1) matrix, so the value at q in
// [max(g-m,1), min(g+m,G)] is (w(q) + w(1-q)) + (w(2G+1-q) + w(q-2G)) in the
// reference's order of additions (a missing term is an exact zero).
template <typename Tap>
__device__ inline double folded(const Tap &t, int q, int g, int G, double norm) {
  return (tap_at(t, q, g, norm) + tap_at(t, 1 - q, g, norm)) +
         (tap_at(t, 2 * G + 1 - q, g, norm) + tap_at(t, q - 2 * G, g, norm));
}

struct MinOp {
  __device__ double operator()(double a, double b) const { return fmin(a, b); }
};
struct MaxOp {
  __device__ double operator()(double a, double b) const { return fmax(a, b); }
};

__device__ inline double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ inline SdTap make_sd(double h, double b, double c0) {
  SdTap t;
  t.m = (int)ceil(4.0 * h / b);
  t.hd = h / b;
  t.c = -1.0 / (c0 * pow(t.hd, 3.0));
  return t;
}

// ---- one block per bin ----
// The taps of neighbouring distances share their erf (or exp) values, and
// both halves of a kernel are equal, so a block evaluates each value once into
// shared memory (kernels of up to kTapCap distances; wider ones evaluate every
// tap where it is used): 1 erf per distance instead of 4 and, with the folded
// gather's own, 8.  With four warps per bin the ~500 bins of a curve occupy
// every SM (one warp per bin left each with three).  1,000,000 records in 560
// bins, per launch: nEstimate 127 -> 22 us, roughness 70 -> 13, the density's
// gather from the table 21 -> 5, curvature 22 -> 6.
constexpr int kTapThreads = 128;
constexpr int kTapCap = 2048;
constexpr int64_t kTableBytes = 32 << 20;  // tap tables up to this size

struct TapShared {
  double e[kTapCap];
  double red[kTapThreads / 32];
};

__device__ inline double block_sum(double v, double *red) {
  v = warp_sum(v);
  __syncthreads();  // red is free
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = red[0];
  for (int k = 1; k < kTapThreads / 32; ++k) t += red[k];
  return t;
}

// W taps of smoothing h from the block's erf values (or evaluated)
struct WTapBlock {
  WTap t;
  const double *e;  // erf((k + 1/2) / hs2), k = 0..m, or null
  __device__ double zp(int k) const {
    if (!e) return t.zp(k);
    return k == 0 ? e[0] : 0.5 * (e[k] - e[k - 1]);
  }
};

__device__ inline WTapBlock make_w_block(double h, double b, TapShared &sh) {
  WTapBlock w;
  w.t.m = (int)ceil(3.0 * h / b);
  w.t.hs2 = (h / b) * kSqrt2;
  w.e = w.t.m < kTapCap ? sh.e : nullptr;
  __syncthreads();  // sh.e is free
  if (w.e)
    for (int k = threadIdx.x; k <= w.t.m; k += kTapThreads) sh.e[k] = erf((k + 0.5) / w.t.hs2);
  __syncthreads();
  double s = 0.0;
  for (int k = threadIdx.x; k <= w.t.m; k += kTapThreads) s += (k ? 2.0 : 1.0) * w.zp(k);
  w.t.sum = block_sum(s, sh.red);
  return w;
}

// sum over the kernel's span of field * folded W taps (every thread gets it)
__device__ inline double w_gather(const double *field, double h, int g, const SerParams &P, TapShared &sh) {
  if (h == 0.0) return 0.0;
  const WTapBlock w = make_w_block(h, P.b, sh);
  const int m = w.t.m, q0 = max(g - m, 1), q1 = min(g + m, P.G);
  auto at = [&](int p) {
    const int j = p < g ? g - p : p - g;
    return j <= m ? w.zp(j) : 0.0;
  };
  const bool inside = g - m >= 1 && g + m <= P.G;
  double acc = 0.0;
  for (int q = q0 + threadIdx.x; q <= q1; q += kTapThreads) {
    double v = at(q);
    if (!inside) v = (v + at(1 - q)) + (at(2 * P.G + 1 - q) + at(q - 2 * P.G));
    acc += field[q - 1] * v;
  }
  return block_sum(acc, sh.red) / w.t.sum;
}

// ---------------------------------------------------------------------------
// statistics, histogram, active bins
// ---------------------------------------------------------------------------
// Statistics of the records: kStatBlocks blocks reduce their shares, one
// block the partial results, in a fixed order (1,000,000 records: one block
// took 2.59 ms and, for the variance, 0.57 ms; these 0.03 and 0.01 ms).
constexpr int kStat = 7;  // slots S_SUMX..S_BAD and S_SUMABSW, in this order
constexpr int kStatBlocks = 304;

__global__ void __launch_bounds__(kThreads) ser_stats_kernel(const double *x, const double *w, int64_t n,
                                                             double *part) {
  using BR = cub::BlockReduce<double, kThreads>;
  __shared__ typename BR::TempStorage tmp;
  double v[kStat] = {0.0, INFINITY, -INFINITY, 0.0, 0.0, 0.0, 0.0};
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    const double xi = x[i], wi = w[i];
    if (!isfinite(xi) || !isfinite(wi)) v[5] += 1.0;
    v[0] += xi;
    v[1] = fmin(v[1], xi);
    v[2] = fmax(v[2], xi);
    v[3] += wi;
    v[4] += wi * wi;
    v[6] += fabs(wi);
  }
#pragma unroll
  for (int k = 0; k < kStat; ++k) {
    const double r = k == 1 ? BR(tmp).Reduce(v[k], MinOp()) : (k == 2 ? BR(tmp).Reduce(v[k], MaxOp()) : BR(tmp).Sum(v[k]));
    if (threadIdx.x == 0) part[k * gridDim.x + blockIdx.x] = r;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kThreads) ser_stats_final_kernel(const double *part, int nblk, double *S) {
  using BR = cub::BlockReduce<double, kThreads>;
  __shared__ typename BR::TempStorage tmp;
  const int slot[kStat] = {S_SUMX, S_MINX, S_MAXX, S_SUMW, S_SUMW2, S_BAD, S_SUMABSW};
  const int k = blockIdx.x;
  double v = k == 1 ? INFINITY : (k == 2 ? -INFINITY : 0.0);
  for (int i = threadIdx.x; i < nblk; i += kThreads) {
    const double p = part[k * nblk + i];
    v = k == 1 ? fmin(v, p) : (k == 2 ? fmax(v, p) : v + p);
  }
  const double r = k == 1 ? BR(tmp).Reduce(v, MinOp()) : (k == 2 ? BR(tmp).Reduce(v, MaxOp()) : BR(tmp).Sum(v));
  if (threadIdx.x == 0) S[slot[k]] = r;
}

// sum of squared deviations from the mean S[S_SUMX] / n
__global__ void __launch_bounds__(kThreads) ser_var_kernel(const double *x, int64_t n, const double *S, double *part) {
  using BR = cub::BlockReduce<double, kThreads>;
  __shared__ typename BR::TempStorage tmp;
  const double mean = S[S_SUMX] / (double)n;
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    const double d = x[i] - mean;
    v += d * d;
  }
  const double r = BR(tmp).Sum(v);
  if (threadIdx.x == 0) part[blockIdx.x] = r;
}

// the second stage of ser_var_kernel, and the order statistics of the sorted
// records that the automatic bin size reads (1-based elements; 0: none)
struct OrderIdx {
  int64_t i[4];
};
__global__ void __launch_bounds__(kThreads) ser_var_final_kernel(const double *part, int nblk, const double *sorted,
                                                                 OrderIdx q, double *S) {
  using BR = cub::BlockReduce<double, kThreads>;
  __shared__ typename BR::TempStorage tmp;
  double v = 0.0;
  for (int i = threadIdx.x; i < nblk; i += kThreads) v += part[i];
  const double r = BR(tmp).Sum(v);
  if (threadIdx.x == 0) S[S_SUMDX2] = r;
  if (threadIdx.x < 4 && q.i[threadIdx.x] > 0) S[S_ORDER + threadIdx.x] = sorted[q.i[threadIdx.x] - 1];
}

// Histogram%ComputeCounts{Weighted,AndWeights} / ComputeEffectiveCountsAndWeights
// (Histogram.F90:276-490): bin = floor((t - origin)/binSize) + 1 (+ 0 for an
// exact point), points outside [1, G] skipped.  The sums are 64-bit
// fixed-point integers (scale 2^shift_c for counts, 2^shift_w for wcounts,
// chosen by the host from the totals so that no sum overflows): integer
// additions do not depend on the order of the atomics, so the histogram is
// bit-for-bit repeatable; ser_fixed_kernel turns them into doubles.
// A block first adds into its own copy in shared memory when that fits (the
// grids have 10^2-10^4 bins: a million global atomics on 560 addresses took
// 199 us, these 39).
constexpr int kHistThreads = 512;
constexpr size_t kHistShared = 96 * 1024;

template <bool SHARED>
__global__ void __launch_bounds__(kHistThreads) ser_hist_kernel(const double *x, const double *w, int64_t n,
                                                                double origin, double b, int G, int exact, int fmt,
                                                                double sc, double sw, unsigned long long *counts,
                                                                unsigned long long *wcounts) {
  extern __shared__ unsigned long long sh[];
  const int total = fmt >= 2 ? 2 * G : G;
  if (SHARED) {
    for (int k = threadIdx.x; k < total; k += blockDim.x) sh[k] = 0ull;
    __syncthreads();
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double q = floor((x[i] - origin) / b) + (exact ? 0.0 : 1.0);
    if (!(q >= 1.0 && q <= (double)G)) continue;
    const int k = (int)q - 1;
    const double wi = w[i];
    const double c = fmt == 2 ? 1.0 : (fmt == 3 ? wi * wi : wi);
    atomicAdd((SHARED ? sh : counts) + k, (unsigned long long)__double2ll_rn(c * sc));
    if (fmt >= 2) atomicAdd((SHARED ? sh + G : wcounts) + k, (unsigned long long)__double2ll_rn(wi * sw));
  }
  if (SHARED) {
    __syncthreads();
    for (int k = threadIdx.x; k < total; k += blockDim.x)
      if (sh[k]) atomicAdd(k < G ? counts + k : wcounts + (k - G), sh[k]);
  }
}

__global__ void ser_fixed_kernel(const unsigned long long *a, double inv, double *out, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = (double)(long long)a[i] * inv;
}

// mode 0: a /= f; mode 1: a *= f; mode 2: format 3's effective counts
// (counts = wcounts^2 / counts where counts != 0)
__global__ void ser_grid_op_kernel(double *a, const double *bw, int G, int mode, double f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < G; i += gridDim.x * blockDim.x) {
    if (mode == 0) a[i] = a[i] / f;
    else if (mode == 1) a[i] = a[i] * f;
    else if (a[i] != 0.0) a[i] = bw[i] * bw[i] / a[i];
  }
}

// active bins (counts != 0) in ascending order (Histogram.F90:493-527)
__global__ void __launch_bounds__(kRed) ser_active_kernel(const double *counts, const double *wcounts, int G,
                                                          int *act, double *cnt, double *wcnt, double *S) {
  using BS = cub::BlockScan<int, kRed>;
  __shared__ typename BS::TempStorage tmp;
  __shared__ int base;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  for (int c0 = 0; c0 < G; c0 += kRed) {
    const int i = c0 + threadIdx.x;
    const int flag = (i < G && counts[i] != 0.0) ? 1 : 0;
    int ofs, total;
    BS(tmp).ExclusiveSum(flag, ofs, total);
    if (flag) {
      const int k = base + ofs;
      act[k] = i;
      cnt[k] = counts[i];
      wcnt[k] = wcounts ? wcounts[i] : 0.0;
    }
    __syncthreads();
    if (threadIdx.x == 0) base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) S[S_NA] = (double)base;
}

// ---------------------------------------------------------------------------
// the optimisation loop (GridProjectedKDE.F90:4396-5160, nd = 1)
// ---------------------------------------------------------------------------
// kernelSmoothing = initial smoothing; scale = its geometric mean (itself in
// 1-D, zero for a zero smoothing); support = 2 scale; shape = 1.
__global__ void ser_init_kernel(SerBins B, double hs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B.na) return;
  B.ks[i] = hs;
  const double sc = hs;
  B.scale[i] = sc;
  B.scale_old[i] = sc;
  B.support[i] = 2.0 * sc;
  B.nest[i] = 0.0;
  B.netr[i] = 0.0;
}

// density: the sum of (w)counts times the folded W taps of kernelSmoothing
// (check_negative skips a negative smoothing, the first estimate, :4640).
// The reference scatters bin by bin in ascending order; here each grid
// position gathers the bins whose folded kernel reaches it, in the same
// ascending order, so the sums are the reference's and repeatable.  First the
// taps of every bin (one warp per bin; m = -1 for a bin that adds nothing)
// and the largest half-width, then the gather.
// With a table (tab, stride entries per bin) the normalised taps are stored too.
__global__ void __launch_bounds__(kTapThreads) ser_wtap_kernel(SerParams P, SerBins B, int check_negative, WTap *taps,
                                                               int *mmax, double *tab, int stride) {
  __shared__ TapShared sh;
  const int i = blockIdx.x;
  const double h = B.ks[i];
  if ((check_negative && h < 0.0) || h == 0.0) {
    if (threadIdx.x == 0) taps[i].m = -1;
    return;
  }
  const WTapBlock w = make_w_block(h, P.b, sh);
  if (tab)
    for (int k = threadIdx.x; k <= w.t.m; k += kTapThreads) tab[(int64_t)i * stride + k] = w.zp(k) / w.t.sum;
  if (threadIdx.x == 0) {
    taps[i] = w.t;
    atomicMax(mmax, w.t.m);
  }
}

// the first active bin index whose grid position (1-based) is >= g
__device__ inline int first_bin_at(const SerBins &B, int g) {
  int lo = 0, hi = B.na;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (B.act[mid] + 1 < g) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// out[q-1] = sum over the bins i reaching q of val[i] * folded taps: one warp
// per grid position, lane l taking the candidate bins l, l+32, ... in
// ascending order, then a fixed shuffle tree -- a fixed order, so the sum is
// the same on every run.
// With a table the taps are read instead of evaluated.
template <typename Tap, bool NORM>
__global__ void __launch_bounds__(kThreads) ser_gather_kernel(SerParams P, SerBins B, const Tap *taps,
                                                              const int *mmax, const double *val, const double *tab,
                                                              int stride, double *out) {
  const int M = *mmax;
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * kWarps + (threadIdx.x >> 5) + 1;
  if (q > P.G) return;  // warp-uniform
  double acc = 0.0;
  if (M >= 0) {
    for (int i = first_bin_at(B, q - M) + lane; i < B.na && B.act[i] + 1 <= q + M; i += 32) {
      const Tap t = taps[i];
      const int g = B.act[i] + 1;
      if (t.m < 0 || q < g - t.m || q > g + t.m) continue;
      if (tab) {
        const double *row = tab + (int64_t)i * stride;
        auto at = [&](int p) {
          const int j = p < g ? g - p : p - g;
          return j <= t.m ? row[j] : 0.0;
        };
        acc += val[i] * ((at(q) + at(1 - q)) + (at(2 * P.G + 1 - q) + at(q - 2 * P.G)));
        continue;
      }
      double norm = 0.0;
      if constexpr (NORM) norm = t.sum;
      acc += val[i] * folded(t, q, g, P.G, norm);
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) out[q - 1] = acc;
}

// nEstimate with the current support, the support update, nEstimate again
// (GridProjectedKDE.F90:4826-4880)
// (the powers 1/2, 5/4 and 1/4 as square roots)
__global__ void __launch_bounds__(kTapThreads) ser_nest_kernel(SerParams P, SerBins B, const double *dens) {
  __shared__ TapShared sh;
  const int i = blockIdx.x;
  const int g = B.act[i] + 1;
  const double dn = dens[g - 1];
  double ssc = B.support[i];
  const double kscale = B.scale[i];
  double ne = w_gather(dens, ssc, g, P, sh);
  ssc = sqrt(ne) * (kscale * sqrt(sqrt(kscale))) / sqrt(sqrt(4.0 * dn)) * P.support_c;
  if (ssc > P.max_sigma_growth * B.support[i]) ssc = P.max_sigma_growth * B.support[i];
  ssc = fmin(ssc, P.max_k);
  if (ssc < P.min_k) ssc = P.min_k;
  ne = w_gather(dens, ssc, g, P, sh);
  if (threadIdx.x == 0) {
    B.nest[i] = ne;
    B.support[i] = ssc;
  }
}

// curvature bandwidth (GridProjectedKDE.F90:5207-5275), shape = 1
__global__ void ser_cb_kernel(SerParams P, SerBins B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B.na) return;
  const double d = B.darr[i];
  double nvpb = 0.0;
  if (d > 0.0) {
    const double p = P.sqrt8pi * B.support[i];
    nvpb = pow(p * (B.nest[i] * B.nest[i]) / d, P.beta_c);
  }
  double cb = P.alpha_c * nvpb * P.shape_term * B.scale[i];
  if (cb > P.max_sd) cb = P.max_sd;
  if (cb < P.min_sd) cb = P.min_sd;
  B.cb[i] = cb;
}

// curvature: the sum of counts times the second-derivative taps of the
// curvature bandwidth (prComputeNetRoughness1D, GridProjectedKDE.F90:1666-1760),
// as a gather like the density: the taps of every bin (m = -1 where the
// reference skips the bin: a negative, NaN or zero bandwidth, or a kernel
// whose sum of squares is zero), then ser_gather_kernel<SdTap, false>.
__global__ void __launch_bounds__(kTapThreads) ser_sdtap_kernel(SerParams P, SerBins B, SdTap *taps, int *mmax,
                                                                double *tab, int stride) {
  __shared__ TapShared sh;
  const int i = blockIdx.x;
  const double h = B.cb[i];
  if (h < 0.0 || h != h || h == 0.0) {
    if (threadIdx.x == 0) taps[i].m = -1;
    return;
  }
  const SdTap t = make_sd(h, P.b, P.sd_c0);
  // the sum of squares decides a zero kernel; its first term alone when positive
  const double v0 = t.zp(0);
  double ss = v0 * v0;
  if (!(ss > 0.0)) {
    double s = 0.0;
    for (int k = threadIdx.x; k <= t.m; k += kTapThreads) {
      const double v = t.zp(k);
      s += (k ? 2.0 : 1.0) * (v * v);
    }
    ss = block_sum(s, sh.red);
  }
  if (ss <= 0.0) {
    if (threadIdx.x == 0) taps[i].m = -1;
    return;
  }
  if (tab) {
    // zp(k) = c (X(k) - X(k-1)), X(k) = (k+1/2) e^{-(k+1/2)^2/(2 hd^2)}, X(-1) = -X(0)
    const bool cached = t.m < kTapCap;
    if (cached) {
      for (int k = threadIdx.x; k <= t.m; k += kTapThreads) {
        const double a = k + 0.5;
        sh.e[k] = a * exp(-1.0 * (a * a) / (2.0 * (t.hd * t.hd)));
      }
      __syncthreads();
    }
    for (int k = threadIdx.x; k <= t.m; k += kTapThreads)
      tab[(int64_t)i * stride + k] = cached ? t.c * (sh.e[k] - (k ? sh.e[k - 1] : -sh.e[0])) : t.zp(k);
  }
  if (threadIdx.x == 0) {
    taps[i] = t;
    atomicMax(mmax, t.m);
  }
}

// curvature / binVolume / binSize^2, squared
__global__ void ser_curv_square_kernel(double *curv, int G, double b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < G; i += gridDim.x * blockDim.x) {
    double c = curv[i] / b;
    c = c / (b * b);
    curv[i] = c * c;
  }
}

// roughness: W gather of the squared curvature with the support; the raw
// optimal scale where the roughness is positive (GridProjectedKDE.F90:5404-5440)
__global__ void __launch_bounds__(kTapThreads) ser_rough_kernel(SerParams P, SerBins B, const double *curv) {
  __shared__ TapShared sh;
  const int i = blockIdx.x;
  const int g = B.act[i] + 1;
  const double r = w_gather(curv, B.support[i], g, P, sh);
  if (threadIdx.x == 0) {
    B.netr[i] = r;
    B.scale[i] = (r > 0.0) ? pow(1.0 * B.nest[i] / (P.fourpi_half * r), P.one_over_nd4) : 0.0;
  }
}

// max net roughness and max positive scale
__global__ void __launch_bounds__(kRed) ser_rough_reduce_kernel(SerBins B, double *S) {
  using BR = cub::BlockReduce<double, kRed>;
  __shared__ typename BR::TempStorage tmp;
  double mr = -INFINITY, ms = 0.0;
  for (int i = threadIdx.x; i < B.na; i += kRed) {
    mr = fmax(mr, B.netr[i]);
    if (B.scale[i] > 0.0) ms = fmax(ms, B.scale[i]);
  }
  double r = BR(tmp).Reduce(mr, MaxOp());
  if (threadIdx.x == 0) S[S_NETMAX] = r;
  __syncthreads();
  r = BR(tmp).Reduce(ms, MaxOp());
  if (threadIdx.x == 0) S[S_MAXSCALE] = r;
}

// zero roughness takes the largest scale; kernelSmoothing = scale bounded to
// [minKernelSize, maxKernelSize]; the scale of a 1-D kernel is the kernel
// itself (GridProjectedKDE.F90:5440-5724)
__global__ void ser_optimal_kernel(SerParams P, SerBins B, const double *S) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B.na) return;
  double sc = B.scale[i];
  if (B.netr[i] == 0.0) sc = S[S_MAXSCALE];
  double k = 1.0 * sc;
  if (k > P.max_k) k = P.max_k;
  if (k < P.min_k) k = P.min_k;
  B.ks[i] = k;
  B.scale[i] = k;
}

// previous density and scale (saved at the start of each loop)
__global__ void ser_loop_init_kernel(SerBins B, double *S) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) S[S_MAXD_OLD] = S[S_MAXD];
  if (i >= B.na) return;
  B.darr_old[i] = B.darr[i];
  B.scale_old[i] = B.scale[i];
}

// density grid / binVolume; density at the active bins; the convergence
// measures (GridProjectedKDE.F90:4960-5040)
__global__ void ser_dens_finish_kernel(double *dens, int G, double b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < G; i += gridDim.x * blockDim.x) dens[i] = dens[i] / b;
}

__global__ void __launch_bounds__(kRed) ser_measures_kernel(SerParams P, SerBins B, const double *dens, double *S) {
  using BR = cub::BlockReduce<double, kRed>;
  __shared__ typename BR::TempStorage tmp;
  __shared__ double smax;
  double mx = -INFINITY;
  for (int i = threadIdx.x; i < B.na; i += kRed) {
    const double d = dens[B.act[i]];
    B.darr[i] = d;
    mx = fmax(mx, d);
  }
  const double r = BR(tmp).Reduce(mx, MaxOp());
  if (threadIdx.x == 0) {
    smax = r;
    S[S_MAXD] = r;
  }
  __syncthreads();
  const double mo = S[S_MAXD_OLD];
  double ed = 0.0, es = 0.0, ea = 0.0;
  for (int i = threadIdx.x; i < B.na; i += kRed) {
    const double d = B.darr[i], o = B.darr_old[i];
    if (o != 0.0) {
      const double e = fabs(d / smax - o / mo) / (o / mo);
      ed += e * e;
    }
    const double sc = B.scale[i], so = B.scale_old[i];
    if (so != 0.0) {
      const double e = fabs(sc - so) / so;
      es += e * e;
    }
    if (sc != 0.0) {
      const double e = (B.nest[i] / (sc * P.fourpi_half) + 0.25 * B.netr[i] * ((sc * sc) * (sc * sc))) / P.npts2;
      ea += e * e;
    }
  }
  double v = BR(tmp).Sum(ed);
  if (threadIdx.x == 0) S[S_ERRD] = v;
  __syncthreads();
  v = BR(tmp).Sum(es);
  if (threadIdx.x == 0) S[S_ERRS] = v;
  __syncthreads();
  v = BR(tmp).Sum(ea);
  if (threadIdx.x == 0) S[S_ALMISE] = v;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
int rc_of(cudaError_t e) { return e == cudaErrorMemoryAllocation ? MPRW_E_OOM : MPRW_E_CUDA; }

#define SCK(x)                          \
  do {                                  \
    cudaError_t e_ = (x);               \
    if (e_ != cudaSuccess) {            \
      (void)cudaGetLastError();         \
      return rc_of(e_);                 \
    }                                   \
  } while (0)

int blocks_of(int64_t n, int threads) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 152 * 16));
}

// Q1 and Q3 as prEstimateBinSizeFD picks them from the sorted points
// (Histogram.F90:680-712): the 1-based elements i[0] (and i[1]) whose mean is
// Q1, i[2] (and i[3]) for Q3; i[1] = i[3] = 0 where one element is taken.
OrderIdx fd_elements(int64_t n) {
  if (n % 2 == 0) {
    if (std::fmod((double)n / 2.0, 2.0) == 0.0) return {{n / 4, n / 4 + 1, n / 2 + n / 4, n / 2 + n / 4 + 1}};
    return {{n / 4 + 1, 0, n / 2 + n / 4 + 1, 0}};
  }
  const int64_t m = (n - 1) / 4;
  if (std::fmod((double)(n - 1) / 2.0, 2.0) == 0.0) return {{m, m + 1, n / 2 + 1 + m, n / 2 + 1 + m + 1}};
  return {{m + 1, 0, n / 2 + 1 + m + 1, 0}};
}

// Device memory of one call: two blocks (the records', then the grid's),
// handed out in 256-byte pieces; every cudaMalloc and cudaFree costs about as
// much as a kernel, and the call used 24 of each.
struct Arena {
  char *base = nullptr;
  size_t size = 0, used = 0;
  ~Arena() {
    if (base) cudaFree(base);
  }
  static size_t up(size_t b) { return (std::max<size_t>(b, 1) + 255) / 256 * 256; }
  cudaError_t open(size_t bytes) {
    size = bytes;
    return cudaMalloc(reinterpret_cast<void **>(&base), bytes);
  }
  template <typename T>
  T *take(int64_t n) {
    T *p = reinterpret_cast<T *>(base + used);
    used += up(sizeof(T) * (size_t)std::max<int64_t>(n, 1));
    return used <= size ? p : nullptr;
  }
};

}  // namespace

extern "C" int mprw_gpkde_series(const double *times, const double *weights, int64_t n,
                                 const mprw_series_options *o, int32_t capacity, double *counts_out,
                                 double *wcounts_out, double *density_out, mprw_series_result *res, void *stream) {
  if (!times || !weights || !o || !res || !counts_out || n < 1 || n > (int64_t)INT32_MAX) return MPRW_E_INVAL;
  *res = mprw_series_result{};
  const int fmt = o->effective_weight_format;
  if (o->bin_format < 0 || o->bin_format > 3 || fmt < 0 || fmt > 3 || o->initial_smoothing_selection < 0 ||
      o->initial_smoothing_selection > 2 || o->n_opt_loops < 0 || !std::isfinite(o->rel_err_convergence) ||
      !std::isfinite(o->origin) || !std::isfinite(o->domain_size) || !std::isfinite(o->bin_size) ||
      !std::isfinite(o->initial_smoothing_factor) || o->domain_size < 0.0 || (!o->adapt_grid && o->domain_size <= 0.0))
    return MPRW_E_INVAL;
  if (o->bin_format <= 1 && !(o->bin_size_fraction > 0.0 && o->bin_size_fraction <= 2.0)) return MPRW_E_INVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (o->bin_format == 1 && n < 2) return MPRW_E_INVAL;
  Arena rec;
  size_t tb = 0;
  if (o->bin_format == 1)
    SCK(cub::DeviceRadixSort::SortKeys(nullptr, tb, (const double *)nullptr, (double *)nullptr, (int)n, 0, 64, s));
  const int sblk = (int)std::max<int64_t>(1, std::min<int64_t>((n + kThreads - 1) / kThreads, kStatBlocks));
  const size_t nb8 = Arena::up(sizeof(double) * (size_t)n);
  SCK(rec.open((o->bin_format == 1 ? 3 : 2) * nb8 + Arena::up(tb) + Arena::up(sizeof(double) * S_COUNT) +
               Arena::up(sizeof(double) * kStat * sblk)));
  double *dx = rec.take<double>(n), *dw = rec.take<double>(n), *S = rec.take<double>(S_COUNT);
  double *part = rec.take<double>(kStat * sblk);
  SCK(cudaMemcpyAsync(dx, times, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  SCK(cudaMemcpyAsync(dw, weights, sizeof(double) * n, cudaMemcpyHostToDevice, s));
  SCK(cudaMemsetAsync(S, 0, sizeof(double) * S_COUNT, s));
  double h[S_COUNT];
  auto fetch = [&](void) -> cudaError_t {
    cudaError_t e = cudaMemcpyAsync(h, S, sizeof(h), cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
  };
  // statistics, and the sorted points of the Freedman-Diaconis bin size
  OrderIdx fd = {{0, 0, 0, 0}};
  double *sorted = nullptr;
  ser_stats_kernel<<<sblk, kThreads, 0, s>>>(dx, dw, n, part);
  ser_stats_final_kernel<<<kStat, kThreads, 0, s>>>(part, sblk, S);
  ser_var_kernel<<<sblk, kThreads, 0, s>>>(dx, n, S, part);
  SCK(cudaGetLastError());
  if (o->bin_format == 1) {
    fd = fd_elements(n);
    sorted = rec.take<double>(n);
    void *tmp = rec.take<char>((int64_t)tb);
    SCK(cub::DeviceRadixSort::SortKeys(tmp, tb, dx, sorted, (int)n, 0, 64, s));
  }
  ser_var_final_kernel<<<1, kThreads, 0, s>>>(part, sblk, sorted, fd, S);
  SCK(cudaGetLastError());
  SCK(fetch());
  if (h[S_BAD] != 0.0) return MPRW_E_INVAL;
  const double nd_n = (double)n;
  const double var = h[S_SUMDX2] / nd_n;
  const double mn = h[S_MINX], mx = h[S_MAXX], delta = std::fabs(mx - mn);
  const double origin = o->origin;
  // domain adapted to the data (GridProjectedKDE.F90:3794-3800)
  double ds = o->domain_size;
  if (o->adapt_grid && ds == 0.0 && delta != 0.0) ds = (mx + 1.0 * kBorderFraction * delta) - origin;
  // bin size (Histogram.F90:603-720; GridProjectedKDE.F90:3806-3890)
  double b = o->bin_size;
  if (o->bin_format == 0) {
    b = (var == 0.0) ? 0.0 : (double)3.49f * std::sqrt(var) / std::pow(nd_n, 1.0 / 3.0);
    b = o->bin_size_fraction * b;
  } else if (o->bin_format == 1) {
    const double *v = h + S_ORDER;
    const double q1 = fd.i[1] ? (v[0] + v[1]) / 2.0 : v[0], q3 = fd.i[3] ? (v[2] + v[3]) / 2.0 : v[2];
    b = 2.0 * (q3 - q1) / std::pow(nd_n, 1.0 / 3.0);
    b = o->bin_size_fraction * b;
  }
  if (!(b > 0.0) || !std::isfinite(b) || ds == 0.0) return MPRW_E_INVAL;
  const double gsd = ds / b + 0.5;
  if (!(gsd < (double)kMaxSeriesBins)) return MPRW_E_INVAL;
  const int gs = (int)gsd;
  if (gs < 2) return MPRW_E_INVAL;
  // the grid: a sub-grid around the data when adapted (:3903-3960)
  int nb = gs, dbo = 0;
  double gorigin = origin;
  if (o->adapt_grid) {
    const double lo = std::max(mn - 0.5 * kBorderFraction * delta, origin);
    const double hi = std::min(mx + 0.5 * kBorderFraction * delta, ds + origin);
    const double od = (lo - origin) / b, ld = std::ceil((hi - origin) / b);
    if (!(od < (double)kMaxSeriesBins) || !(ld < (double)kMaxSeriesBins)) return MPRW_E_INVAL;
    dbo = (int)od;
    nb = (int)ld - dbo;
    gorigin = dbo * b + origin;
    if (nb > gs || nb < 1) return MPRW_E_INVAL;
  }
  res->n_bins = nb;
  res->delta_bins_origin = dbo;
  res->bin_size = b;
  res->grid_origin = gorigin;
  if (nb > capacity) return MPRW_E_SIZE;

  // weighted histogram (Histogram.F90:276-490), fixed-point sums: a bin's
  // sum is at most the total over all records (weights are >= 0), and
  // 2^shift times that stays below 2^62
  const bool wfmt = (fmt >= 2);
  // the grid's memory: counts and fixed-point sums (4), the grids (2), the
  // active bins' index, counts, state (13) and taps, none longer than nb; and
  // a table of every active bin's taps where that stays small (the kernels'
  // sizes are bounded by 0.9 of the domain grid)
  Arena mem;
  const int stride = std::max(4, (int)std::ceil(0.9 * gs) + 2);
  const int64_t tab_n = (int64_t)nb * stride * (int64_t)sizeof(double) <= kTableBytes ? (int64_t)nb * stride : 0;
  SCK(mem.open(Arena::up(sizeof(double) * (size_t)tab_n) + (size_t)20 * Arena::up(sizeof(double) * (size_t)nb) + Arena::up(sizeof(WTap) * (size_t)nb) +
               Arena::up(sizeof(SdTap) * (size_t)nb) + Arena::up(2 * sizeof(int))));
  double *counts = mem.take<double>(nb), *wcounts = wfmt ? mem.take<double>(nb) : nullptr;
  unsigned long long *fc = mem.take<unsigned long long>(nb), *fw = wfmt ? mem.take<unsigned long long>(nb) : nullptr;
  SCK(cudaMemsetAsync(fc, 0, sizeof(unsigned long long) * nb, s));
  if (wfmt) SCK(cudaMemsetAsync(fw, 0, sizeof(unsigned long long) * nb, s));
  auto shift_for = [](double bound) {
    int e = 0;
    std::frexp(std::max(bound, 1e-300), &e);
    return 61 - e;
  };
  {
    // totals of the statistics pass (with a margin for their rounding)
    const double tw = 1.0001 * h[S_SUMABSW], tw2 = 1.0001 * h[S_SUMW2];
    const double cb = fmt == 2 ? (double)n : (fmt == 3 ? tw2 : tw);
    const int shc = shift_for(cb), shw = shift_for(tw);
    const size_t hb = sizeof(unsigned long long) * (size_t)nb * (wfmt ? 2 : 1);
    const int exact = o->exact_point ? 1 : 0;
    // about 16 records per thread, so that the blocks' copies pay
    const int hblk = (int)std::max<int64_t>(1, std::min<int64_t>((n + 16 * kHistThreads - 1) / (16 * kHistThreads), 304));
    if (hb <= kHistShared) {
      SCK(cudaFuncSetAttribute(ser_hist_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHistShared));
      ser_hist_kernel<true><<<hblk, kHistThreads, hb, s>>>(dx, dw, n, gorigin, b, nb, exact, fmt,
                                                           std::ldexp(1.0, shc), std::ldexp(1.0, shw), fc, fw);
    } else {
      ser_hist_kernel<false><<<blocks_of(n, kHistThreads), kHistThreads, 0, s>>>(
          dx, dw, n, gorigin, b, nb, exact, fmt, std::ldexp(1.0, shc), std::ldexp(1.0, shw), fc, fw);
    }
    ser_fixed_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(fc, std::ldexp(1.0, -shc), counts, nb);
    if (wfmt) ser_fixed_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(fw, std::ldexp(1.0, -shw), wcounts, nb);
  }
  double eff = 1.0;
  if (!wfmt) {
    const double total = h[S_SUMW];
    if (fmt == 1) {
      eff = total / nd_n;
    } else {
      const double neff = total * total / h[S_SUMW2];
      eff = total / neff;
    }
    ser_grid_op_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(counts, nullptr, nb, 0, eff);
  } else if (fmt == 3) {
    ser_grid_op_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(counts, wcounts, nb, 2, 0.0);
  }
  SCK(cudaGetLastError());
  auto scale_grid = [&](double *a, int mode, double f) {
    ser_grid_op_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(a, nullptr, nb, mode, f);
  };
  auto copy_out = [&](double *dens) -> cudaError_t {
    cudaError_t e = cudaMemcpyAsync(counts_out, counts, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && wcounts_out) {
      e = wfmt ? cudaMemcpyAsync(wcounts_out, wcounts, sizeof(double) * nb, cudaMemcpyDeviceToHost, s)
               : cudaSuccess;
      if (!wfmt) std::fill(wcounts_out, wcounts_out + nb, 0.0);
    }
    if (e == cudaSuccess && density_out) {
      if (dens) e = cudaMemcpyAsync(density_out, dens, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
      else std::fill(density_out, density_out + nb, 0.0);
    }
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
  };
  if (o->only_histogram) {
    // counts * effective mass, raw density (GridProjectedKDE.F90:3987-4005)
    scale_grid(counts, 1, eff);
    if (o->compute_raw_density) {
      scale_grid(counts, 0, b);
      if (wfmt) scale_grid(wcounts, 0, b);
    }
    SCK(cudaGetLastError());
    SCK(copy_out(nullptr));
    return MPRW_OK;
  }

  // active bins
  int *act = mem.take<int>(nb);
  SerBins B{};
  B.cnt = mem.take<double>(nb);
  B.wcnt = mem.take<double>(nb);
  ser_active_kernel<<<1, kRed, 0, s>>>(counts, wcounts, nb, act, B.cnt, B.wcnt, S);
  SCK(cudaGetLastError());
  SCK(fetch());
  const int na = (int)h[S_NA];
  res->active_bins = na;
  if (na == 0) {
    SCK(copy_out(nullptr));
    return MPRW_OK;
  }
  B.na = na;
  B.act = act;
  for (double **p : {&B.ks, &B.scale, &B.scale_old, &B.support, &B.nest, &B.netr, &B.cb, &B.darr, &B.darr_old})
    *p = mem.take<double>(na);
  SCK(cudaMemsetAsync(B.darr_old, 0, sizeof(double) * na, s));
  double *dens = mem.take<double>(nb), *curv = mem.take<double>(nb);
  WTap *wtaps = mem.take<WTap>(na);
  SdTap *sdtaps = mem.take<SdTap>(na);
  int *mmax = mem.take<int>(2);
  double *tab = tab_n ? mem.take<double>(tab_n) : nullptr;
  if (!mmax || (tab_n && !tab)) return MPRW_E_OOM;

  // data statistics and the initial smoothing (GridProjectedKDE.F90:4020-4110)
  const double std_x = std::sqrt(var);
  double hsig = std_x * std::pow(4.0 / ((1.0 + 2.0) * nd_n), 1.0 / (1.0 + 4.0));
  bool apply = o->apply_initial_factor != 0;
  if (std_x == 0.0) {
    hsig = kDefaultInitialFactor * b;
    apply = false;
  }
  const double fac = o->initial_smoothing_factor;
  double init;
  if (o->initial_smoothing_selection == 0)
    init = (apply && fac > 0.0 && fac != 1.0) ? hsig * fac : hsig;
  else if (o->initial_smoothing_selection == 1)
    init = fac * b;
  else
    init = kDefaultInitialFactor * b;
  // the first support (twice the initial smoothing) is not bounded by the
  // kernel-size limits: refuse one wider than the grid limit
  if (!(init >= 0.0) || !(6.0 * init / b <= (double)kMaxSeriesBins)) return MPRW_E_INVAL;

  // constants of the 1-D reconstruction (prInitializeModuleConstants and
  // the kernel-size bounds of the domain grid, GridProjectedKDE.F90:1296-1310)
  const double nd = 1.0, pi = 4.0 * std::atan(1.0);
  SerParams P{};
  P.G = nb;
  P.b = b;
  P.max_k = b * (0.9 * gs - 1) / 3.0;
  P.max_sd = b * (0.9 * gs - 1) / 4.0;
  P.min_k = 1.2 * b / 3.0;
  P.min_sd = 1.2 * b / 4.0;
  P.support_c = std::pow((nd + 2.0) * std::pow(8.0 * pi, 0.5 * nd), 0.25);
  P.alpha_c = std::pow((1.0 + std::pow(2.0, 0.5 * nd + 2.0)) / (3.0 * std::pow(2.0, 4.0 / (nd + 4.0))),
                       1.0 / (nd + 6.0)) *
              std::pow(nd + 2.0, 1.0 / (nd + 4.0)) / std::pow(nd + 4.0, 1.0 / (nd + 6.0));
  P.beta_c = 2.0 / (nd + 4.0) / (nd + 6.0);
  P.one_over_nd4 = 1.0 / (nd + 4.0);
  P.minus_one_over_nd6 = -1.0 / (nd + 6.0);
  P.one_plus_nd_quarter = 1.0 + 0.25 * nd;
  P.sqrt8pi = std::sqrt(8.0 * pi);
  P.fourpi_half = std::pow(4.0 * pi, 0.5 * nd);
  P.max_sigma_growth = 1.5;
  P.npts2 = std::pow(nd_n, 2.0);
  P.shape_term = std::pow(P.one_over_nd4 * 5.0, P.minus_one_over_nd6);
  P.sd_c0 = std::pow(2.0, nd - 0.5) * std::sqrt(4.0 * std::atan(1.0));

  const int eb = blocks_of(na, kThreads);      // one thread per bin
  // the initial smoothing is not bounded: its taps may not fit the table
  double *wtab = std::ceil(3.0 * init / b) < (double)stride ? tab : nullptr;
  auto density = [&](const double *val, int check_negative) -> cudaError_t {
    cudaError_t e = cudaMemsetAsync(mmax, 0xff, sizeof(int), s);  // -1
    if (e != cudaSuccess) return e;
    ser_wtap_kernel<<<na, kTapThreads, 0, s>>>(P, B, check_negative, wtaps, mmax, wtab, stride);
    ser_gather_kernel<WTap, true><<<(nb + kWarps - 1) / kWarps, kThreads, 0, s>>>(P, B, wtaps, mmax, val, wtab, stride,
                                                                                  dens);
    ser_dens_finish_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(dens, nb, b);
    return cudaGetLastError();
  };
  ser_init_kernel<<<eb, kThreads, 0, s>>>(B, init);
  SCK(density(B.cnt, 1));
  ser_measures_kernel<<<1, kRed, 0, s>>>(P, B, dens, S);
  SCK(cudaGetLastError());
  SCK(fetch());
  double alm = std::sqrt(h[S_ALMISE] / na);
  double alm_old = alm, cum = alm, cum_old = alm;
  const double rel_err = o->rel_err_convergence;
  int m = 0;
  for (m = 1; m <= o->n_opt_loops; ++m) {
    ser_loop_init_kernel<<<eb, kThreads, 0, s>>>(B, S);
    ser_nest_kernel<<<na, kTapThreads, 0, s>>>(P, B, dens);
    ser_cb_kernel<<<eb, kThreads, 0, s>>>(P, B);
    SCK(cudaMemsetAsync(mmax + 1, 0xff, sizeof(int), s));
    ser_sdtap_kernel<<<na, kTapThreads, 0, s>>>(P, B, sdtaps, mmax + 1, tab, stride);
    ser_gather_kernel<SdTap, false><<<(nb + kWarps - 1) / kWarps, kThreads, 0, s>>>(P, B, sdtaps, mmax + 1, B.cnt,
                                                                                   tab, stride, curv);
    ser_curv_square_kernel<<<blocks_of(nb, kThreads), kThreads, 0, s>>>(curv, nb, b);
    ser_rough_kernel<<<na, kTapThreads, 0, s>>>(P, B, curv);
    ser_rough_reduce_kernel<<<1, kRed, 0, s>>>(B, S);
    ser_optimal_kernel<<<eb, kThreads, 0, s>>>(P, B, S);
    wtab = tab;
    SCK(density(B.cnt, 0));
    ser_measures_kernel<<<1, kRed, 0, s>>>(P, B, dens, S);
    SCK(cudaGetLastError());
    SCK(fetch());
    // maxval(netRoughness) == 0: the reference stops (GridProjectedKDE.F90:5443-5446)
    if (h[S_NETMAX] == 0.0) return MPRW_E_INVAL;
    const double err_dens = std::sqrt(h[S_ERRD] / na), err_smooth = std::sqrt(h[S_ERRS] / na);
    alm = std::sqrt(h[S_ALMISE] / na);
    cum = cum + alm;
    if (!o->skip_error_convergence) {
      if (alm_old > 0.0 && std::fabs(alm - alm_old) / alm_old < rel_err) break;
      if (err_dens < rel_err) break;
      if (err_smooth < rel_err) break;
      if (m > 7 && std::fabs(cum_old / (double)(m - 1) - cum / (double)m) / cum_old / (double)(m - 1) < rel_err)
        break;
    }
    alm_old = alm;
    cum_old = cum;
  }
  res->loops_done = (m > o->n_opt_loops) ? o->n_opt_loops : m;

  // closing weights (GridProjectedKDE.F90:5070-5120) and scalings (:4286-4306)
  if (!wfmt) {
    scale_grid(counts, 1, eff);
    scale_grid(dens, 1, eff);
  } else {
    SCK(density(B.wcnt, 0));
  }
  if (o->compute_raw_density) {
    scale_grid(counts, 0, b);
    if (wfmt) scale_grid(wcounts, 0, b);
  }
  if (o->unit_volume) scale_grid(dens, 1, b);
  SCK(cudaGetLastError());
  SCK(copy_out(dens));
  return MPRW_OK;
}
