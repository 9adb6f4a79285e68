// sort.cu -- radix sorts used around the hot path (CUB, header-only part of
// the CUDA toolkit):
//   * sort_cells: particle processing order by cell, so the warps of the step
//     kernel read neighbouring cell records, heaviest first in buckets of
//     expected passes (cell order within a bucket), so the persistent kernel's
//     queue does not end on a few long particles;
//   * ordered_bin_sums: per-bin sums of non-unit particle weights in particle
//     order, bit-identical to the reference's sequential loop
//     (Histogram.F90:302-325) together with the sequential totals
//     sum(weights) and sum(weights**2) (Histogram.F90:328-340).
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

#include "mprw_kernels.cuh"

namespace mprw {

static cudaError_t ensure(void **buf, size_t *have, size_t need) {
  if (*have >= need) return cudaSuccess;
  if (*buf) cudaFree(*buf);
  *buf = nullptr;
  *have = 0;
  size_t grow = need + need / 4 + 1024;
  cudaError_t e = cudaMalloc(buf, grow);
  if (e == cudaSuccess) *have = grow;
  return e;
}

__global__ void iota_keys_kernel(const int32_t *cell, uint32_t *keys, uint32_t *vals, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    keys[i] = (uint32_t)cell[i];
    vals[i] = (uint32_t)i;
  }
}

// keys (top - bucket of the expected passes, cell); per_pass: counter blocks per
// pass
__global__ void lpt_keys_kernel(const int32_t *cell, const uint64_t *ctr, const uint64_t *ctr_prev, uint32_t per_pass,
                                PassGuess g, uint32_t top, float per_bucket, int ncell_bits, uint32_t *keys,
                                uint32_t *vals, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t d = ctr_prev && ctr[i] >= ctr_prev[i] ? ctr[i] - ctr_prev[i] : 0;
    float passes = (float)d / (float)per_pass;
    if (d == 0) {
      const float dt = (float)*reinterpret_cast<const double *>(g.dtcell + (size_t)cell[i] * g.stride);
      passes = fmaxf((float)(g.t_end - fmax(g.t[i], g.t_begin)), 0.0f) / dt;
    }
    const float b = passes * per_bucket;
    const uint32_t bucket = b < (float)top ? (uint32_t)b : top;  // (a time step of zero or NaN: the top)
    keys[i] = ((top - bucket) << ncell_bits) | (uint32_t)cell[i];
    vals[i] = (uint32_t)i;
  }
}

static int grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  return b < 1 ? 1 : (int)b;
}

cudaError_t sort_cells(const int32_t *cell, const uint64_t *ctr, const uint64_t *ctr_prev, uint64_t ctr_per_pass,
                       const PassGuess &guess, uint32_t *perm, int64_t n, int ncell_bits, void **scratch, size_t *scratch_bytes,
                       cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int bucket_bits = std::min(kPassBucketBits, 32 - ncell_bits);
  const bool lpt = ctr && ctr_per_pass > 0 && bucket_bits >= kMinBucketBits;
  const int bits = lpt ? ncell_bits + bucket_bits : ncell_bits;
  size_t temp = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, temp, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                                  (const uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0,
                                                  bits, s);
  if (e != cudaSuccess) return e;
  size_t arr = ((size_t)n * 4 + 255) / 256 * 256;
  e = ensure(scratch, scratch_bytes, 3 * arr + temp);
  if (e != cudaSuccess) return e;
  char *b = (char *)*scratch;
  uint32_t *kin = (uint32_t *)b, *kout = (uint32_t *)(b + arr), *vin = (uint32_t *)(b + 2 * arr);
  void *tmp = b + 3 * arr;
  if (lpt)
    lpt_keys_kernel<<<grid_for(n), 256, 0, s>>>(cell, ctr, ctr_prev, (uint32_t)ctr_per_pass, guess,
                                                (1u << bucket_bits) - 1, bucket_bits == kPassBucketBits ? 0.25f : 0.125f,
                                                ncell_bits, kin, vin, n);
  else
    iota_keys_kernel<<<grid_for(n), 256, 0, s>>>(cell, kin, vin, n);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cub::DeviceRadixSort::SortPairs(tmp, temp, kin, kout, vin, perm, (int)n, 0, bits, s);
}

// ---- sequential sums in parallel ------------------------------------------------
// The reference adds weights one after another, each addition rounded; the
// results here are those sums to the bit.  While a running sum s >= 0 stays in
// one binade it is a multiple S of that binade's unit u, and adding w >= 0
// moves S by w/u rounded to nearest: by q or q + 1, and where w lies midway
// between two multiples (a tie), to the even one, which depends only on the
// parity of S + q.  So an element is a pair (move from an even S, move from an
// odd S), pairs compose associatively, and a block scans a tile of them at
// once.  The tile's first element that would take the sum out of its binade
// (or that is negative, infinite or NaN) ends the scan; the thread that holds
// it adds its elements in FP64 and the tile restarts behind them, with the new
// binade.  A sum of n similar weights crosses log2(n) binades.
// (250,000 weights: one thread's chain 24.5 ms; each of the four kernels
// below under 0.05 ms.)
struct Moves {
  unsigned long long d0, d1;
};
constexpr unsigned long long kLeave = 1ull << 60;   // beyond any binade
constexpr unsigned long long kBinade = 1ull << 53;  // S of the binade's end

__device__ __forceinline__ Moves compose(Moves a, Moves b) {
  Moves r;
  r.d0 = a.d0 + ((a.d0 & 1ull) ? b.d1 : b.d0);
  r.d1 = a.d1 + ((a.d1 & 1ull) ? b.d0 : b.d1);
  r.d0 = r.d0 < kLeave ? r.d0 : kLeave;
  r.d1 = r.d1 < kLeave ? r.d1 : kLeave;
  return r;
}

// the moves of adding w to a sum of biased exponent e (1..2046)
__device__ __forceinline__ Moves moves_of(double w, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(w);
  if ((b << 1) == 0ull) return {0ull, 0ull};
  int ew = (int)(b >> 52);  // sign and exponent: a negative w has ew > 2047
  if (ew >= 2047) return {kLeave, kLeave};
  const unsigned long long m = (b & 0x000FFFFFFFFFFFFFull) | (ew ? 0x0010000000000000ull : 0ull);
  ew = ew ? ew : 1;
  const int sh = e - ew;
  if (sh < 0) return {kLeave, kLeave};
  if (sh > 53) return {0ull, 0ull};
  const unsigned long long q = m >> sh, rem = m & ((1ull << sh) - 1ull), half = (1ull << sh) >> 1;
  if (sh == 0 || rem < half) return {q, q};
  if (rem > half) return {q + 1ull, q + 1ull};
  return {q + (q & 1ull), q + ((q + 1ull) & 1ull)};
}

__device__ __forceinline__ Moves shfl_up(Moves a, int o) {
  return {__shfl_up_sync(0xffffffffu, a.d0, o), __shfl_up_sync(0xffffffffu, a.d1, o)};
}

// The particles are cut into chunks.  Each chunk's plain sum, prefix-summed,
// predicts the binade its running sum starts in; every chunk then composes its
// moves for that binade at once, and one block folds the chunks in order, 32
// at a time.  A chunk whose prediction fails or whose sum leaves the binade is
// run through the block's own scan.  Two sums side by side: the weights of the
// active particles and their (rounded) squares.
constexpr int kTotThreads = 256, kTotPer = 8, kChunk = kTotThreads * kTotPer, kTotWarps = kTotThreads / 32;

struct TotArgs {
  const double *mass;
  const int32_t *status;
  int64_t n, nchunk;
  double *approx;  // 2 x nchunk
  int *expo;       // 2 x nchunk: predicted biased exponent before the chunk
  Moves *moves;    // 2 x nchunk
  double *out;     // 2
};

__device__ __forceinline__ double tot_value(const TotArgs &a, int64_t i, bool square) {
  if (i >= a.n || a.status[i] != ST_ACTIVE) return 0.0;
  const double w = a.mass[i];
  return square ? __dmul_rn(w, w) : w;
}

__global__ void __launch_bounds__(kTotThreads) tot_approx_kernel(TotArgs a) {
  __shared__ double red[2][kTotWarps];
  const int64_t base = (int64_t)blockIdx.x * kChunk;
  double w = 0.0, w2 = 0.0;
#pragma unroll
  for (int k = 0; k < kTotPer; ++k) {
    const double v = tot_value(a, base + k * kTotThreads + threadIdx.x, false);
    w += v;
    w2 += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    w += __shfl_down_sync(0xffffffffu, w, o);
    w2 += __shfl_down_sync(0xffffffffu, w2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = w;
    red[1][threadIdx.x >> 5] = w2;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int k = 0; k < kTotWarps; ++k) t += red[threadIdx.x][k];
    a.approx[threadIdx.x * a.nchunk + blockIdx.x] = t;
  }
}

// the exponent of the prefix sum before every chunk, one block per sum
__global__ void __launch_bounds__(1024) tot_predict_kernel(TotArgs a) {
  __shared__ double part[1024];
  const double *x = a.approx + blockIdx.x * a.nchunk;
  int *expo = a.expo + blockIdx.x * a.nchunk;
  const int64_t per = (a.nchunk + 1023) / 1024, i0 = threadIdx.x * per;
  const int64_t i1 = i0 + per < a.nchunk ? i0 + per : a.nchunk;
  double own = 0.0;
  for (int64_t i = i0; i < i1; ++i) own += x[i];
  part[threadIdx.x] = own;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const double v = threadIdx.x >= o ? part[threadIdx.x - o] : 0.0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  double run = threadIdx.x ? part[threadIdx.x - 1] : 0.0;
  for (int64_t i = i0; i < i1; ++i) {
    expo[i] = (int)((unsigned long long)__double_as_longlong(run) >> 52);
    run += x[i];
  }
}

__device__ __forceinline__ Moves warp_scan(Moves m, int lane) {
  for (int o = 1; o < 32; o <<= 1) {
    const Moves up = shfl_up(m, o);
    if (lane >= o) m = compose(up, m);
  }
  return m;
}

// this thread's kTotPer consecutive elements from base on (zero from end on)
__device__ __forceinline__ void tot_load(const TotArgs &a, int64_t base, int64_t end, bool square,
                                         double (&v)[kTotPer]) {
#pragma unroll
  for (int k = 0; k < kTotPer; ++k) {
    const int64_t i = base + (int64_t)threadIdx.x * kTotPer + k;
    v[k] = i < end ? tot_value(a, i, square) : 0.0;
  }
}

__device__ __forceinline__ Moves own_moves(const double (&v)[kTotPer], int e) {
  Moves m = moves_of(v[0], e);
#pragma unroll
  for (int k = 1; k < kTotPer; ++k) m = compose(m, moves_of(v[k], e));
  return m;
}

__global__ void __launch_bounds__(kTotThreads) tot_moves_kernel(TotArgs a) {
  __shared__ Moves wtot[kTotWarps];
  const bool square = blockIdx.y == 1;
  const int64_t c = blockIdx.x;
  const int e = a.expo[blockIdx.y * a.nchunk + c];
  const int lane = threadIdx.x & 31;
  Moves r = {kLeave, kLeave};
  if (e >= 1 && e < 2047) {
    double v[kTotPer];
    tot_load(a, c * kChunk, a.n, square, v);
    const Moves inc = warp_scan(own_moves(v, e), lane);
    if (lane == 31) wtot[threadIdx.x >> 5] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
      r = wtot[0];
      for (int k = 1; k < kTotWarps; ++k) r = compose(r, wtot[k]);
    }
  }
  if (threadIdx.x == 0) a.moves[blockIdx.y * a.nchunk + c] = r;
}

__device__ __forceinline__ double from_units(int e, unsigned long long S) {
  return __longlong_as_double((long long)(((unsigned long long)e << 52) + (S - 0x0010000000000000ull)));
}

// one block per sum: the chunks in order
__global__ void __launch_bounds__(kTotThreads) tot_fold_kernel(TotArgs a) {
  __shared__ double sum;
  __shared__ Moves wtot[kTotWarps];
  __shared__ int first, done;
  __shared__ int64_t chunk;
  const bool square = blockIdx.x == 1;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int *expo = a.expo + blockIdx.x * a.nchunk;
  const Moves *moves = a.moves + blockIdx.x * a.nchunk;
  if (t == 0) {
    sum = 0.0;
    done = 0;
  }
  __syncthreads();
  for (int64_t c = 0; c < a.nchunk && !done;) {
    // as many of the next 32 chunks as stay in the present binade
    if (wid == 0) {
      const unsigned long long bs = (unsigned long long)__double_as_longlong(sum);
      const int e = (int)(bs >> 52);
      const unsigned long long S = (bs & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
      Moves m = {0ull, 0ull};
      if (c + lane < a.nchunk) m = (expo[c + lane] == e) ? moves[c + lane] : Moves{kLeave, kLeave};
      m = warp_scan(m, lane);
      const unsigned long long after = S + ((S & 1ull) ? m.d1 : m.d0);
      const unsigned out = __ballot_sync(0xffffffffu, after >= kBinade);
      const int f = out ? __ffs(out) - 1 : 32;
      if (lane == f - 1 && e >= 1 && e < 2047) sum = from_units(e, after);
      if (lane == 0) {
        chunk = c + f;
        first = f;
      }
    }
    __syncthreads();
    c = chunk;
    const bool hard = first < 32 && c < a.nchunk;
    __syncthreads();
    if (!hard) continue;
    // the chunk that does not: scanned here, piece by piece
    const int64_t end = (c + 1) * kChunk < a.n ? (c + 1) * kChunk : a.n;
    for (int64_t base = c * kChunk; base < end;) {
      double cur[kTotPer];
      tot_load(a, base, end, square, cur);
      if (t == 0) first = kTotThreads;
      __syncthreads();
      const double s = sum;
      const unsigned long long bs = (unsigned long long)__double_as_longlong(s);
      const int e = (int)(bs >> 52);
      const bool scan = e >= 1 && e < 2047;  // else the sum is zero, subnormal, negative, infinite or NaN
      const unsigned long long S = (bs & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
      unsigned long long before = S, after = S;  // S before and after this thread's elements
      bool stop = false;
      if (scan) {
        Moves inc = warp_scan(own_moves(cur, e), lane);
        if (lane == 31) wtot[wid] = inc;
        __syncthreads();
        Moves pre = {0ull, 0ull};
        for (int k = 0; k < wid; ++k) pre = compose(pre, wtot[k]);
        Moves exc = shfl_up(inc, 1);
        exc = lane ? compose(pre, exc) : pre;
        inc = compose(pre, inc);
        before = S + ((S & 1ull) ? exc.d1 : exc.d0);
        after = S + ((S & 1ull) ? inc.d1 : inc.d0);
        stop = after >= kBinade;
      } else {
#pragma unroll
        for (int k = 0; k < kTotPer; ++k) stop = stop || cur[k] != 0.0 || cur[k] != cur[k];
      }
      if (stop) atomicMin(&first, t);
      __syncthreads();
      const int f = first;
      if (f == kTotThreads) {
        // the rest of the chunk stays in the binade (or adds only zeros)
        if (scan && t == kTotThreads - 1) sum = from_units(e, after);
        base += kChunk;
      } else {
        if (t == f) {
          double x = scan ? from_units(e, before) : s;
          bool odd = false;  // a negative or non-finite term: the rest one by one
#pragma unroll
          for (int k = 0; k < kTotPer; ++k) {
            odd = odd || !(cur[k] >= 0.0 && cur[k] <= 1.7976931348623157e308);
            x = x + cur[k];
          }
          if (odd || !(x <= 1.7976931348623157e308)) {
            for (int64_t i = base + (int64_t)(f + 1) * kTotPer; i < a.n; ++i) x = x + tot_value(a, i, square);
            done = 1;
          }
          sum = x;
        }
        base += (int64_t)(f + 1) * kTotPer;
      }
      __syncthreads();
      if (done) break;
    }
    ++c;
  }
  if (t == 0) a.out[blockIdx.x] = sum;
}

// Per-bin sums in particle order over the particles sorted by bin (a stable
// sort keeps their order): the head of each bin's run adds its first kHeadRun
// weights, longer runs go to the whole warp, which loads 32 weights at a time
// and adds them in order.
constexpr int kHeadRun = 16;
__global__ void __launch_bounds__(256) segment_sum_kernel(const uint32_t *keys, const uint32_t *idx, int64_t n,
                                                          uint32_t nbins, const double *mass, double *counts) {
  const int lane = threadIdx.x & 31;
  for (int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; w0 < n;
       w0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = w0 + lane;
    const uint32_t k = i < n ? keys[i] : nbins;
    const bool head = k < nbins && (i == 0 || keys[i - 1] != k);
    double acc = 0.0;
    bool more = false;
    if (head) {
      int64_t j = i;
      for (; j < n && j < i + kHeadRun && keys[j] == k; ++j) acc = acc + mass[idx[j]];
      more = j < n && j == i + kHeadRun && keys[j] == k;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, more); m; m &= m - 1) {
      const int o = __ffs(m) - 1;
      const uint32_t ko = __shfl_sync(0xffffffffu, k, o);
      double a = __shfl_sync(0xffffffffu, acc, o);
      for (int64_t j0 = w0 + o + kHeadRun;; j0 += 32) {
        const int64_t j = j0 + lane;
        const bool in = j < n && keys[j] == ko;
        const double v = in ? mass[idx[j]] : 0.0;
        const int c = __popc(__ballot_sync(0xffffffffu, in));
        for (int l = 0; l < c; ++l) a = a + __shfl_sync(0xffffffffu, v, l);
        if (c < 32) break;
      }
      if (lane == o) acc = a;
    }
    if (head) counts[k] = acc;
  }
}

__global__ void iota_kernel(uint32_t *vals, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    vals[i] = (uint32_t)i;
}

cudaError_t ordered_bin_sums(HistArgs a, const double *mass, int64_t nbins, double *counts, double *total_mass,
                             double *sum_w2, void **scratch, size_t *scratch_bytes, cudaStream_t s) {
  // bins as 32-bit keys (nbins: no bin), sorted on the bits they have
  const int64_t n = a.n;
  int bits = 1;
  while (bits < 32 && ((int64_t)1 << bits) <= nbins) ++bits;
  size_t temp = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, temp, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                                  (const uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0, bits, s);
  if (e != cudaSuccess) return e;
  const size_t arr = ((size_t)n * 4 + 255) / 256 * 256;
  const int64_t nchunk = std::max<int64_t>(1, (n + kChunk - 1) / kChunk);
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t o_tot = 4 * arr, o_appr = o_tot + 256, o_expo = o_appr + up(16 * (size_t)nchunk);
  const size_t o_mov = o_expo + up(8 * (size_t)nchunk), o_tmp = o_mov + up(2 * sizeof(Moves) * (size_t)nchunk);
  e = ensure(scratch, scratch_bytes, o_tmp + temp);
  if (e != cudaSuccess) return e;
  char *b = (char *)*scratch;
  uint32_t *kin = (uint32_t *)b, *kout = (uint32_t *)(b + arr);
  uint32_t *vin = (uint32_t *)(b + 2 * arr), *vout = (uint32_t *)(b + 3 * arr);
  double *tot = (double *)(b + o_tot);
  void *tmp = b + o_tmp;
  e = cudaMemsetAsync(counts, 0, sizeof(double) * (size_t)nbins, s);
  if (e != cudaSuccess) return e;
  if (n > 0) {
    a.bin_of = kin;
    e = launch_hist_bins(a, s);
    if (e != cudaSuccess) return e;
    iota_kernel<<<grid_for(n), 256, 0, s>>>(vin, n);
    e = cub::DeviceRadixSort::SortPairs(tmp, temp, kin, kout, vin, vout, (int)n, 0, bits, s);
    if (e != cudaSuccess) return e;
    segment_sum_kernel<<<grid_for(n), 256, 0, s>>>(kout, vout, n, (uint32_t)nbins, mass, counts);
  }
  const TotArgs t{mass, a.status, n, nchunk, (double *)(b + o_appr), (int *)(b + o_expo), (Moves *)(b + o_mov), tot};
  tot_approx_kernel<<<(unsigned)nchunk, kTotThreads, 0, s>>>(t);
  tot_predict_kernel<<<2, 1024, 0, s>>>(t);
  tot_moves_kernel<<<dim3((unsigned)nchunk, 2), kTotThreads, 0, s>>>(t);
  tot_fold_kernel<<<2, kTotThreads, 0, s>>>(t);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  double h[2] = {0.0, 0.0};
  e = cudaMemcpyAsync(h, tot, sizeof h, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *total_mass = h[0];
  *sum_w2 = h[1];
  return e;
}

}  // namespace mprw
