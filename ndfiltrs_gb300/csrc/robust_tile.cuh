// Fast path of the robust statistics for float32 windows of up to 128 samples:
// the MAD, sigma clipping and the mode estimators (device code; robust_tile.cu
// and robust_tile_wide.cu instantiate it so that the two compile in parallel).
//
// The reference computes these per window in float64 (src/robust.rs:376-689,
// src/location.rs:36-84). The general kernel (robust.cuh) restates that
// operation for operation and is bound by the FP64 pipe (two lanes per clock
// and SM on this GPU) and by its thread-local sample arrays. Almost none of
// that arithmetic reaches the result:
//  * the MAD is |2 v - (a + b)| / 2 for one sample v (two for even counts):
//    which sample follows from float32 differences, because rounding is
//    monotone; where the differences are exact they are the answer, else the
//    few rounding ties are settled by exact differences;
//  * a clipping pass only decides which sorted samples stay. The spread is
//    evaluated in float32 with a bound on its error; a sample so close to the
//    limit that the bound does not decide it sends the pass to float64 with a
//    bound of its own;
//  * the mean of the kept samples is the exact sum, rounded once, divided once;
//    samples are integer multiples of the tile's lowest set bit, so their
//    deviations from the median add up in integers.
// The few float64 operations that remain per output are the reference's own,
// on the same operands, so the results are the same bits. A window that none
// of the bounds decides (an infinity in the middle, magnitudes that mix
// beyond the float64 significand, a sample on the limit to 2^-42) is stored as
// a NaN with the payload kUndecided, which no filter output can hold, and the
// general kernel fills those in afterwards. No state is kept beside the
// output, so runs of one plan on several streams stay independent.
//
// One thread per output: its taps' keys go through a register sorting network
// of the window's width; the sorted samples lie in a shared-memory column of
// the thread, where the runs that clipping leaves are indexed at run time.
// 128 threads take a tile of 512 outputs so that the halo is staged once for
// four outputs per thread.
//
// Bound now by the min / max pipe of the sort and by the shared-memory loads
// of the passes over the column. Measured with the filling-in pass (frames of
// noise with outliers, NaN and infinities): MAD 5 x 5 on 4096^2 7.63 -> 0.71 ms
// (0.91 with a few float64 operations per output, which cost a third of a 3 x 3
// MAD), clipped mode 7 x 7 on 2048^2 30.7 -> 0.80 ms.
#pragma once

#include "network.cuh"
#include "robust.cuh"

namespace ndf {

namespace robust_tile {

constexpr int kT = 128;
// Shared memory of a block: two blocks fit an SM at the widest windows.
constexpr size_t kRobustTileSmem = 112 * 1024;

// Exponent of the lowest set bit of the finite nonzero float behind `key`
// (x = odd * 2^result); INT_MAX for zero and the sentinel.
__device__ __forceinline__ int lowest_bit(uint32_t key) {
  if (key == KeyOf<float>::kSentinel) return INT_MAX;
  const unsigned int b = __float_as_uint(KeyOf<float>::value(key));
  const int e = (int)((b >> 23) & 0xFFu);
  const unsigned int m = (b & 0x7FFFFFu) | (e ? 0x800000u : 0u);
  if (m == 0 || e == 255) return INT_MAX;
  return (e ? e : 1) - 150 + __ffs((int)m) - 1;
}

// Whether a + b, and so the midpoint, is exact in float64: equal values, or
// zero or normal values whose exponents are at most 28 apart.
__device__ __forceinline__ bool sum_exact(float a, float b) {
  const unsigned int ba = __float_as_uint(a), bb = __float_as_uint(b);
  const int ea = (int)((ba >> 23) & 0xFF), eb = (int)((bb >> 23) & 0xFF);
  if (ba == bb) return ea != 255;
  const bool za = (ba << 1) == 0u, zb = (bb << 1) == 0u;
  const bool na = ea >= 30 && ea <= 253, nb = eb >= 30 && eb <= 253;
  const int diff = ea > eb ? ea - eb : eb - ea;
  return (za || na) && (zb || nb) && (za || zb || diff <= 28);
}

// The rounding error of x - y (exact difference minus `d` = RN(x - y)).
__device__ __forceinline__ float difference_error(float x, float y, float d) {
  const float yy = __fsub_rn(x, d);
  return __fadd_rn(__fsub_rn(x, __fadd_rn(d, yy)), __fsub_rn(yy, y));
}

// A thread's sorted samples: a column of shared memory.
struct Column {
  const float* c;
  __device__ __forceinline__ float operator[](int i) const { return c[i * kT]; }
};

// The sample at the `rank`-th (0-based) smallest deviation from the middle of
// the n sorted samples s, as an index, from float32 differences. The rank + 1
// smallest deviations belong to consecutive samples i..i + rank, and the
// largest of them is max(a - s[i], s[i + rank] - b) up to the half gap
// (b - a) / 2 that every deviation shares (a, b the middle samples), so the
// wanted one is the least of those maxima. `*value` gets it. Equal rounded
// maxima are compared by their exact values. -1: not decided (overflow).
__device__ __forceinline__ int deviation_at(const Column& s, int n, int rank, float a, float b, float* value) {
  float best = __int_as_float(0x7f800000);
  int at = -1;
  bool tie = false;
  for (int i = 0; i + rank < n; ++i) {
    const float l = __fsub_rn(a, s[i]), r = __fsub_rn(s[i + rank], b);
    const float m = fmaxf(l, r);
    tie = m < best ? l == r : (tie || m == best);
    if (m < best) {
      best = m;
      at = l >= r ? i : i + rank;
    }
  }
  *value = best;
  if (at < 0 || !tie) return at;
  float low = 0.0f;
  at = -1;
  for (int i = 0; i + rank < n; ++i) {
    const float l = __fsub_rn(a, s[i]), r = __fsub_rn(s[i + rank], b);
    if (fmaxf(l, r) != best) continue;
    const float el = difference_error(a, s[i], l), er = difference_error(s[i + rank], b, r);
    const bool left = l > r || (l == r && el >= er);
    const float e = left ? el : er;
    if (at < 0 || e < low) {
      low = e;
      at = left ? i : i + rank;
    }
  }
  return at;
}

// The MAD of the n sorted samples times `scale`, rounded to float32; kUndecided
// when not decided. (Samples of any set bits; out of line, as mad_value takes
// nearly every window.)
static __device__ __noinline__ float mad_general(const float* c, int n, double scale) {
  const Column s{c};
  const float undecided = __uint_as_float(kUndecided);
  const float a = s[(n - 1) / 2], b = s[n / 2];
  if (!sum_exact(a, b)) return undecided;
  float value;
  const int at = deviation_at(s, n, n / 2, a, b, &value);
  if (at < 0) return undecided;
  const double center = __dadd_rn(widen(a), widen(b));
  Scaled d{abs64(__dsub_rn(twice(widen(s[at])), center)), -1};
  if ((n & 1) == 0) {
    const int before = deviation_at(s, n, n / 2 - 1, a, b, &value);
    if (before < 0) return undecided;
    // scaled_midpoint of two deviations of exponent -1: their float64 sum.
    d = {__dadd_rn(abs64(__dsub_rn(twice(widen(s[before])), center)), d.value), -2};
  }
  const double product = multiply_scaled(d, scale);
  return nan64(product) ? nan_of(0.0f) : __double2float_rn(product);
}

// The same for samples that are multiples of 2^low. Differences below 2^24 of
// those units are exact in float32, so the least maxima are the deviations
// themselves and ties are equal deviations; their product with the scale (a pair
// of floats, to 2^-49; zero where a pair does not hold the scale so well) is the
// float32 rounding of the float64 one when it rounds the same 2^-40 above and below.
__device__ __forceinline__ float mad_value(const Column& s, int n, int low, float2 scale, double scale64) {
  const int h = n / 2;
  const bool even = (n & 1) == 0;
  const float a = s[(n - 1) / 2], b = s[h];
  float mid = __int_as_float(0x7f800000), before = mid, r0 = __fsub_rn(s[max(h - 1, 0)], b);
#pragma unroll 4
  for (int i = 0; i < n - h; ++i) {
    const float l = __fsub_rn(a, s[i]), r = __fsub_rn(s[i + h], b);
    mid = fminf(mid, fmaxf(l, r));
    before = fminf(before, fmaxf(l, r0));
    r0 = r;
  }
  float d = mid;
  if (even) {
    before = fminf(before, fmaxf(__fsub_rn(a, s[h]), r0));
    // Both deviations lack half the gap b - a; their mean is half of all three.
    d = __fadd_rn(__fadd_rn(mid, before), __fsub_rn(b, a));
  }
  // 2^(low + 23) as a float; nothing is below it when that is out of range.
  const float limit = low >= -140 && low <= 100 ? __uint_as_float((unsigned int)(low + 150) << 23) : 0.0f;
  if (d < limit) {
    if (even) d = __fmul_rn(d, 0.5f);
    const float p = __fmul_rn(d, scale.x);
    const float e = __fmaf_rn(d, scale.y, __fmaf_rn(d, scale.x, -p)), off = p * 9.094947e-13f;
    const float value = __fadd_rn(p, __fadd_rn(e, off));
    if (d == 0.0f) return 0.0f;
    if (value == __fadd_rn(p, __fsub_rn(e, off)) && p >= 1e-25f && p <= 1e37f) return value;
  }
  return mad_general(s.c, n, scale64);
}

__device__ __forceinline__ float difference(float x, float y, float) { return __fsub_rn(x, y); }
__device__ __forceinline__ double difference(float x, float y, double) { return __dsub_rn(widen(x), widen(y)); }

// Sums of the deviations from `a` and of their squares over s[lo, hi), in F
// (float or double), and the population standard deviation from them. With
// `a` a median of the run, |mean - a| is at most one standard deviation, so
// the subtraction costs at most a factor of three: the relative error of the
// result is below (3 n + 16) u for terms within the range of F.
template <typename F>
struct Moments {
  F mean;  // minus a
  F std;
};

template <typename F>
__device__ __forceinline__ Moments<F> moments_of(const Column& s, int lo, int hi, float a) {
  F s1 = 0, s2 = 0;
#pragma unroll 4
  for (int j = lo; j < hi; ++j) {
    const F d = difference(s[j], a, F());
    s1 += d;
    s2 += d * d;
  }
  const F n = (F)(hi - lo);
  const F mean = s1 / n;
  const F var = s2 / n - mean * mean;
  if constexpr (sizeof(F) == 4)
    return {mean, sqrtf(fmaxf(var, 0.0f))};
  else
    return {mean, sqrt(fmax(var, 0.0))};
}

__device__ __forceinline__ float unit_roundoff(float) { return 5.9604645e-8f; }
__device__ __forceinline__ double unit_roundoff(double) { return 1.1102230246251565e-16; }

// Bound on the relative error of a limit computed in F for n samples and
// multipliers of at least 1/2: (3 n + 30) u covers the spread, the half gap
// and the distance; float64 adds the reference's own roundings, below 2^-44.
__device__ __forceinline__ float limit_error(int n, float) { return (float)(8 * n + 64) * 5.9604645e-8f; }
__device__ __forceinline__ double limit_error(int, double) { return 2.2737367544323206e-13; }

// The MAD of s[lo, hi) as a spread, in F (relative error a few u).
template <typename F>
__device__ __forceinline__ F mad_spread(const Column& s, int lo, int hi, float a, float b) {
  const int n = hi - lo, h = n / 2;
  F m1 = (F)__int_as_float(0x7f800000), m0 = m1;
  F before = difference(s[lo + max(h - 1, 0)], b, F());
  for (int i = 0; i < n - h; ++i) {
    const F l = difference(a, s[lo + i], F()), r = difference(s[lo + i + h], b, F());
    m0 = min(m0, max(l, before));
    m1 = min(m1, max(l, r));
    before = r;
  }
  if (n & 1) return m1;
  // The last run of h samples: [h, n).
  m0 = min(m0, max(difference(a, s[lo + h], F()), before));
  return (F)0.5 * (m0 + m1) + (F)0.5 * difference(b, a, F());
}

// One clipping pass over s[lo, hi): the run that stays. 1: done, 0: some
// sample lies too close to its limit to be decided in F.
template <typename F>
__device__ __forceinline__ int clip_pass(const Column& s, int lo, int hi, const RobustArgs& ra, int* new_lo,
                                         int* new_hi, float* std) {
  const int n = hi - lo;
  const float a = s[lo + (n - 1) / 2], b = s[lo + n / 2];
  F center = (F)0.5 * difference(b, a, F()), spread = 0;  // center minus a
  // The reference rounds a mean center to float64; the mean of n terms in F
  // is off by at most n u of the mean magnitude, which 1.5 std bounds.
  F slack = (F)fabsf(a) * (F)4.440892098500626e-16;
  if (ra.spread == 0 || ra.center == 0) {
    const Moments<F> m = moments_of<F>(s, lo, hi, a);
    spread = m.std;
    *std = (float)m.std;
    if (ra.center == 0) {
      center = m.mean;
      slack += (F)(4 * n) * unit_roundoff(F()) * m.std;
    }
  }
  int x = lo, y = hi;
  if (ra.spread == 1) {
    const F mad = mad_spread<F>(s, lo, hi, a, b);
    // Zero spread: only samples equal to the center stay. About a mean the test below
    // decides it where no sample is so close to the mean that it might equal it (data of
    // few values, most of them alike).
    if (mad == (F)0 && ra.center != 0) {
      while (x < hi && s[x] != a) ++x;
      while (y > x && s[y - 1] != a) --y;
      *new_lo = x;
      *new_hi = y;
      return 1;
    }
    spread = mad * (F)1.4826022185056018;
  }
  const F lower = (F)ra.lower * spread, upper = (F)ra.upper * spread;
  const F e = limit_error(n, F());
  const F lower_in = lower * ((F)1 - e) - slack, lower_out = lower * ((F)1 + e) + slack;
  const F upper_in = upper * ((F)1 - e) - slack, upper_out = upper * ((F)1 + e) + slack;
  bool sure = true;
  while (x < hi) {
    const F distance = center - difference(s[x], a, F());
    if (distance <= lower_in) break;
    sure = sure && distance >= lower_out;
    ++x;
  }
  while (y > x) {
    const F distance = difference(s[y - 1], a, F()) - center;
    if (distance <= upper_in) break;
    sure = sure && distance >= upper_out;
    --y;
  }
  *new_lo = x;
  *new_hi = y;
  return sure ? 1 : 0;
}

// Rare: kept out of line.
static __device__ __noinline__ int clip_pass_f64(const float* c, int lo, int hi, const RobustArgs& ra, int* new_lo,
                                                 int* new_hi, float* std) {
  return clip_pass<double>(Column{c}, lo, hi, ra, new_lo, new_hi, std);
}

// Whether the differences of the finite run s[lo, hi) stay clear of float32
// underflow and overflow in the squares.
__device__ __forceinline__ bool in_range(const Column& s, int lo, int hi) {
  const float span = __fsub_rn(s[hi - 1], s[lo]);
  return span >= 8.8817842e-16f && span <= 1.1529215e18f;
}

// finite_mean (src/robust.rs:572-592) of s[lo, hi): the exact sum rounded
// once (the sequential Neumaier sum of samples that are multiples of 2^low
// and below 2^H equals it when low >= 2 k + H - 105, n < 2^k; see ExactSum)
// over n. Samples are multiples of 2^low: deviations from `a` below 2^23 of
// those units are exact float32 differences and add up as integers; else
// float64 adds, exact while H + k - low is at most 53.
__device__ __forceinline__ bool exact_mean_of(const Column& s, int lo, int hi, int low, double* mean) {
  const int n = hi - lo;
  const float first = s[lo], last = s[hi - 1];
  if (first == last) {
    *mean = __dadd_rn(widen(first), 0.0);
    return true;
  }
  const float top = fmaxf(fabsf(first), fabsf(last));
  const int H = max((int)((__float_as_uint(top) >> 23) & 0xFF), 1) - 126;
  const int k = 32 - __clz(n);
  if (low < 2 * k + H - 105) return false;
  const float a = s[lo + (n - 1) / 2];
  double total;
  const float dm = fmaxf(__fsub_rn(a, first), __fsub_rn(last, a));
  const bool scaled = low >= -120 && low <= 100;
  const float unit = scaled ? __int_as_float((127 - low) << 23) : 0.0f;  // 2^-low
  if (scaled && dm * unit < 8388608.0f) {
    int sum = 0;
#pragma unroll 4
    for (int j = lo; j < hi; ++j) sum += __float2int_rn(__fmul_rn(__fsub_rn(s[j], a), unit));
    // n a exactly plus the integers' 2^low, rounded once.
    const double q = __longlong_as_double((long long)(1023 + low) << 52);
    total = __fma_rn((double)n, widen(a), __dmul_rn((double)sum, q));
  } else {
    if (H + k - low > 53) return false;
    total = 0.0;
    for (int j = lo; j < hi; ++j) total = __dadd_rn(total, widen(s[j]));
  }
  *mean = __ddiv_rn(total, (double)n);
  return true;
}

// |difference| / std >= 0.3 for the standard deviation of n samples: 1 or 0,
// -1 when F does not decide.
template <typename F>
__device__ __forceinline__ int far_from_mean(int n, F std, double difference) {
  const F d = (F)abs64(difference), limit = (F)0.3 * std, e = limit_error(n, F());
  if (d >= limit * ((F)1 + e)) return 1;
  if (d <= limit * ((F)1 - e)) return 0;
  return -1;
}

static __device__ __noinline__ int far_from_mean_f64(const float* c, int lo, int hi, double difference) {
  const Column s{c};
  return far_from_mean<double>(hi - lo, moments_of<double>(s, lo, hi, s[lo + (hi - lo - 1) / 2]).std, difference);
}

// mode_estimate (src/location.rs:36-54) of the sorted run; `std` is its standard
// deviation in float32 where the last clipping pass has it already, else negative.
__device__ __forceinline__ bool mode_value(const Column& s, int lo, int hi, int low, const RobustArgs& ra, float std,
                                           double* out) {
  const int n = hi - lo;
  double mean;
  if (!exact_mean_of(s, lo, hi, low, &mean)) return false;
  const float a = s[lo + (n - 1) / 2], b = s[lo + n / 2];
  if (!sum_exact(a, b)) return false;
  const double median =
      __float_as_uint(a) == __float_as_uint(b) ? widen(a) : __dmul_rn(__dadd_rn(widen(a), widen(b)), 0.5);
  if (ra.estimator != kModeSex) {
    *out = mode_from_moments(mean, median, 0.0, ra.estimator, ra.pearson);
    return true;
  }
  if (s[lo] == s[hi - 1]) {
    *out = mean;
    return true;
  }
  if (!in_range(s, lo, hi)) return false;
  const double off = __dsub_rn(median, mean);
  if (std < 0.0f) std = moments_of<float>(s, lo, hi, a).std;
  int far = far_from_mean<float>(n, std, off);
  if (far < 0) far = far_from_mean_f64(s.c, lo, hi, off);
  if (far < 0) return false;
  *out = far ? median : __dadd_rn(median, __dmul_rn(__dsub_rn(ra.pearson, 1.0), off));
  return true;
}

// clipped (src/robust.rs:632-689) of the n sorted finite samples.
__device__ __forceinline__ bool clipped_value(const Column& s, int n, int low, const RobustArgs& ra, double* out) {
  int lo = 0, hi = n;
  long long iteration = 0;
  float std = -1.0f;
  while (hi - lo >= ra.clip_min_count && (ra.maxiters < 0 || iteration < ra.maxiters)) {
    if (s[lo] == s[hi - 1]) break;  // no spread: every sample equals the center
    if (!in_range(s, lo, hi)) return false;
    int x, y;
    if (!clip_pass<float>(s, lo, hi, ra, &x, &y, &std) && !clip_pass_f64(s.c, lo, hi, ra, &x, &y, &std)) return false;
    ++iteration;
    if (x == lo && y == hi) break;
    lo = x;
    hi = y;
    std = -1.0f;
  }
  if (hi - lo < ra.clip_min_count) {
    *out = nan_of(0.0);
    return true;
  }
  if (ra.kind == kRobustSigmaMean) return exact_mean_of(s, lo, hi, low, out);
  if (ra.kind == kRobustSigmaMode) return mode_value(s, lo, hi, low, ra, std, out);
  const float a = s[lo + (hi - lo - 1) / 2], b = s[lo + (hi - lo) / 2];
  if (!sum_exact(a, b)) return false;
  *out = __float_as_uint(a) == __float_as_uint(b) ? widen(a) : __dmul_rn(__dadd_rn(widen(a), widen(b)), 0.5);
  return true;
}

// Blocks per SM the registers must allow: the network's wires and a few more.
template <int N>
constexpr int min_blocks() {
  return N <= 32 ? 8 : N <= 49 ? 6 : N <= 64 ? 5 : N <= 81 ? 4 : 2;
}

// MAD: the MAD kind; otherwise sigma clipping and the mode kind.
template <int N, bool MAD>
__global__ void __launch_bounds__(kT, min_blocks<N>())
    robust_tile_kernel(const float* __restrict__ in, float* __restrict__ out, const __grid_constant__ TileArgs a,
                       const __grid_constant__ net::TapTable<N> taps, const __grid_constant__ CUtensorMap tmap,
                       const __grid_constant__ RobustArgs ra, float2 scale, int column_offset) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int lowest;
  const Geom3& g = a.g;
  const Tile& t = a.t;
  long long* maps = reinterpret_cast<long long*>(smem_raw);
  uint32_t* keys = reinterpret_cast<uint32_t*>(maps + (t.SW + t.SH + g.kd));
  float* column = reinterpret_cast<float*>(smem_raw + column_offset) + threadIdx.x;
  long long z, y0, x0;
  net::tile_coords(a, blockIdx.x, z, y0, x0);
  const bool clip = !MAD && ra.kind >= kRobustSigmaMean;
  const bool drop_inf = clip || a.r.drop_inf;
  const uint32_t outside = sample_key<float>((float)a.r.cval, drop_inf);
  if (threadIdx.x == 0) lowest = INT_MAX;
  if (!stage_tile<true>(keys, maps, smem_raw, in, a, &tmap, z, y0, x0, outside,
                  [&](float v) { return sample_key<float>(v, drop_inf); }))
    return;
  __syncthreads();
  int low = 0;
  if (MAD || ra.kind != kRobustSigmaMedian) {
    const int staged = g.kd * t.SH * t.SW;
    int mine = INT_MAX;
    for (int i = threadIdx.x; i < staged; i += kT) mine = min(mine, lowest_bit(keys[i]));
    mine = __reduce_min_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0) atomicMin(&lowest, mine);
    __syncthreads();
    low = lowest;
  }
  const int V = a.r.count;
  for (int o = threadIdx.x; o < t.TW * t.TH; o += kT) {
    const int ty = o / t.TW, tx = o - ty * t.TW;
    const long long y = y0 + ty, x = x0 + tx;
    if (y >= g.H || x >= g.W) continue;
    const uint32_t* base = keys + ty * t.SW + tx;
    uint32_t k[N];
    int n = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      k[i] = i < V ? base[taps.off[i]] : KeyOf<float>::kSentinel;
      n += k[i] != KeyOf<float>::kSentinel ? 1 : 0;
    }
    net::batcher_sort<N>(k);
#pragma unroll
    for (int i = 0; i < N; ++i) column[i * kT] = KeyOf<float>::value(k[i]);
    const Column s{column};
    const bool none = clip ? n < ra.clip_min_count : (n == 0 || (a.r.omit ? n < a.r.min_count : n != V));
    float result = nan_of(0.0f);
    if constexpr (MAD) {
      if (!none) result = mad_value(s, n, low, scale, ra.parameter);
    } else if (!none && (clip || !(isinf(s[0]) || isinf(s[n - 1])))) {
      double value = 0.0;
      const bool ok = clip ? clipped_value(s, n, low, ra, &value) : mode_value(s, 0, n, low, ra, -1.0f, &value);
      result = !ok ? __uint_as_float(kUndecided) : nan64(value) ? nan_of(0.0f) : __double2float_rn(value);
    }
    out[(z * g.H + y) * g.W + x] = result;
  }
}

template <int N, bool MAD>
cudaError_t launch_width(const Plan& p, const float* in, float* out, cudaStream_t s) {
  net::TapTable<N> taps{};
  TileArgs args = p.tile;
  for (int i = 0; i < N && i < p.r.count; ++i) {
    const int* bt = &p.box_taps[(size_t)i * 3];
    taps.off[i] = (bt[0] * args.t.SH + bt[1]) * args.t.SW + bt[2];
  }
  auto kernel = robust_tile_kernel<N, MAD>;
  cudaError_t e = allow_max_smem((const void*)kernel);
  if (e != cudaSuccess) return e;
  CUtensorMap map{};
  size_t smem = p.smem_bytes;
  // The raw tile of a TMA copy comes on top of the keys and the columns.
  constexpr size_t kColumns = (size_t)N * kT * sizeof(float);
  tma_prepare(p, args.t, in, &map, &args, &smem);
  if (smem + 16 + kColumns > kRobustTileSmem) {
    args.tma_bw = 0;
    smem = p.smem_bytes;
  }
  const size_t columns = (smem + 15) & ~(size_t)15;
  // The second float of a scale below 2^-100 lies among the subnormals and lacks
  // bits that the product's bound counts on: no pair, every window in float64.
  const float scale = p.robust.parameter >= 7.888609052210118e-31 ? (float)p.robust.parameter : 0.0f;
  const float rest = scale > 0.0f ? (float)(p.robust.parameter - (double)scale) : 0.0f;
  kernel<<<(unsigned)args.t.tiles, kT, columns + kColumns, s>>>(in, out, args, taps, map, p.robust,
                                                                make_float2(scale, rest), (int)columns);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_kind(const Plan& p, const float* in, float* out, cudaStream_t s) {
  return p.robust.kind == kRobustMad ? launch_width<N, true>(p, in, out, s) : launch_width<N, false>(p, in, out, s);
}

}  // namespace robust_tile
}  // namespace ndf
