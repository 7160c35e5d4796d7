// K8 folding (fold::profile_at, fold/src/lib.rs:16-80) and K9 grid refinement
// (fold::refine, fold/src/lib.rs:81-97) for many trial periods in one launch.
//
// bin(t) = min(floor(fract(((t + offset) * tsamp) / period) * bins), bins-1)
// in f64 exactly as the reference (found in fixed point where that is certain).  Bin sums are f64; the per-CTA partial
// sums are combined in a fixed order.  For integer-valued series (sums of
// integer samples) every partial sum is an exact integer, so the result is
// independent of the order and equals the reference's sequential sum.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "psr_internal.h"

namespace psr {
namespace {

constexpr int FOLD_NT = 256;
constexpr int FOLD_MAXBINS = 1024;

// A fold's phase in fixed point: frac((t + offset) tsamp / period) as a 64-bit
// fraction of a cycle, from the exact ratio to 2^-106 (rhi:rlo, 128 fraction
// bits).  The reference's bin comes from three rounded f64 operations, whose
// error is bounded by the cycles folded; a fraction of a bin further than
// `margin` (in 2^-32 bins, that bound and the fixed point's) from both bin
// edges has the reference's bin for certain, and the few samples that do not
// (about 1 in 10^7) take the f64 operations themselves.  FP64 runs at 1/64 of
// the f32 rate on this part and has no divide instruction.
struct FoldPhase {
  unsigned long long rhi, rlo;
  double period, tsamp;
  uint32_t margin, pad;
};

// The rows' phases of a launch, as a kernel argument.
constexpr uint64_t FOLD_ROWS = 64;
struct FoldPhases {
  FoldPhase p[FOLD_ROWS];
};

// x 2^128 modulo 2^128 for a finite x >= 0.
unsigned __int128 fixed128(double x) {
  int e = 0;
  const double m = std::frexp(x, &e);  // x = m 2^e, m in [0.5, 1)
  const unsigned __int128 i = (unsigned __int128)(uint64_t)std::ldexp(m, 53);
  const int sh = e - 53 + 128;
  if (sh >= 128 || sh <= -53) return 0;
  return sh >= 0 ? i << sh : i >> -sh;
}

FoldPhase fold_phase(double tsamp, double period, uint64_t last, uint64_t bins) {
  const double r = tsamp / period, d = std::fma(-r, period, tsamp) / period;
  unsigned __int128 f = 0;
  if (r >= 0.0 && std::isfinite(r) && std::isfinite(d)) {
    f = fixed128(r);
    if (d >= 0.0) f += fixed128(d);
    else f -= fixed128(-d);
  }
  FoldPhase p{};
  p.rhi = (unsigned long long)(f >> 64);
  p.rlo = (unsigned long long)f;
  p.period = period;
  p.tsamp = tsamp;
  // bins (cycles 2^-51 + 2^-32 + 2^-52) in units of 2^-32 bins, and 2; a negative
  // ratio leaves every sample to the f64 operations
  const double cycles = (double)last * r;
  const double m = (double)bins * (cycles * 0x1p-19 + 1.0 + 0x1p-20) + 2.0;
  p.margin = r >= 0.0 && m < 2147483648.0 ? (uint32_t)std::ceil(m) : 0x80000000u;
  return p;
}

__device__ __forceinline__ unsigned long long phase_at(const FoldPhase &p,
                                                       unsigned long long i) {
  return i * p.rhi + __umul64hi(i, p.rlo);
}
// The bin of sample index i = t + offset with phase F.
__device__ __forceinline__ uint32_t bin_of(const FoldPhase &p, unsigned long long F, uint64_t i,
                                           uint32_t bins) {
  const unsigned long long u = (F >> 32) * bins;
  const uint32_t fr = (uint32_t)u;
  if (fr > p.margin && fr < 0u - p.margin) return (uint32_t)(u >> 32);
  const double q = __ddiv_rn(__dmul_rn((double)i, p.tsamp), p.period);
  const uint64_t b = (uint64_t)__dmul_rn(__dsub_rn(q, trunc(q)), (double)bins);
  return b > bins - 1 ? bins - 1 : (uint32_t)b;
}

// Samples as non-negative integers below 2^24, where they are (a dedispersed
// series of integer samples): false otherwise.
template <class T>
__device__ __forceinline__ bool as_count(T x, uint32_t &v) {
  if constexpr (sizeof(T) < 4) {
    v = (uint32_t)x;
    return true;
  } else {
    v = x >= 0.0f && x < 16777216.0f ? (uint32_t)x : 0u;
    return x >= 0.0f && x < 16777216.0f && (float)v == x;
  }
}

// Fold of row blockIdx.y (x + row * xstride) at period ph[row * phstride],
// samples [blockIdx.x * per_cta, ..).  Integer values add exactly in any order, so
// they go to 32-bit shared atomics: word A of a bin holds the sum of the low 11
// bits and, from bit 21, the count; word B the sum of the rest (left out while
// every value is below 2^11).  Each bin has `copies` pairs, thread t using copy t
// mod copies, which keeps lanes of one bin in different banks and every copy at
// 1024 samples or fewer (per_cta / copies), so neither field overflows.  Other
// values add in f64 as before.
// Measured on a GB300: 41 periods x 263,571 samples, 64 bins: 349 us with an f64
// divide and an f64 shared atomic (a CAS loop) per sample, 29 now; 96 8-bit
// rows of 263,500 samples 1.05 ms, 0.04 now.
template <class T>
__global__ void __launch_bounds__(FOLD_NT, 4)
    k_fold(const T *__restrict__ x, uint64_t xstride, uint64_t n, uint64_t offset,
           const __grid_constant__ FoldPhases ph, int phstride, uint32_t bins, int copies,
           uint64_t per_cta, double *__restrict__ psums, unsigned long long *__restrict__ pcounts) {
  extern __shared__ unsigned char sm_raw[];
  constexpr int VEC = 4 / (int)sizeof(T);        // samples per 32-bit load
  constexpr int PER = 8192 / FOLD_NT / VEC;      // loads per thread (per_cta <= 8192)
  const uint64_t row = blockIdx.y;
  x += row * xstride;
  const FoldPhase p = ph.p[row * phstride];
  const uint64_t t0 = (uint64_t)blockIdx.x * per_cta, t1 = min(t0 + per_cta, n);
  // 32 bits of samples from t (rows of 8- and 16-bit samples are 64-element
  // aligned and padded)
  auto load = [&](uint64_t t) -> uint32_t {
    if (t >= t1) return 0u;
    if constexpr (VEC > 1) return __ldg(reinterpret_cast<const uint32_t *>(x + t));
    else return __float_as_uint((float)__ldg(x + t));
  };
  // are the samples integers, and above 11 bits? (32 KB: read again from cache)
  bool ints = true, wide = false;
  if constexpr (sizeof(T) > 1) {
#pragma unroll 8
    for (int i = 0; i < PER; ++i) {
      const uint32_t raw = load(t0 + (uint64_t)VEC * (threadIdx.x + (uint64_t)i * FOLD_NT));
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        uint32_t v = 0;
        if constexpr (sizeof(T) == 4) ints &= as_count(__uint_as_float(raw), v);
        else v = (raw >> (16 * k)) & 0xffffu;
        wide |= v >= 2048u;
      }
    }
  }
  uint32_t *A = reinterpret_cast<uint32_t *>(sm_raw), *B = A + bins * copies;
  double *s = reinterpret_cast<double *>(sm_raw);
  unsigned *c = reinterpret_cast<unsigned *>(s + bins);
  ints = __syncthreads_and(ints);
  wide = __syncthreads_or(wide);
  if (ints) {
    for (uint32_t b = threadIdx.x; b < 2 * bins * copies; b += FOLD_NT) A[b] = 0;
  } else {
    for (uint32_t b = threadIdx.x; b < bins; b += FOLD_NT) {
      s[b] = 0.0;
      c[b] = 0;
    }
  }
  __syncthreads();
  const uint32_t copy = threadIdx.x & (uint32_t)(copies - 1);
  unsigned long long F = phase_at(p, t0 + (uint64_t)VEC * threadIdx.x + offset);
  const unsigned long long D1 = phase_at(p, 1), D = phase_at(p, (uint64_t)VEC * FOLD_NT);
#pragma unroll 4
  for (int i = 0; i < PER; ++i) {
    const uint64_t t = t0 + (uint64_t)VEC * (threadIdx.x + (uint64_t)i * FOLD_NT);
    const uint32_t raw = load(t);
    unsigned long long Fk = F;
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      if (t + k < t1) {
        const uint32_t b = bin_of(p, Fk, t + k + offset, bins);
        if (ints) {
          uint32_t v;
          if constexpr (sizeof(T) == 4) as_count(__uint_as_float(raw), v);
          else if constexpr (sizeof(T) == 2) v = (raw >> (16 * k)) & 0xffffu;
          else v = (raw >> (8 * k)) & 255u;
          atomicAdd(&A[b * copies + copy], (v & 2047u) | 1u << 21);
          if (wide) atomicAdd(&B[b * copies + copy], v >> 11);
        } else {
          atomicAdd(&s[b], (double)__uint_as_float(raw));
          atomicAdd(&c[b], 1u);
        }
      }
      Fk += D1;
    }
    F += D;
  }
  __syncthreads();
  const uint64_t slot = (row * gridDim.x + blockIdx.x) * bins;
  for (uint32_t b = threadIdx.x; b < bins; b += FOLD_NT) {
    if (ints) {
      unsigned long long sum = 0;
      unsigned cnt = 0;
      for (int k = 0; k < copies; ++k) {
        const int kk = (k + (int)threadIdx.x) & (copies - 1);
        const uint32_t a = A[b * copies + kk];
        sum += (a & 0x1fffffu) + ((unsigned long long)B[b * copies + kk] << 11);
        cnt += a >> 21;
      }
      psums[slot + b] = (double)sum;
      pcounts[slot + b] = cnt;
    } else {
      psums[slot + b] = s[b];
      pcounts[slot + b] = c[b];
    }
  }
}

// Launch shape of a fold: copies per bin, samples per CTA, shared memory.
struct FoldShape {
  int copies;
  uint64_t per_cta;
  size_t smem;
};
FoldShape fold_shape(uint64_t bins) {
  FoldShape f{bins <= 128 ? 16 : bins <= 256 ? 8 : 4, bins <= 256 ? 8192u : 4096u, 0};
  f.smem = std::max<size_t>(bins * f.copies * 8, bins * 12);
  return f;
}

__global__ void k_fold_reduce(const double *__restrict__ psums,
                              const unsigned long long *__restrict__ pcounts, uint64_t nparts,
                              uint64_t bins, uint64_t nper, double *__restrict__ sums,
                              unsigned long long *__restrict__ counts) {
  const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= nper * bins) return;
  const uint64_t per = id / bins, b = id % bins;
  double s = 0.0;
  unsigned long long cnt = 0;
  for (uint64_t p = 0; p < nparts; ++p) {
    s += psums[(per * nparts + p) * bins + b];
    cnt += pcounts[(per * nparts + p) * bins + b];
  }
  sums[id] = s;
  counts[id] = cnt;
}

// Sum and sum of squares of an integer series, exact: per CTA of MOM_PER samples
// (each below 2^24, so a CTA's squares stay below 2^61).  part[3 i + 2] is 0
// where a sample is not a non-negative integer below 2^24: the f64 passes below
// then give the moments.
constexpr int MI_NT = 256;
__global__ void __launch_bounds__(MI_NT)
    k_series_moments(const float *__restrict__ x, uint64_t xstride, uint64_t n,
                     uint64_t per, unsigned long long *__restrict__ part) {
  __shared__ unsigned long long red[2][MI_NT / 32];
  x += blockIdx.y * xstride;
  const uint64_t t0 = (uint64_t)blockIdx.x * per, t1 = min(t0 + per, n);
  unsigned long long s = 0, q = 0;
  bool ints = true;
  for (uint64_t t = t0 + threadIdx.x; t < t1; t += MI_NT) {
    uint32_t v;
    ints &= as_count(x[t], v);
    s += v;
    q += (unsigned long long)v * v;
  }
  for (int o = 16; o; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    q += __shfl_down_sync(0xffffffffu, q, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = s;
    red[1][threadIdx.x >> 5] = q;
  }
  ints = __syncthreads_and(ints);
  if (threadIdx.x == 0) {
    for (int w = 1; w < MI_NT / 32; ++w) {
      s += red[0][w];
      q += red[1][w];
    }
    unsigned long long *o = part + 3 * (blockIdx.y * (uint64_t)gridDim.x + blockIdx.x);
    o[0] = s;
    o[1] = q;
    o[2] = ints ? 1u : 0u;
  }
}

// Series mean and variance in f64 (fold/src/lib.rs:63-68), for series at
// x + blockIdx.y * xstride: pass 1 sums each CTA's slice (partials), pass 2
// (k_series_var) sums (x - mean)^2 with the mean taken from all partials.
constexpr int MOM_NT = 256, MOM_PER = 8192;
__global__ void __launch_bounds__(MOM_NT)
    k_series_sum(const float *__restrict__ x, uint64_t xstride, uint64_t n,
                 double *__restrict__ parts) {
  __shared__ double red[MOM_NT / 32];
  x += blockIdx.y * xstride;
  const uint64_t t0 = (uint64_t)blockIdx.x * MOM_PER, t1 = min(t0 + MOM_PER, n);
  double acc = 0.0;
  for (uint64_t t = t0 + threadIdx.x; t < t1; t += MOM_NT) acc += (double)x[t];
  for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < MOM_NT / 32; ++w) s += red[w];
    parts[blockIdx.y * gridDim.x + blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(MOM_NT)
    k_series_var(const float *__restrict__ x, uint64_t xstride, uint64_t n,
                 const double *__restrict__ sparts, uint32_t nparts,
                 double *__restrict__ vparts) {
  __shared__ double red[MOM_NT / 32];
  __shared__ double mean_s;
  x += blockIdx.y * xstride;
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (uint32_t i = 0; i < nparts; ++i) s += sparts[blockIdx.y * nparts + i];
    mean_s = s / (double)n;
  }
  __syncthreads();
  const double m = mean_s;
  const uint64_t t0 = (uint64_t)blockIdx.x * MOM_PER, t1 = min(t0 + MOM_PER, n);
  double acc = 0.0;
  for (uint64_t t = t0 + threadIdx.x; t < t1; t += MOM_NT) {
    const double d = __dsub_rn((double)x[t], m);
    acc = __dadd_rn(acc, __dmul_rn(d, d));
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < MOM_NT / 32; ++w) s += red[w];
    vparts[blockIdx.y * gridDim.x + blockIdx.x] = s;
  }
}

// confirmation::measure (search/src/confirmation.rs:107-141): on/off sums.
// Each warp covers 32 consecutive samples per step, so the on/off decision
// of every sample also lands in `bits` (one word per 32 samples) for the
// sequential pass.  part[block][8] = n0, s0, q0, n1, s1, q1, sum |v|, and the
// finest quantum exponent among the values (as a double).
constexpr int MEAS_NT = 256;
__global__ void __launch_bounds__(MEAS_NT)
    k_measure(const float *__restrict__ x, uint64_t n, uint64_t offset, double tsamp,
              double period, uint64_t start_bin, uint64_t width_bins, uint64_t bins,
              double *__restrict__ part, uint32_t *__restrict__ bits) {
  __shared__ double red[7][MEAS_NT / 32];
  __shared__ int redq[MEAS_NT / 32];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};  // n0, s0, q0, n1, s1, q1, sum |v|
  int qm = kNoQuantum;
  const double dbins = (double)bins;
  const int lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n;
       base += stride) {  // warp-uniform: base is a multiple of 32
    const uint64_t i = base + lane;
    int k = 0;
    if (i < n) {
      const double q = __ddiv_rn(__dmul_rn((double)(i + offset), tsamp), period);
      uint64_t b = (uint64_t)__dmul_rn(__dsub_rn(q, trunc(q)), dbins);
      if (b > bins - 1) b = bins - 1;
      k = ((b + bins - start_bin) % bins) < width_bins ? 1 : 0;
      const float xf = x[i];
      const double v = (double)xf;
      acc[3 * k] += 1.0;
      acc[3 * k + 1] = __dadd_rn(acc[3 * k + 1], v);
      acc[3 * k + 2] = __dadd_rn(acc[3 * k + 2], __dmul_rn(v, v));
      acc[6] = __dadd_rn(acc[6], fabs(v));
      qm = min(qm, quantum_exponent(xf));
    }
    const unsigned w = __ballot_sync(0xffffffffu, k);
    if (lane == 0) bits[base >> 5] = w;
  }
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    double a = acc[j];
    for (int o = 16; o; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) red[j][threadIdx.x >> 5] = a;
  }
  for (int o = 16; o; o >>= 1) qm = min(qm, __shfl_down_sync(0xffffffffu, qm, o));
  if (lane == 0) redq[threadIdx.x >> 5] = qm;
  __syncthreads();
  if (threadIdx.x < 7) {
    double a = 0.0;
    for (int w = 0; w < MEAS_NT / 32; ++w) a += red[threadIdx.x][w];
    part[blockIdx.x * 8 + threadIdx.x] = a;
  } else if (threadIdx.x == 7) {
    int q = kNoQuantum;
    for (int w = 0; w < MEAS_NT / 32; ++w) q = min(q, redq[w]);
    part[blockIdx.x * 8 + 7] = (double)q;
  }
}

// The same sums of an integer series, exact in 64-bit integers, with the bin
// from the fixed-point phase: part[block][7] = n0, s0, q0, n1, s1, q1, integers
// only.  (k_measure takes about 16 us of FP64 per 150,000 samples, this
// 3.)
__global__ void __launch_bounds__(MEAS_NT)
    k_measure_int(const float *__restrict__ x, uint64_t n, uint64_t offset, FoldPhase p,
                  uint32_t start_bin, uint32_t width_bins, uint32_t bins,
                  unsigned long long *__restrict__ part) {
  __shared__ unsigned long long red[6][MEAS_NT / 32];
  unsigned long long a[6] = {0, 0, 0, 0, 0, 0};
  bool ints = true;
  const uint64_t stride = (uint64_t)gridDim.x * MEAS_NT;
  uint64_t i = (uint64_t)blockIdx.x * MEAS_NT + threadIdx.x;
  unsigned long long F = phase_at(p, i + offset);
  const unsigned long long D = phase_at(p, stride);
  for (; i < n; i += stride, F += D) {
    uint32_t v;
    ints &= as_count(x[i], v);
    const uint32_t b = bin_of(p, F, i + offset, bins);
    uint32_t d = b + bins - start_bin;  // (b + bins - start) mod bins
    if (d >= bins) d -= bins;
    const unsigned long long q = (unsigned long long)v * v;
    if (d < width_bins) {
      a[3] += 1;
      a[4] += v;
      a[5] += q;
    } else {
      a[0] += 1;
      a[1] += v;
      a[2] += q;
    }
  }
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    for (int o = 16; o; o >>= 1) a[j] += __shfl_down_sync(0xffffffffu, a[j], o);
    if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = a[j];
  }
  ints = __syncthreads_and(ints);
  if (threadIdx.x < 6) {
    unsigned long long t = 0;
    for (int w = 0; w < MEAS_NT / 32; ++w) t += red[threadIdx.x][w];
    part[blockIdx.x * 7 + threadIdx.x] = t;
  }
  if (threadIdx.x == 6) part[blockIdx.x * 7 + 6] = ints ? 1u : 0u;
}

// The reference's own order for the on/off sums: one thread adds every
// sample in turn (each class from 0.0), as measure() does.  Used when the
// values make a reassociated f64 sum inexact (non-integer series).
__global__ void k_measure_seq(const float *__restrict__ x, uint64_t n,
                              const uint32_t *__restrict__ bits, double *__restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double s0 = 0.0, q0 = 0.0, s1 = 0.0, q1 = 0.0;
  for (uint64_t i = 0; i < n; ++i) {
    const double v = (double)x[i];
    const double v2 = __dmul_rn(v, v);
    if ((bits[i >> 5] >> (i & 31)) & 1u) {
      s1 = __dadd_rn(s1, v);
      q1 = __dadd_rn(q1, v2);
    } else {
      s0 = __dadd_rn(s0, v);
      q0 = __dadd_rn(q0, v2);
    }
  }
  out[0] = s0;
  out[1] = q0;
  out[2] = s1;
  out[3] = q1;
}

int32_t key32(float x) {
  int32_t i;
  std::memcpy(&i, &x, 4);
  return i ^ (int32_t)((uint32_t)(i >> 31) >> 1);
}
bool tless(float a, float b) { return key32(a) < key32(b); }

float upper_median(std::vector<float> v) {
  if (v.empty()) return 0.0f;
  size_t i = v.size() / 2;
  std::nth_element(v.begin(), v.begin() + i, v.end(), tless);
  return v[i];
}

}  // namespace

// Profile statistics from bin sums/counts (fold/src/lib.rs:39-79), host.
void profile_stats(const double *sums, const unsigned long long *cnts, uint64_t bins,
                   double smean, double svar, double period, psr_profile_stats *st,
                   float *values, uint64_t *counts) {
  std::vector<float> vals(bins);
  for (uint64_t b = 0; b < bins; ++b)
    vals[b] = cnts[b] > 0 ? (float)(sums[b] / (double)cnts[b]) : 0.0f;
  const float center = upper_median(vals);
  std::vector<float> off;
  for (uint64_t b = 0; b < bins; ++b)
    if (cnts[b] > 0) off.push_back(vals[b]);
  std::sort(off.begin(), off.end(), tless);
  off.resize(std::max<size_t>(off.size() * 3 / 4, 1));
  double mean = -0.0;
  for (float v : off) mean += (double)v;
  mean /= (double)off.size();
  double var = -0.0;
  for (float v : off) {
    const double d = (double)v - mean;
    var += d * d;
  }
  const double sigma = std::sqrt(var / (double)off.size());
  float peak = -INFINITY;
  for (float v : vals) peak = std::fmax(peak, v);
  st->period_s = period;
  st->snr = sigma > 1e-12 ? ((double)peak - (double)center) / sigma : 0.0;
  uint64_t populated = 0;
  for (uint64_t b = 0; b < bins; ++b) populated += cnts[b] > 0;
  if (svar > 1e-12 && populated > 1) {
    double s = -0.0;
    for (uint64_t b = 0; b < bins; ++b) {
      const double d = (double)vals[b] - smean;
      s += (double)cnts[b] * (d * d) / svar;
    }
    st->reduced_chi_square = s / (double)(populated - 1);
  } else {
    st->reduced_chi_square = 0.0;
  }
  if (values) std::copy(vals.begin(), vals.end(), values);
  if (counts)
    for (uint64_t b = 0; b < bins; ++b) counts[b] = cnts[b];
}

int fold_profiles(const float *d_x, uint64_t n, double tsamp, const double *periods,
                  uint64_t nper, uint64_t bins, uint64_t offset, psr_profile_stats *stats,
                  float *values, uint64_t *counts, cudaStream_t st) {
  return fold_profiles_ex(d_x, 0, n, tsamp, periods, nper, bins, offset, stats, values, counts,
                          st);
}

// Fold nper (series, period) pairs: series p starts at d_x + p * xstride
// (xstride 0: one series at every period); stats/values/counts are arrays of
// nper entries (values/counts nper*bins).
int fold_profiles_ex(const float *d_x, uint64_t xstride, uint64_t n, double tsamp,
                     const double *periods, uint64_t nper, uint64_t bins, uint64_t offset,
                     psr_profile_stats *stats, float *values, uint64_t *counts,
                     cudaStream_t st) {
  if (bins < 4 || bins > FOLD_MAXBINS || n == 0) {
    set_error("profile_at: 4 <= bins <= 1024 and a non-empty series are required");
    return PSR_EINVAL;
  }
  const FoldShape f = fold_shape(bins);
  const uint64_t nparts = (n + f.per_cta - 1) / f.per_cta;
  const uint64_t nser = xstride ? nper : 1;
  const uint32_t mparts = (uint32_t)((n + MOM_PER - 1) / MOM_PER);
  // partial sums and counts; then sums, counts and moments, read back in one copy
  const size_t nb = (size_t)(nper * bins), np = nb * nparts, nm = (size_t)nser * mparts * 3;
  DevBuf parts, res;
  PSR_TRY(parts.ensure(2 * np * 8));
  PSR_TRY(res.ensure((2 * nb + nm) * 8));
  double *psums = parts.as<double>(), *sums = res.as<double>();
  unsigned long long *pcounts = parts.as<unsigned long long>() + np;
  unsigned long long *cnts = res.as<unsigned long long>() + nb, *mom = cnts + nb;
  FoldPhases ph{};
  for (uint64_t r0 = 0; r0 < nper; r0 += FOLD_ROWS) {
    const uint64_t nr = std::min(FOLD_ROWS, nper - r0);
    for (uint64_t p = 0; p < nr; ++p)
      ph.p[p] = fold_phase(tsamp, periods[r0 + p], n + offset, bins);
    k_fold<float><<<dim3((unsigned)nparts, (unsigned)nr), FOLD_NT, f.smem, st>>>(
        d_x + r0 * xstride, xstride, n, offset, ph, 1, (uint32_t)bins, f.copies, f.per_cta,
        psums + r0 * nparts * bins, pcounts + r0 * nparts * bins);
  }
  PSR_CUDA(cudaGetLastError());
  k_fold_reduce<<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(psums, pcounts, nparts, bins, nper,
                                                             sums, cnts);
  k_series_moments<<<dim3(mparts, (unsigned)nser), MI_NT, 0, st>>>(d_x, xstride, n, MOM_PER, mom);
  PSR_CUDA(cudaGetLastError());
  std::vector<unsigned long long> back(2 * nb + nm), hc(nb), hmom(nm);
  std::vector<double> hs(nb), hm(2 * nser);
  PSR_CUDA(cudaMemcpyAsync(back.data(), res.p, back.size() * 8, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  std::memcpy(hs.data(), back.data(), nb * 8);
  std::memcpy(hc.data(), back.data() + nb, nb * 8);
  std::memcpy(hmom.data(), back.data() + 2 * nb, nm * 8);
  bool ints = true;
  for (size_t i = 0; i < hmom.size(); i += 3) ints = ints && hmom[i + 2] != 0;
  if (ints) {
    // n sum x^2 - (sum x)^2 in exact integers: n times the squared deviations
    for (uint64_t m = 0; m < nser; ++m) {
      unsigned __int128 s1 = 0, s2 = 0;
      for (uint32_t i = 0; i < mparts; ++i) {
        s1 += hmom[3 * (m * mparts + i)];
        s2 += hmom[3 * (m * mparts + i) + 1];
      }
      hm[2 * m] = (double)s1;
      hm[2 * m + 1] = (double)((unsigned __int128)n * s2 - s1 * s1) / (double)n;
    }
  } else {
    DevBuf sp, vp;
    PSR_TRY(sp.ensure((size_t)nser * mparts * 8));
    PSR_TRY(vp.ensure((size_t)nser * mparts * 8));
    k_series_sum<<<dim3(mparts, (unsigned)nser), MOM_NT, 0, st>>>(d_x, xstride, n,
                                                                 sp.as<double>());
    k_series_var<<<dim3(mparts, (unsigned)nser), MOM_NT, 0, st>>>(d_x, xstride, n,
                                                                 sp.as<double>(), mparts,
                                                                 vp.as<double>());
    PSR_CUDA(cudaGetLastError());
    std::vector<double> hsp((size_t)nser * mparts), hvp((size_t)nser * mparts);
    PSR_CUDA(cudaMemcpyAsync(hsp.data(), sp.p, hsp.size() * 8, cudaMemcpyDeviceToHost, st));
    PSR_CUDA(cudaMemcpyAsync(hvp.data(), vp.p, hvp.size() * 8, cudaMemcpyDeviceToHost, st));
    PSR_CUDA(cudaStreamSynchronize(st));
    for (uint64_t m = 0; m < nser; ++m) {
      double s1 = 0.0, s2 = 0.0;
      for (uint32_t i = 0; i < mparts; ++i) {
        s1 += hsp[m * mparts + i];
        s2 += hvp[m * mparts + i];
      }
      hm[2 * m] = s1;
      hm[2 * m + 1] = s2;
    }
  }
  for (uint64_t p = 0; p < nper; ++p) {
    const uint64_t m = xstride ? p : 0;
    const double smean = hm[2 * m] / (double)n;
    const double svar = hm[2 * m + 1] / (double)n;
    profile_stats(hs.data() + p * bins, hc.data() + p * bins, bins, smean, svar, periods[p],
                  &stats[p], values ? values + p * bins : nullptr,
                  counts ? counts + p * bins : nullptr);
  }
  return PSR_OK;
}

}  // namespace psr

namespace psr {

int measure_device(const float *d_x, uint64_t n, uint64_t offset, double tsamp, double period,
                   uint64_t start_bin, uint64_t width_bins, uint64_t bins, psr_measurement *out,
                   cudaStream_t st) {
  const unsigned nb = (unsigned)std::min<uint64_t>((n + 1023) / 1024, 1024);
  uint64_t cnt[2];
  double sum[2], sum2[2];
  DevBuf part, bits;
  bool ints = bins <= 0x40000000ull;
  if (ints) {
    PSR_TRY(part.ensure((size_t)nb * 7 * 8));
    k_measure_int<<<nb, MEAS_NT, 0, st>>>(d_x, n, offset, fold_phase(tsamp, period, n + offset, bins),
                                          (uint32_t)start_bin, (uint32_t)width_bins,
                                          (uint32_t)bins, part.as<unsigned long long>());
    PSR_CUDA(cudaGetLastError());
    std::vector<unsigned long long> h((size_t)nb * 7);
    PSR_CUDA(cudaMemcpyAsync(h.data(), part.p, h.size() * 8, cudaMemcpyDeviceToHost, st));
    PSR_CUDA(cudaStreamSynchronize(st));
    unsigned __int128 a[6] = {0, 0, 0, 0, 0, 0};
    for (unsigned b = 0; b < nb; ++b) {
      ints = ints && h[(size_t)b * 7 + 6] != 0;
      for (int j = 0; j < 6; ++j) a[j] += h[(size_t)b * 7 + j];
    }
    // (below 2^53 the reference's sequential f64 sums are these integers)
    for (int j = 0; j < 6; ++j) ints = ints && a[j] < ((unsigned __int128)1 << 53);
    for (int k = 0; k < 2; ++k) {
      cnt[k] = (uint64_t)a[3 * k];
      sum[k] = (double)(uint64_t)a[3 * k + 1];
      sum2[k] = (double)(uint64_t)a[3 * k + 2];
    }
  }
  if (!ints) {
    PSR_TRY(part.ensure((size_t)nb * 8 * 8 + 4 * 8));
    PSR_TRY(bits.ensure(((n + 31) / 32 + 1) * 4));
    k_measure<<<nb, MEAS_NT, 0, st>>>(d_x, n, offset, tsamp, period, start_bin, width_bins, bins,
                                      part.as<double>(), bits.as<uint32_t>());
    PSR_CUDA(cudaGetLastError());
    std::vector<double> h((size_t)nb * 8);
    PSR_CUDA(cudaMemcpyAsync(h.data(), part.p, h.size() * 8, cudaMemcpyDeviceToHost, st));
    PSR_CUDA(cudaStreamSynchronize(st));
    double a[7] = {0, 0, 0, 0, 0, 0, 0};
    int qmin = kNoQuantum;
    for (unsigned b = 0; b < nb; ++b) {
      for (int j = 0; j < 7; ++j) a[j] += h[(size_t)b * 8 + j];
      qmin = std::min(qmin, (int)h[(size_t)b * 8 + 7]);
    }
    for (int k = 0; k < 2; ++k) {
      cnt[k] = (uint64_t)a[3 * k];
      sum[k] = a[3 * k + 1];
      sum2[k] = a[3 * k + 2];
    }
    // Integer-valued series (sums of integer samples) give exact partial sums
    // in any order.  Otherwise the order matters: sums of v are exact while
    // sum |v| < 2^(53+q), sums of v^2 (multiples of 2^2q) while
    // sum v^2 < 2^(53+2q); failing either, add in the reference's order.
    const bool exact = f64_sums_exact(a[6], qmin) &&
                       (qmin >= kNoQuantum || f64_sums_exact(a[2] + a[5], 2 * qmin));
    if (!exact) {
      double *d_seq = part.as<double>() + (size_t)nb * 8;
      k_measure_seq<<<1, 32, 0, st>>>(d_x, n, bits.as<uint32_t>(), d_seq);
      PSR_CUDA(cudaGetLastError());
      double hq[4];
      PSR_CUDA(cudaMemcpyAsync(hq, d_seq, sizeof(hq), cudaMemcpyDeviceToHost, st));
      PSR_CUDA(cudaStreamSynchronize(st));
      sum[0] = hq[0];
      sum2[0] = hq[1];
      sum[1] = hq[2];
      sum2[1] = hq[3];
    }
  }
  out->on_samples = cnt[1];
  out->off_samples = cnt[0];
  if (cnt[0] < 2 || cnt[1] < 2) {
    out->snr = 0.0;
    out->mean_difference = 0.0;
    out->standard_error = 0.0;
    return PSR_OK;
  }
  const double diff = sum[1] / (double)cnt[1] - sum[0] / (double)cnt[0];
  auto var = [&](int k) {
    return std::fmax((sum2[k] - sum[k] * sum[k] / (double)cnt[k]) / (double)(cnt[k] - 1), 0.0);
  };
  const double err = std::sqrt(var(1) / (double)cnt[1] + var(0) / (double)cnt[0]);
  out->snr = err > 1e-10 ? diff / err : 0.0;
  out->mean_difference = diff;
  out->standard_error = err;
  return PSR_OK;
}

}  // namespace psr

// ---------------------------------------------------------------------------
// Per-channel discovery profiles and the DM response of
// confirmation::analyze (search/src/confirmation.rs:391-433).
namespace psr {
namespace {

// comb[trial][b] = sum over channels (in channel order) of the linearly
// interpolated, mean-removed channel profile shifted by delay*tsamp/period
// bins; the f64 operations and their order follow confirmation.rs:403-413.
// One CTA per trial.  The position b + shift is b added to the shift's whole and
// fractional parts while the sum stays in the shift's binade (both are multiples
// of its ulp there, so the rounded sum is exact); bins at or past `lim` take the
// rounded sum.  Then a term is two products and two sums in f64, instead of a
// remainder, a floor and three differences more; FP64 (1/64 of the f32 rate)
// bounds the kernel.  Measured on a GB300: 96 channels, 2000 trials, 64 bins: 640
// us, 205 now.
struct DmShift {
  double f, w;   // fraction, 1 - fraction
  int whole, lim;  // whole part modulo bins; first bin outside the binade
};
// dev[c][b] = profile - its mean.
__global__ void __launch_bounds__(256)
    k_dm_deviations(const float *__restrict__ chp, const double *__restrict__ chmean,
                    uint64_t nch, uint64_t bins, double *__restrict__ dev) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < nch * bins) dev[i] = __dsub_rn((double)chp[i], chmean[i / bins]);
}
constexpr int DR_C = 256;  // channels' shifts held at a time
__global__ void __launch_bounds__(128)
    k_dm_response(const double *__restrict__ dev, const uint32_t *__restrict__ delays,
                  uint64_t nch, int bins, double tsamp, double period,
                  double *__restrict__ comb) {
  __shared__ double shift[DR_C];
  __shared__ DmShift sh[DR_C];
  const uint64_t trial = blockIdx.x;
  const double dbins = (double)bins;
  double out[8];  // bins <= 8 threads' worth
#pragma unroll
  for (int k = 0; k < 8; ++k) out[k] = 0.0;
  for (uint64_t c0 = 0; c0 < nch; c0 += DR_C) {
    const int nc = (int)min((uint64_t)DR_C, nch - c0);
    __syncthreads();
    for (int c = threadIdx.x; c < nc; c += (int)blockDim.x) {
      const double d = (double)delays[trial * nch + c0 + c];
      const double x = __dmul_rn(__ddiv_rn(__dmul_rn(d, tsamp), period), dbins);
      shift[c] = x;
      const double fl = floor(x);
      DmShift s;
      s.f = __dsub_rn(x, fl);
      s.w = __dsub_rn(1.0, s.f);
      s.whole = (int)((unsigned long long)fl % (unsigned)bins);
      // the binade's end, 2^(e + 1), minus x: b below it keeps b + x exact
      const int e = (int)((unsigned long long)__double_as_longlong(x) >> 52);  // biased
      s.lim = bins;
      if (x > 0.0) {
        const double end = __longlong_as_double((long long)(e + 1) << 52);
        s.lim = (int)fmin(ceil(__dsub_rn(end, x)), dbins);
      }
      sh[c] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int b = (int)threadIdx.x + (int)blockDim.x * k;
      if (b >= bins) break;
      double o = out[k];
      for (int c = 0; c < nc; ++c) {
        const DmShift s = sh[c];
        int index = s.whole + b;
        if (index >= bins) index -= bins;
        double f = s.f, w = s.w;
        if (b >= s.lim) {
          const double x = __dadd_rn((double)b, shift[c]), fl = floor(x);
          index = (int)((unsigned long long)fl % (unsigned)bins);
          f = __dsub_rn(x, fl);
          w = __dsub_rn(1.0, f);
        }
        const double *row = dev + (c0 + c) * (uint64_t)bins;
        const double v0 = __ldg(row + index), v1 = __ldg(row + (index + 1 == bins ? 0 : index + 1));
        o = __dadd_rn(o, __dadd_rn(__dmul_rn(v0, w), __dmul_rn(v1, f)));
      }
      out[k] = o;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int b = (int)threadIdx.x + (int)blockDim.x * k;
    if (b < bins) comb[trial * (uint64_t)bins + b] = out[k];
  }
}

}  // namespace

int fold_channels(const DeviceObs &o, uint64_t n, double tsamp, double period, uint64_t bins,
                  std::vector<float> &values, cudaStream_t st) {
  if (bins < 4 || bins > FOLD_MAXBINS || n == 0 || n > o.ns) {
    set_error("profile: 4 <= bins <= 1024 and 0 < n <= nsamples are required");
    return PSR_EINVAL;
  }
  const FoldShape f = fold_shape(bins);
  const uint64_t nparts = (n + f.per_cta - 1) / f.per_cta;
  const size_t nb = (size_t)(o.nch * bins), np = nb * nparts;
  DevBuf parts, res;
  PSR_TRY(parts.ensure(2 * np * 8));
  PSR_TRY(res.ensure(2 * nb * 8));
  double *psums = parts.as<double>();
  unsigned long long *pcounts = parts.as<unsigned long long>() + np;
  FoldPhases ph{};
  ph.p[0] = fold_phase(tsamp, period, n, bins);
  const dim3 grid((unsigned)nparts, (unsigned)o.nch);
  auto run = [&](auto *x) {
    k_fold<<<grid, FOLD_NT, f.smem, st>>>(x, o.ld, n, (uint64_t)0, ph, 0, (uint32_t)bins,
                                          f.copies, f.per_cta, psums, pcounts);
  };
  switch (o.kind) {
    case SAMPLE_U8: run(o.samples.as<const uint8_t>()); break;
    case SAMPLE_U16: run(o.samples.as<const uint16_t>()); break;
    default: run(o.samples.as<const float>());
  }
  PSR_CUDA(cudaGetLastError());
  k_fold_reduce<<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(
      psums, pcounts, nparts, bins, o.nch, res.as<double>(), res.as<unsigned long long>() + nb);
  PSR_CUDA(cudaGetLastError());
  std::vector<unsigned long long> back(2 * nb), hc(nb);
  std::vector<double> hs(nb);
  PSR_CUDA(cudaMemcpyAsync(back.data(), res.p, back.size() * 8, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  std::memcpy(hs.data(), back.data(), nb * 8);
  std::memcpy(hc.data(), back.data() + nb, nb * 8);
  values.resize(o.nch * bins);
  for (uint64_t i = 0; i < o.nch * bins; ++i)
    values[i] = hc[i] > 0 ? (float)(hs[i] / (double)hc[i]) : 0.0f;
  return PSR_OK;
}

int dm_response(const std::vector<float> &chp, const std::vector<double> &chmean,
                const uint32_t *d_delays, uint64_t ntrials, uint64_t nch, uint64_t bins,
                double tsamp, double period, std::vector<double> &comb, cudaStream_t st) {
  DevBuf dp, dm, dc, dv;
  PSR_TRY(dp.ensure(chp.size() * 4));
  PSR_TRY(dm.ensure(chmean.size() * 8));
  PSR_TRY(dv.ensure(chp.size() * 8));
  PSR_TRY(dc.ensure(ntrials * bins * 8));
  PSR_CUDA(cudaMemcpyAsync(dp.p, chp.data(), chp.size() * 4, cudaMemcpyHostToDevice, st));
  PSR_CUDA(cudaMemcpyAsync(dm.p, chmean.data(), chmean.size() * 8, cudaMemcpyHostToDevice, st));
  k_dm_deviations<<<(unsigned)((nch * bins + 255) / 256), 256, 0, st>>>(
      dp.as<float>(), dm.as<double>(), nch, bins, dv.as<double>());
  k_dm_response<<<(unsigned)ntrials, bins <= 64 ? 64 : 128, 0, st>>>(dv.as<double>(), d_delays, nch, (int)bins,
                                                   tsamp, period, dc.as<double>());
  PSR_CUDA(cudaGetLastError());
  comb.resize(ntrials * bins);
  PSR_CUDA(cudaMemcpyAsync(comb.data(), dc.p, comb.size() * 8, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  return PSR_OK;
}

}  // namespace psr

extern "C" int psr_test_fold_phase(double tsamp, double period, uint64_t last, uint64_t bins,
                                   uint64_t *out) {
  if (!out) {
    psr::set_error("test_fold_phase: null argument");
    return PSR_EINVAL;
  }
  const psr::FoldPhase p = psr::fold_phase(tsamp, period, last, bins);
  out[0] = p.rhi;
  out[1] = p.rlo;
  out[2] = p.margin;
  return PSR_OK;
}
