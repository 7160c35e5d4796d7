// Gradient refinement on a folded cube: fold once, then optimise on the
// folded data.  Used by psr_refine_gradient for groups of nearby starting
// points (up to 16 of them).
//
// One pass over the filterbank folds every channel at a reference (nu_r,
// nudot_r, DM_r) into a cube C[c][s][b] (channels x subints x bins),
// channel c at its own dispersion-delayed phase
//   phi_r(c, T) = nu_r (T - tau_c) + nudot_r (T - tau_c)^2 / 2,
//   tau_c(DM) = 4148.808 DM (f_c^-2 - f_max^-2) seconds (fractional),
// with cloud-in-cell weights.  For parameters theta near the reference, the
// samples of (c, s) move in phase by d_cs = B (phi_theta(c, T_s) -
// phi_r(c, T_s)) bins, T_s the subint centre (the drift within one subint is
// neglected).  Each cube row's DFT R_cs[k] (k = 1..B/2) is taken once;
// shifting a row by d bins multiplies harmonic k by e^(-2 pi i k d / B) (a
// band-limited shift: no interpolation smoothing that would depend on the
// fractional shift), so the profile's harmonics are
//   P_k = sum_cs R_cs[k] e^(-2 pi i k d_cs / B)
// and, by Parseval, J = sum_b (p_b - mean)^2 / (n v) = sum_k w_k |P_k|^2 /
// (B n v), w_k = 2 (k < B/2), 1 (k = B/2), v = sum_c var(x_c).  Adjoint:
//   dJ/dd_cs = sum_k Re(A_k R_cs[k] e^(-2 pi i k d_cs/B) (-2 pi i k / B)),
//   A_k = 2 w_k conj(P_k) / (B n v),
//   dd_cs/dnu = B (T_s - tau_c), dd_cs/dnudot = B (T_s - tau_c)^2 / 2,
//   dd_cs/dDM = -B (nu + nudot (T_s - tau_c)) dtau_c/dDM.
// Evaluations of every candidate of a group run in the same launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "psr_internal.h"
#include "refine.h"

namespace psr {

// Device buffers of one cube, reused by every group of a refinement call.
struct CubeWork {
  DevBuf cube, R, chsum, tau, kc, ref, dsh, anchors, prof, g;
  uint64_t rows = 0;
  double var = 1.0;
};
CubeCache::~CubeCache() { delete w; }

namespace {

constexpr double K_DM_C = 4148.808;  // dedisperse/src/lib.rs:3
constexpr int CB_NT = 256;
constexpr int CB_MAXB = 1024;

// Fold subint s of channel c (one CTA) into C[c][s][*] (the row's mean
// removed, which leaves every shifted profile's deviations unchanged and keeps
// f32 sums accurate) and the channel's sum / sum of squares.
//
// The row is cut into runs of 32 samples aligned to the global sample grid
// (rows start 64-element aligned and carry >= 64 elements of padding, so a
// run is one to eight aligned 16-byte loads that never leave the row); thread
// j folds a contiguous stretch of runs of the subint, prefetching its next run
// while it folds the current one.  Samples of a boundary run outside [t0, t1) are
// zeroed.  Phases are fixed-point fractions of a cycle (u64, 2^-64 cycle
// resolution): an f64 anchor at the first run (k_cube_anchors), then per-thread
// offsets and per-stride advances by exact integer second differences, so no
// thread does f64 work per run.  Inside a run the bin position u (in bins)
// advances in f32; for du < 1 bin per sample the bin index is walked
// incrementally (one compare per sample), otherwise floored per sample.
// Consecutive samples of one bin are summed in registers (a0 = sum v, a1 =
// sum w v; CIC weights 1 - w and w), across run boundaries, and flushed with
// two shared-memory atomics when the bin changes.  Channel sums are integer (u8, u16) or f32
// per run (f32 data) before the f64 reduction.
constexpr int CB_RUN = 32;

template <class T>
struct RunRegs {
  static constexpr int W = (CB_RUN * (int)sizeof(T)) / 16;  // 16-byte words per run
  uint4 r[W];
};

template <class T>
__device__ __forceinline__ void load_run(const T *p, RunRegs<T> &x) {
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
#pragma unroll
  for (int k = 0; k < RunRegs<T>::W; ++k) x.r[k] = __ldg(q + k);
}

__device__ __forceinline__ uint32_t word_of(const uint4 &v, int k) {
  return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

// Sample i (0..31) of a run as f32 (integer samples are exact: 2^23 + v
// assembled by a byte permute, then 2^23 subtracted).
template <class T>
__device__ __forceinline__ float run_sample(const RunRegs<T> &x, int i);
template <>
__device__ __forceinline__ float run_sample<uint8_t>(const RunRegs<uint8_t> &x, int i) {
  const uint32_t w = word_of(x.r[i >> 4], (i >> 2) & 3);
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (unsigned)(i & 3))) - 8388608.0f;
}
template <>
__device__ __forceinline__ float run_sample<uint16_t>(const RunRegs<uint16_t> &x, int i) {
  const uint32_t w = word_of(x.r[i >> 3], (i >> 1) & 3);
  const unsigned lo = (unsigned)(i & 1) * 2u;
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7500u | ((lo + 1u) << 4) | lo)) -
         8388608.0f;
}
template <>
__device__ __forceinline__ float run_sample<float>(const RunRegs<float> &x, int i) {
  return __uint_as_float(word_of(x.r[i >> 2], i & 3));
}

// Zero the samples of a run outside [lo, hi) (boundary runs only).
template <class T>
__device__ __forceinline__ void mask_run(RunRegs<T> &x, int lo, int hi) {
  constexpr int PER_WORD = 4 / (int)sizeof(T);
#pragma unroll
  for (int k = 0; k < RunRegs<T>::W; ++k) {
    uint32_t w[4] = {x.r[k].x, x.r[k].y, x.r[k].z, x.r[k].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int b = 0; b < PER_WORD; ++b) {
        const int i = (k * 4 + e) * PER_WORD + b;
        if (i < lo || i >= hi) {
          const uint32_t m = sizeof(T) == 4 ? 0xffffffffu
                                            : (((1u << (8 * sizeof(T))) - 1u) << (8 * sizeof(T) * b));
          w[e] &= ~m;
        }
      }
    }
    x.r[k] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Channel-sum accumulators: exact integers for 8/16-bit samples.
template <class T>
struct RunSums {
  unsigned long long s = 0, q = 0;
  __device__ __forceinline__ void add(const RunRegs<T> &x) {
    unsigned s32 = 0, q32 = 0;
#pragma unroll
    for (int k = 0; k < RunRegs<T>::W; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t w = word_of(x.r[k], e);
        if (sizeof(T) == 1) {
          s32 = __dp4a(w, 0x01010101u, s32);
          q32 = __dp4a(w, w, q32);  // <= 32 * 255^2 per run
        } else {
          const uint32_t a = w & 0xffffu, b = w >> 16;
          s32 += a + b;
          q += (unsigned long long)(a * a) + (unsigned long long)(b * b);
        }
      }
    s += s32;
    q += q32;
  }
  // One 16-byte chunk (staged tiles).
  __device__ __forceinline__ void add_chunk(const uint4 &v) {
    unsigned s32 = 0, q32 = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t w = word_of(v, e);
      if (sizeof(T) == 1) {
        s32 = __dp4a(w, 0x01010101u, s32);
        q32 = __dp4a(w, w, q32);
      } else {
        const uint32_t a = w & 0xffffu, b = w >> 16;
        s32 += a + b;
        q += (unsigned long long)(a * a) + (unsigned long long)(b * b);
      }
    }
    s += s32;
    q += q32;
  }
  __device__ __forceinline__ void end_tile(const uint4 *, int) {}
  // Lane 0: the warp's sums (integers below 2^53).
  __device__ __forceinline__ void warp_total(double &sum, double &sq) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      s += __shfl_down_sync(0xffffffffu, s, o);
      q += __shfl_down_sync(0xffffffffu, q, o);
    }
    sum = (double)s;
    sq = (double)q;
  }
};
// f32 sums of v and v^2 over a chunk of 4 (or a run of 32) join sums of three
// f32 words, each the exact error of the one before (TwoSum): with the 24 bits
// of the terms nothing is lost that an f64 sum keeps.  What passes f32's range
// goes to f64 (FP64 runs at 1/64 of the f32 rate: two conversions and two sums
// per chunk and f64 shuffles were half of the time of the fold).
struct Sum3 {
  float h = 0.0f, l = 0.0f, m = 0.0f;
  // a + b, the error left in b
  static __device__ __forceinline__ void two_sum(float &a, float &b) {
    const float t = __fadd_rn(a, b), v = __fsub_rn(t, a);
    b = __fadd_rn(__fsub_rn(a, __fsub_rn(t, v)), __fsub_rn(b, v));
    a = t;
  }
  __device__ __forceinline__ void add(float x) {
    two_sum(h, x);
    two_sum(l, x);
    m = __fadd_rn(m, x);
  }
  __device__ __forceinline__ void add(const Sum3 &o) {
    add(o.h);
    float x = o.l;
    two_sum(l, x);
    m = __fadd_rn(m, __fadd_rn(x, o.m));
  }
  __device__ __forceinline__ bool finite() const { return isfinite(h) && isfinite(l) && isfinite(m); }
  __device__ __forceinline__ double value() const {
    return (double)h + ((double)l + (double)m);
  }
  __device__ __forceinline__ Sum3 from(int o) const {  // the lane o above's
    Sum3 x;
    x.h = __shfl_down_sync(0xffffffffu, h, o);
    x.l = __shfl_down_sync(0xffffffffu, l, o);
    x.m = __shfl_down_sync(0xffffffffu, m, o);
    return x;
  }
};
template <>
struct RunSums<float> {
  Sum3 ps, pq, ts, tq;      // so far; of the open tile
  double s = 0.0, q = 0.0;  // what passed f32's range
  __device__ __forceinline__ void join(const Sum3 &a, const Sum3 &b) {
    const Sum3 os = ps, oq = pq;
    ps.add(a);
    pq.add(b);
    if (!(ps.finite() && pq.finite())) {
      s += os.value() + a.value();
      q += oq.value() + b.value();
      ps = pq = Sum3();
    }
  }
  __device__ __forceinline__ void add(const RunRegs<float> &x) {
    Sum3 a, b;
#pragma unroll
    for (int i = 0; i < CB_RUN; ++i) {
      const float v = run_sample<float>(x, i);
      a.h += v;
      b.h = fmaf(v, v, b.h);
    }
    join(a, b);
  }
  static __device__ __forceinline__ void chunk_sums(const uint4 &v, float &cs, float &cq) {
    cs = cq = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = __uint_as_float(word_of(v, e));
      cs += x;
      cq = fmaf(x, x, cq);
    }
  }
  __device__ __forceinline__ void add_chunk(const uint4 &v) {
    float cs, cq;
    chunk_sums(v, cs, cq);
    ts.add(cs);
    tq.add(cq);
  }
  // The lane's chunks of a tile (every 32nd of n) are done.
  __device__ __forceinline__ void end_tile(const uint4 *tile, int n) {
    if (ts.finite() && tq.finite()) {
      join(ts, tq);
    } else {
      for (int i = (int)(threadIdx.x & 31); i < n; i += 32) {
        float cs, cq;
        chunk_sums(tile[i], cs, cq);
        s += (double)cs;
        q += (double)cq;
      }
    }
    ts = tq = Sum3();
  }
  // Lane 0: the warp's sums.
  __device__ __forceinline__ void warp_total(double &sum, double &sq) {
    Sum3 a = ps, b = pq;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      a.add(a.from(o));
      b.add(b.from(o));
    }
    const bool wide = __shfl_sync(0xffffffffu, !(a.finite() && b.finite()), 0);
    sum = wide ? 0.0 : a.value();
    sq = wide ? 0.0 : b.value();
    if (wide || __any_sync(0xffffffffu, s != 0.0 || q != 0.0)) {
      if (wide) {
        s += ps.value();
        q += pq.value();
      }
      for (int o = 16; o; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        q += __shfl_down_sync(0xffffffffu, q, o);
      }
      sum += s;
      sq += q;
    }
  }
};

// frac(x) as a u64 fraction of a cycle.
__device__ __forceinline__ unsigned long long fix_frac(double x) {
  const double f = x - floor(x);
  return __double2ull_rz(ldexp(f, 64));
}

// Phase anchors of every (channel, subint) in units of `unit` samples, at the
// unit that holds the subint's first sample: fx[0] phase, fx[1] cycles per sample
// there, fx[2] unit 1 - unit 0, fx[3] its change per unit, fx[4] the change of
// fx[1] per unit.  In a kernel of their own: one thread's f64 chain held a fold CTA
// for a fifth of its time.
__global__ void __launch_bounds__(CB_NT)
    k_cube_anchors(uint64_t n, int S, uint64_t nrows, double unit, double tsamp, double nu,
                   double nudot, const double *__restrict__ tau,
                   unsigned long long *__restrict__ anchors) {
  const uint64_t r = (uint64_t)blockIdx.x * CB_NT + threadIdx.x;
  if (r >= nrows) return;
  const uint64_t c = r / (uint64_t)S, s = r % (uint64_t)S;
  const uint64_t u0 = (n * s) / (uint64_t)S / (uint64_t)unit;
  const double td = (double)(u0 * (uint64_t)unit) * tsamp - tau[c];
  const double f = (nu + nudot * td) * tsamp, g = nudot * tsamp * tsamp;
  unsigned long long *fx = anchors + 5 * r;
  fx[0] = fix_frac(nu * td + 0.5 * nudot * td * td);
  fx[1] = fix_frac(f);
  fx[2] = fix_frac(unit * f + 0.5 * g * unit * unit);
  fx[3] = fix_frac(g * unit * unit);
  fx[4] = fix_frac(g * unit);
}

// Bin accumulators of one CTA.  PrivateBins: one column per thread,
// h[b * nt + tid] (bank = tid mod 32 for every b: no conflicts, no atomics),
// summed over threads at the end; for (B + 1) * threads <= CB_PRIV floats.
// SharedBins: one row updated with shared-memory atomics (large B).
constexpr int CB_PRIV = 8448;  // 33 KB: 64 threads at B = 128
// Both carry B + 1 rows: add2 puts a sample's second cloud-in-cell share in
// row b + 1 without wrapping, and row B is folded into row 0 at the end.
struct PrivateBins {
  float *h;  // this thread's column: h[b * nt]
  int nt;
  __device__ __forceinline__ void add(int b, float x) const { h[b * nt] += x; }
  __device__ __forceinline__ void add2(int b, float x0, float x1) const {
    float *p = h + b * nt;
    p[0] += x0;
    p[nt] += x1;
  }
};
struct SharedBins {
  float *h;
  __device__ __forceinline__ void add(int b, float x) const { atomicAdd(&h[b], x); }
  __device__ __forceinline__ void add2(int b, float x0, float x1) const {
    atomicAdd(&h[b], x0);
    atomicAdd(&h[b + 1], x1);
  }
};

template <class Bins>
__device__ __forceinline__ void flush_bins(const Bins &bins, int bin, int B, float a0, float a1) {
  bins.add(bin, a0 - a1);
  bins.add(bin + 1 == B ? 0 : bin + 1, a1);
}

// Open bin of a thread's walk: samples of bin `bin` summed so far (a0 = sum
// v, a1 = sum w v); bin < 0 when nothing is open.
struct OpenBin {
  int bin = -1;
  float a0 = 0.0f, a1 = 0.0f;
  template <class Bins>
  __device__ __forceinline__ void move_to(int b, const Bins &bins, int B) {
    if (b != bin) {
      if (bin >= 0) flush_bins(bins, bin, B, a0, a1);
      bin = b;
      a0 = a1 = 0.0f;
    }
  }
};

// du >= 1 bin per sample: every sample starts a new bin, so each goes
// straight to its two bins (the open bin, if any, is flushed first).
template <class T, class Bins>
__device__ __forceinline__ void scatter_run(const RunRegs<T> &x, float u, float du, int B,
                                            const Bins &bins, OpenBin &ob) {
  if (ob.bin >= 0) {
    flush_bins(bins, ob.bin, B, ob.a0, ob.a1);
    ob.bin = -1;
    ob.a0 = ob.a1 = 0.0f;
  }
  const float fB = (float)B;
#pragma unroll
  for (int i = 0; i < CB_RUN; ++i) {
    // 0 <= u < B here (u >= B is wrapped below and at run starts), so
    // floor(u) <= B - 1 and its second share lands in rows 1..B
    const float v = run_sample<T>(x, i);
    const float fl = floorf(u);
    const float wv = (u - fl) * v;
    bins.add2((int)fl, v - wv, wv);
    u += du;
    if (u >= fB) u -= fB;
  }
}

// Fold one run starting at bin position u (bins) advancing du per sample;
// the open bin carries over from the previous run of the same thread.
template <class T, class Bins>
__device__ __forceinline__ void fold_run(const RunRegs<T> &x, float u, float du, int B,
                                         const Bins &bins, OpenBin &ob, RunSums<T> &sums) {
  sums.add(x);
  if (du < 1.0f) {
    int b = (int)u;
    if (b >= B) b = 0, u = 0.0f;
    float w = u - (float)b;
    ob.move_to(b, bins, B);
#pragma unroll
    for (int i = 0; i < CB_RUN; ++i) {
      const float v = run_sample<T>(x, i);
      ob.a0 += v;
      ob.a1 = fmaf(w, v, ob.a1);
      w += du;
      if (w >= 1.0f) {
        flush_bins(bins, ob.bin, B, ob.a0, ob.a1);
        ob.bin = ob.bin + 1 == B ? 0 : ob.bin + 1;
        w -= 1.0f;
        ob.a0 = ob.a1 = 0.0f;
      }
    }
  } else {
    scatter_run(x, u, du, B, bins, ob);
  }
}

// 8-bit runs: a run that stays inside one bin (or crosses one bin edge) is
// folded from two integer sums instead of sample by sample.  With w_i = w0 +
// i du the run adds sum (1 - w_i) v_i and sum w_i v_i to bins b and b + 1,
// i.e. a0 += S and a1 += w0 S + du T with S = sum v_i, T = sum i v_i (dp4a
// over the packed bytes, exact); a run whose w reaches 1 at sample p is split
// there (byte-masked dp4a for the prefix).  Runs with more crossings (du >=
// 1/31 bins per sample) take the sample-by-sample walk.
__device__ __forceinline__ uint32_t prefix_mask(int p, int k) {
  const int cnt = min(max(p - 4 * k, 0), 4);
  return cnt == 0 ? 0u : (0xffffffffu >> (32 - 8 * cnt));
}

template <class Bins>
__device__ __forceinline__ void fold_run(const RunRegs<uint8_t> &x, float u, float du, int B,
                                         const Bins &bins, OpenBin &ob,
                                         RunSums<uint8_t> &sums) {
  // S = sum v, Q = sum v^2 (the channel statistics), T = sum i v.
  unsigned S = 0, Q = 0, T = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t wd = word_of(x.r[k >> 2], k & 3);
    S = __dp4a(wd, 0x01010101u, S);
    Q = __dp4a(wd, wd, Q);
    T = __dp4a(wd, 0x03020100u + 0x04040404u * (unsigned)k, T);
  }
  sums.s += S;
  sums.q += Q;
  int b = (int)u;
  if (b >= B) b = 0, u = 0.0f;
  const float w0 = u - (float)b;
  const float wend = fmaf(31.0f, du, w0);
  if (du < 1.0f && wend < 2.0f) {
    ob.move_to(b, bins, B);
    if (wend < 1.0f) {
      ob.a0 += (float)S;
      ob.a1 += fmaf(w0, (float)S, du * (float)T);
      return;
    }
    // first sample with w >= 1 (the walk's rule, with its f32 rounding)
    int p = min(max((int)ceilf((1.0f - w0) / du), 1), 31);
    if (fmaf((float)(p - 1), du, w0) >= 1.0f) --p;
    else if (fmaf((float)p, du, w0) < 1.0f) ++p;
    unsigned S1 = 0, T1 = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t wd = word_of(x.r[k >> 2], k & 3) & prefix_mask(p, k);
      S1 = __dp4a(wd, 0x01010101u, S1);
      T1 = __dp4a(wd, 0x03020100u + 0x04040404u * (unsigned)k, T1);
    }
    const float s1 = (float)S1, t1 = (float)T1, s2 = (float)(S - S1), t2 = (float)(T - T1);
    flush_bins(bins, ob.bin, B, ob.a0 + s1, ob.a1 + fmaf(w0, s1, du * t1));
    ob.bin = ob.bin + 1 == B ? 0 : ob.bin + 1;
    ob.a0 = s2;
    ob.a1 = fmaf(w0 - 1.0f, s2, du * t2);
    return;
  }
  // Sample-by-sample walk.
  if (du < 1.0f) {
    float w = w0;
    ob.move_to(b, bins, B);
#pragma unroll
    for (int i = 0; i < CB_RUN; ++i) {
      const float v = run_sample<uint8_t>(x, i);
      ob.a0 += v;
      ob.a1 = fmaf(w, v, ob.a1);
      w += du;
      if (w >= 1.0f) {
        flush_bins(bins, ob.bin, B, ob.a0, ob.a1);
        ob.bin = ob.bin + 1 == B ? 0 : ob.bin + 1;
        w -= 1.0f;
        ob.a0 = ob.a1 = 0.0f;
      }
    }
  } else {
    scatter_run(x, u, du, B, bins, ob);
  }
}

// PRIV: per-thread bin columns in dynamic shared memory (B * blockDim.x
// floats); otherwise one shared row with atomics.  blockDim.x is a multiple
// of 32, at most CB_NT.
template <class T, bool PRIV>
__global__ void __launch_bounds__(CB_NT)
    k_cube_fold(const T *__restrict__ x, uint64_t ld, uint64_t n, int S, int B,
                const unsigned long long *__restrict__ anchors, float *__restrict__ cube, double *__restrict__ chsum) {
  extern __shared__ float hist[];
  __shared__ unsigned long long fx[5];
  __shared__ double red[2][CB_NT / 32];
  __shared__ float mean_s;
  const int nt = (int)blockDim.x, tid = (int)threadIdx.x;
  const int s = blockIdx.x;
  const uint64_t c = blockIdx.y;
  const int hn = PRIV ? (B + 1) * nt : B + 1;
  for (int i = tid; i < hn; i += nt) hist[i] = 0.0f;
  const uint64_t t0 = (n * (uint64_t)s) / (uint64_t)S, t1 = (n * (uint64_t)(s + 1)) / (uint64_t)S;
  const uint64_t rlo = t0 / CB_RUN, rhi = (t1 + CB_RUN - 1) / CB_RUN;  // runs [rlo, rhi)
  if (tid < 5) fx[tid] = anchors[5 * (c * (uint64_t)S + (uint64_t)s) + tid];
  __syncthreads();
  // Thread j folds the contiguous runs [rlo + j q, rlo + (j + 1) q) so that
  // the open bin carries from run to run.  Phase at run m (from rlo):
  // P0 + m d1 + m (m - 1) / 2 d2, exact modulo 1.
  const uint64_t q = (rhi - rlo + nt - 1) / nt;
  const unsigned long long m = (unsigned long long)tid * q;
  unsigned long long P = fx[0] + m * fx[2] + (m * (m - 1) / 2) * fx[3];
  unsigned long long A = fx[2] + m * fx[3];
  unsigned long long F = fx[1] + m * fx[4];
  const unsigned long long D2 = fx[3], G = fx[4];
  const float Bs = (float)B * 5.42101086242752217e-20f;  // B 2^-64
  const float fB = (float)B;
  const T *row = x + c * ld;
  typename std::conditional<PRIV, PrivateBins, SharedBins>::type bins;
  if constexpr (PRIV) bins = PrivateBins{hist + tid, nt};
  else bins = SharedBins{hist};
  RunSums<T> sums;
  OpenBin ob;
  const uint64_t r0 = rlo + m;
  const int cnt = r0 < rhi ? (int)(min(r0 + q, rhi) - r0) : 0;
  // Only the subint's first and last runs can hold samples outside [t0, t1).
  const int lo0 = (int)(t0 - rlo * CB_RUN), hi1 = (int)(t1 - (rhi - 1) * CB_RUN);
  const bool has_first = r0 == rlo, has_last = r0 + (uint64_t)cnt == rhi;
  const T *src = row + r0 * CB_RUN;
  RunRegs<T> cur, nxt;
  if (cnt > 0) load_run(src, cur);
  for (int i = 0; i < cnt; ++i) {
    if (i + 1 < cnt) load_run(src + (i + 1) * CB_RUN, nxt);
    if ((has_first && i == 0 && lo0 != 0) || (has_last && i == cnt - 1 && hi1 != CB_RUN))
      mask_run(cur, (has_first && i == 0) ? lo0 : 0, (has_last && i == cnt - 1) ? hi1 : CB_RUN);
    float u = __ull2float_rn(P) * Bs;
    if (u >= fB) u -= fB;
    fold_run(cur, u, __ull2float_rn(F) * Bs, B, bins, ob, sums);
    P += A;
    A += D2;
    F += G;
    cur = nxt;
  }
  if (ob.bin >= 0) flush_bins(bins, ob.bin, B, ob.a0, ob.a1);
  double sum, sq;
  sums.warp_total(sum, sq);
  if ((tid & 31) == 0) {
    red[0][tid >> 5] = sum;
    red[1][tid >> 5] = sq;
  }
  __syncthreads();
  if (tid < 2) {
    double a = 0.0;
    for (int w2 = 0; w2 < nt / 32; ++w2) a += red[tid][w2];
    chsum[(c * (uint64_t)S + (uint64_t)s) * 2 + tid] = a;
    if (tid == 0) mean_s = (float)(B & (B - 1) ? a / (double)B : a * (1.0 / (double)B));
  }
  __syncthreads();
  float *dst = cube + (c * (uint64_t)S + (uint64_t)s) * (uint64_t)B;
  for (int b = tid; b < B; b += nt) {
    float v;
    if constexpr (PRIV) {
      // row sums (row B joins row 0), skewed by the thread index so that a
      // warp's reads of 32 consecutive rows fall in 32 different banks
      v = 0.0f;
      for (int r = b; r <= B; r += B) {
        const float *hb = hist + r * nt;
        for (int t = 0; t < nt; ++t) {
          int k = t + tid;
          if (k >= nt) k -= nt;
          v += hb[k];
        }
        if (b != 0) break;
      }
    } else {
      v = hist[b] + (b == 0 ? hist[B] : 0.0f);
    }
    dst[b] = v - mean_s;
  }
}

// A sample as f32 (integers exactly, without the conversion pipe).
__device__ __forceinline__ float sample_float(float v) { return v; }
__device__ __forceinline__ float sample_float(unsigned v) {
  return __fsub_rn(__uint_as_float(0x4B000000u + v), 8388608.0f);
}

// Bin-owner fold for 1/31 <= du < 1 bins per sample (each bin holds 1 to 31
// consecutive samples per period).  Each warp stages tiles of CB_TL samples
// of the subint in shared memory; lane l owns bins l, l + 32, ... < B and,
// for every unwrapped bin index m = b + k B that the tile's phase range
// crosses, gathers the samples i in [Q(m), Q(m + 1)), Q(m) = ceil((m - ua) /
// du) clamped to the tile (ua = bin position of the tile's first sample, the
// phase linear across the tile).  Adjacent bins use the same Q, so every
// sample is counted once.  The lane keeps S_b = sum v and T_b = sum (u - m) v
// in registers; at the end bin b of the cloud-in-cell fold is S_b - T_b +
// T_(b-1).  No atomics, no per-sample branches: an interval is read four
// samples at a time, those past its end as zeros.
// One warp per tile up to 16 tiles (a subint of 16,384 samples touches 9: with 8
// warps, seven of them waited for the one with two tiles), 8 warps above; the
// warps' sums go into their own tiles' memory, so that three CTAs fit an SM.
// Bound: issue; conversions and ceilings, on the quarter-rate pipe, are done by
// sums at 2^23.  Measured on a GB300, 256 channels of 1,048,576 f32 samples, 0.3
// bins per sample: 1.05 ms before, 0.57 now (0.16 for the bytes; 0.50 with channel
// sums in f32 pairs, which are fewer bits than f64).
constexpr int CB_TL = 2048;
constexpr int CB_BO_MAXB = 256;
constexpr int CB_BO_NB = CB_BO_MAXB / 32;
constexpr int CB_BO_SLOTS = 8;   // tile i adds to the sums of slot i mod 8
constexpr int CB_BO_WARPS = 16;  // warps of a CTA, at most
// ceil(x) for |x| < 2^22
__device__ __forceinline__ int ceil_int(float x) {
  return (int)__float_as_uint(__fadd_ru(x, 12582912.0f)) - 0x4B400000;
}
// (float)i for 0 <= i < 2^23
__device__ __forceinline__ float float_of(int i) {
  return __fsub_rn(__uint_as_float(0x4B000000u + (unsigned)i), 8388608.0f);
}

template <class T>
__global__ void __launch_bounds__(32 * CB_BO_WARPS)
    k_cube_fold_bo(const T *__restrict__ x, uint64_t ld, uint64_t n, int S, int B,
                   const unsigned long long *__restrict__ anchors, float *__restrict__ cube, double *__restrict__ chsum) {
  extern __shared__ __align__(16) unsigned char smem_bo[];
  T *tiles = reinterpret_cast<T *>(smem_bo);  // [warp][CB_TL], then [warp][S, T][B]
  static_assert(2 * CB_BO_MAXB * 4 <= CB_TL, "a warp's sums fit its tile");
  auto sums_of = [&](int w) { return reinterpret_cast<float *>(tiles + (size_t)w * CB_TL); };
  __shared__ unsigned long long fx[5];
  __shared__ double red[2][CB_BO_WARPS];
  __shared__ float mean_s;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = (int)blockDim.x >> 5;
  const int s = blockIdx.x;
  const uint64_t c = blockIdx.y;
  const uint64_t t0 = (n * (uint64_t)s) / (uint64_t)S, t1 = (n * (uint64_t)(s + 1)) / (uint64_t)S;
  const uint64_t k0 = t0 / CB_TL, k1 = (t1 + CB_TL - 1) / CB_TL;  // tiles [k0, k1)
  if (tid < 5) fx[tid] = anchors[5 * (c * (uint64_t)S + (uint64_t)s) + tid];
  __syncthreads();
  const float Bs = (float)B * 5.42101086242752217e-20f;  // B 2^-64
  const float fB = (float)B;
  const T *row = x + c * ld;
  T *tile = tiles + (size_t)warp * CB_TL;
  float Sb[CB_BO_NB], Tb[CB_BO_NB];
#pragma unroll
  for (int j = 0; j < CB_BO_NB; ++j) Sb[j] = Tb[j] = 0.0f;
  RunSums<T> sums;
  constexpr int PER = 16 / (int)sizeof(T);  // samples per 16-byte chunk
  for (uint64_t k = k0 + warp; k < k1; k += nw) {
    const uint64_t ta = k * CB_TL;
    if (ta >= t0 && ta + CB_TL <= t1) {
      const uint4 *src = reinterpret_cast<const uint4 *>(row + ta);
#pragma unroll 8
      for (int q = lane; q < CB_TL / PER; q += 32) {
        const uint4 v = __ldg(src + q);
        reinterpret_cast<uint4 *>(tile)[q] = v;
        sums.add_chunk(v);
      }
    } else
    // Stage the tile (chunks wholly outside [t0, t1) are not loaded).
    for (int q = lane; q < CB_TL / PER; q += 32) {
      const uint64_t cs = ta + (uint64_t)q * PER;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (cs < t1 && cs + PER > t0) {
        v = __ldg(reinterpret_cast<const uint4 *>(row + cs));
        if (cs < t0 || cs + PER > t1) {  // mask samples outside [t0, t1)
          T e[PER];
          memcpy(e, &v, 16);
#pragma unroll
          for (int u = 0; u < PER; ++u)
            if (cs + u < t0 || cs + u >= t1) e[u] = (T)0;
          memcpy(&v, e, 16);
        }
      }
      reinterpret_cast<uint4 *>(tile)[q] = v;
      sums.add_chunk(v);
    }
    sums.end_tile(reinterpret_cast<const uint4 *>(tile), CB_TL / PER);
    __syncwarp();
    // Phase of the tile: fixed-point at its first sample, linear across it.
    const unsigned long long kk = k - k0;
    const unsigned long long P = fx[0] + kk * fx[2] + (kk * (kk - 1) / 2) * fx[3];
    const unsigned long long F = fx[1] + kk * fx[4];
    float ua = __ull2float_rn(P) * Bs;
    if (ua >= fB) ua -= fB;
    // (a tile's du only departs from the launch's nominal 1/31..1 through
    // nudot; the floor keeps the partition finite)
    const float du = fmaxf(__ull2float_rn(F) * Bs, 1e-3f);
    const float inv = 1.0f / du;
    const float uend = fmaf((float)CB_TL, du, ua);  // unwrapped phase past the tile
    // an interval of 1/du holds at most floor(1/du) + 1 samples; one more
    // covers the rounding of Q
    const int cmax = (int)inv + 2;
    const int mfirst = (int)ua;  // bin of the tile's first sample
#pragma unroll
    for (int j = 0; j < CB_BO_NB; ++j) {
      const int b = lane + 32 * j;
      if (b >= B) break;
      // first unwrapped m = b + k B >= mfirst (0 <= mfirst < B)
      float m = float_of(b >= mfirst ? b : b + B);
      float sj = 0.0f, tj = 0.0f;
      for (; m < uend; m += fB) {
        const int i0 = max(0, ceil_int((m - ua) * inv));
        const int i1 = min(CB_TL, ceil_int(((m + 1.0f) - ua) * inv));
        // sum v and sum (i - i0) v of the bin's samples, then its weights
        // w_i = w_0 + (i - i0) du, w_0 = ua + i0 du - m
        const T *p = tile + i0;
        const int len = i1 - i0;
        float sl = 0.0f, il = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float v = e < len ? sample_float(std::conditional_t<std::is_same<T, float>::value, float, unsigned>(p[e])) : 0.0f;
          sl += v;
          il = fmaf((float)e, v, il);
        }
        for (int q = 4; q < cmax; q += 4) {
          const float fq = float_of(q);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float v = q + e < len ? sample_float(std::conditional_t<std::is_same<T, float>::value, float, unsigned>(p[q + e])) : 0.0f;
            sl += v;
            il = fmaf(fq + (float)e, v, il);
          }
        }
        sj += sl;
        tj = fmaf(fmaf(float_of(i0), du, ua) - m, sl, fmaf(du, il, tj));
      }
      Sb[j] += sj;
      Tb[j] += tj;
    }
    __syncwarp();
  }
  // Per-warp bin sums into the warp's own tile, then across warps.
#pragma unroll
  for (int j = 0; j < CB_BO_NB; ++j) {
    const int b = lane + 32 * j;
    if (b < B) {
      sums_of(warp)[b] = Sb[j];
      sums_of(warp)[B + b] = Tb[j];
    }
  }
  double sum, sq;
  sums.warp_total(sum, sq);
  if (lane == 0) {
    red[0][warp] = sum;
    red[1][warp] = sq;
  }
  __syncthreads();
  if (tid < 2) {
    double a = 0.0;
    for (int w2 = 0; w2 < nw; ++w2) a += red[tid][w2];
    chsum[(c * (uint64_t)S + (uint64_t)s) * 2 + tid] = a;
    if (tid == 0) mean_s = (float)(B & (B - 1) ? a / (double)B : a * (1.0 / (double)B));
  }
  __syncthreads();
  float *dst = cube + (c * (uint64_t)S + (uint64_t)s) * (uint64_t)B;
  for (int b = tid; b < B; b += nw * 32) {
    const int bp = b == 0 ? B - 1 : b - 1;
    // slot w holds the sums of tiles w and w + 8 (of every eighth with 8 warps)
    auto slot = [&](int w, int i) {
      const float x = sums_of(w)[i];
      return w + CB_BO_SLOTS < nw ? x + sums_of(w + CB_BO_SLOTS)[i] : x;
    };
    float sb = 0.0f, tb = 0.0f, tp = 0.0f;
    for (int w2 = 0; w2 < min(nw, CB_BO_SLOTS); ++w2) {
      sb += slot(w2, b);
      tb += slot(w2, B + b);
      tp += slot(w2, B + bp);
    }
    dst[b] = sb - tb + tp - mean_s;
  }
}

// Threads per fold CTA for B bins: private columns when (B + 1) * threads fits
// CB_PRIV floats with at least 32 threads.
int cube_fold_threads(int B, bool &priv) {
  int nt = (CB_PRIV / (B + 1)) / 32 * 32;
  priv = nt >= 32;
  return priv ? std::min(nt, CB_NT) : CB_NT;
}

// du = bins per sample at the reference: the bin-owner gather for 1/31 <= du
// < 1 (B <= 256), otherwise runs (analytic for 8-bit data at du < 1/31,
// walked or scattered otherwise).
template <class T>
int launch_cube_fold(dim3 grid, int B, cudaStream_t st, const T *x, uint64_t ld, uint64_t n,
                     int S, double tsamp, double nu, double nudot, const double *tau,
                     unsigned long long *anchors, float *cube, double *chsum) {
  const double du = nu * tsamp * (double)B;
  const bool owner = du >= 1.0 / 31.0 && du < 1.0 && B <= CB_BO_MAXB;
  const uint64_t nrows = (uint64_t)grid.x * grid.y;
  k_cube_anchors<<<(unsigned)((nrows + CB_NT - 1) / CB_NT), CB_NT, 0, st>>>(
      n, S, nrows, owner ? (double)CB_TL : (double)CB_RUN, tsamp, nu, nudot, tau, anchors);
  if (owner) {
    // tiles that a subint's samples can touch
    const uint64_t tiles = ((n + S - 1) / S + CB_TL - 2) / CB_TL + 1;
    const int nw = tiles <= CB_BO_WARPS ? (int)tiles : CB_BO_SLOTS;
    const size_t sm = (size_t)nw * CB_TL * sizeof(T);
    PSR_CUDA(cudaFuncSetAttribute(k_cube_fold_bo<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    k_cube_fold_bo<T><<<grid, nw * 32, sm, st>>>(x, ld, n, S, B, anchors, cube, chsum);
    return PSR_OK;
  }
  // Below 1/31 bins per sample runs rarely change bin: one shared row with
  // 256 threads; above 1 every sample changes bin: private columns.
  bool priv = false;
  const int nt = du < 1.0 ? CB_NT : cube_fold_threads(B, priv);
  if (priv)
    k_cube_fold<T, true><<<grid, nt, (size_t)(B + 1) * nt * 4, st>>>(
        x, ld, n, S, B, anchors, cube, chsum);
  else
    k_cube_fold<T, false><<<grid, nt, (size_t)(B + 1) * 4, st>>>(x, ld, n, S, B, anchors, cube,
                                                                chsum);
  return PSR_OK;
}

struct CandDev {
  double nu, nudot, dm;
};
// The candidates of a launch, as a kernel argument.
constexpr int CB_CANDS = 64;
struct CandBatch {
  CandDev c[CB_CANDS];
};

// x - floor(x) for 0 <= x < 2^23, the floor by a sum rounded down at 2^23 (floorf
// runs on the quarter-rate pipe).
__device__ __forceinline__ float frac_pos(float x) {
  return x - __fsub_rn(__fadd_rd(x, 8388608.0f), 8388608.0f);
}

__device__ __forceinline__ double row_time(uint32_t r, int S, double Tsub) {
  return ((double)(r % (uint32_t)S) + 0.5) * Tsub;  // T_s of row r = (channel, subint s)
}

// ref[r] = phase of row r at the reference (cycles), T_s - tau_c(DM_ref).
__global__ void __launch_bounds__(CB_NT)
    k_cube_ref(uint32_t rows, int S, const double *__restrict__ kc, double Tsub, double nu_r,
               double nudot_r, double dm_r, double *__restrict__ ref) {
  const uint32_t r = blockIdx.x * CB_NT + threadIdx.x;
  if (r >= rows) return;
  const double tdr = row_time(r, S, Tsub) - kc[r / (uint32_t)S] * dm_r;
  ref[r] = nu_r * tdr + 0.5 * nudot_r * tdr * tdr;
}

// R[r][k-1] = sum_b C[r][b] e^(-2 pi i k b / B), k = 1..B/2; one CTA per
// CB_ROWS rows, twiddles from a shared table.  A thread takes one harmonic of
// four rows, so that a twiddle (gathered, with bank conflicts) is read once for
// them.  With one thread per (row, harmonic), a row at a time: 16,384 rows of 64
// harmonics 101 us; 41 now.
constexpr int CB_ROWS = 32;
// Rows staged at a time: 16 KB of shared memory, a multiple of 4.
__host__ __device__ inline int cube_dft_group(int B) {
  const int g = 4096 / B & ~3;
  return g < 4 ? 4 : (g > CB_ROWS ? CB_ROWS : g);
}
__global__ void __launch_bounds__(CB_NT)
    k_cube_dft(const float *__restrict__ cube, uint64_t rows, int B, float2 *__restrict__ R) {
  __shared__ float2 tw[CB_MAXB];
  extern __shared__ __align__(16) float row[];  // [rows of a group][B], zeros past the last row
  for (int m = threadIdx.x; m < B; m += blockDim.x) {
    float sn, cs;
    sincospif(-2.0f * (float)m / (float)B, &sn, &cs);
    tw[m] = make_float2(cs, sn);
  }
  const int K = B / 2;
  const int group = cube_dft_group(B);
  const uint64_t r1 = min((uint64_t)(blockIdx.x + 1) * CB_ROWS, rows);
  for (uint64_t r = (uint64_t)blockIdx.x * CB_ROWS; r < r1; r += group) {
    const int nr = (int)min((uint64_t)group, r1 - r);
    __syncthreads();
    for (int i = threadIdx.x; i < group * B; i += blockDim.x)
      row[i] = i < nr * B ? cube[r * (uint64_t)B + i] : 0.0f;
    __syncthreads();
    for (int i = threadIdx.x; i < (nr + 3) / 4 * K; i += blockDim.x) {
      const int g = i / K, k = i - g * K + 1;
      const float *x = row + 4 * g * B;
      float re[4], im[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) re[j] = im[j] = 0.0f;
      int m = 0;
#pragma unroll 4
      for (int b = 0; b < B; ++b) {
        const float2 w = tw[m];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          re[j] += x[j * B + b] * w.x;
          im[j] += x[j * B + b] * w.y;
        }
        m += k;
        if (m >= B) m -= B;
      }
      for (int j = 0; j < min(4, nr - 4 * g); ++j)
        R[(r + 4 * g + j) * (uint64_t)K + (k - 1)] = make_float2(re[j], im[j]);
    }
  }
}

// P[cand][k]: CTA (256 rows, candidate).  The CTA first computes its rows'
// shifts (the only f64 work: about 16 operations per row and candidate, the
// reference's phase coming from k_cube_ref; the gradient reads them back
// from dsh), then takes sub-blocks of rows: every thread turns (row, harmonic)
// entries by their phase into shared memory, one thread per harmonic component
// adds a sub-block in row order, and one f64 atomic per component ends the CTA.
// Bound: issue, about 65 instructions per entry, most of them sincospif's.
// With one thread per harmonic walking the 256 rows, and the phases of both
// ends computed in f64 per row and candidate here and again in the gradient,
// the 22 evaluations of a group of 16 (16,384 rows of 64 harmonics) took 0.77 ms
// here and 0.95 in the gradient; 0.64 and 0.65 now.  Two candidates per CTA
// read R half as often and issue a sixth less, but left the SMs at 27 warps:
// 0.76 and 0.80.
constexpr int CB_HROWS = CB_NT;  // rows per CTA
constexpr int CB_HITEMS = 2048;  // (row, harmonic) entries of a sub-block
__global__ void __launch_bounds__(CB_NT, 8)
    k_cube_harmonics(const float2 *__restrict__ R, uint32_t rows, int S, int B,
                     const double *__restrict__ kc, const double *__restrict__ ref, double Tsub,
                     const __grid_constant__ CandBatch cands, float *__restrict__ dsh,
                     double *__restrict__ P) {
  __shared__ float d[CB_HROWS];  // shift / B, reduced to [0, 1)
  __shared__ float2 z[CB_HITEMS];
  constexpr int ACC = CB_MAXB / CB_NT;  // components per thread
  const int tid = (int)threadIdx.x;
  const int cand = (int)blockIdx.y;
  const uint32_t K = (uint32_t)B / 2;
  const uint32_t r0 = blockIdx.x * CB_HROWS;
  const int nr = (int)min((uint32_t)CB_HROWS, rows - r0);
  if (tid < nr) {
    const uint32_t r = r0 + (uint32_t)tid;
    const CandDev q = cands.c[cand];
    const double tdq = row_time(r, S, Tsub) - kc[r / (uint32_t)S] * q.dm;
    double x = q.nu * tdq + 0.5 * q.nudot * tdq * tdq - ref[r];
    // shift in bins over B: the two roundings cancel at powers of two
    if (B & (B - 1)) x = x * (double)B / (double)B;
    const float f = (float)(x - floor(x));
    d[tid] = f;
    dsh[(uint64_t)cand * rows + r] = f;
  }
  float acc[ACC];
#pragma unroll
  for (int j = 0; j < ACC; ++j) acc[j] = 0.0f;
  const int RB = (int)min((uint32_t)CB_HITEMS / K, (uint32_t)CB_HROWS);
  // idx / K = idx * inv >> 20 exactly for idx < 2048, 2 <= K <= 512
  const uint32_t inv = ((1u << 20) + K - 1) / K;
  const int comps = 2 * (int)K;
  __syncthreads();
  for (int i0 = 0; i0 < nr; i0 += RB) {
    const int m = min(RB, nr - i0), items = m * (int)K;
    const float2 *src = R + (uint64_t)(r0 + (uint32_t)i0) * K;
#pragma unroll 1  // (unrolled four times: 0.71 ms)
    for (int idx = tid; idx < items; idx += CB_NT) {
      const int row = (int)((uint32_t)idx * inv >> 20);
      const float h = (float)(idx - row * (int)K + 1);
      const float2 v = src[idx];
      // e^(-2 pi i h d) with h d reduced mod 1 in f32
      const float x = frac_pos(h * d[i0 + row]);
      float sn, cs;
      sincospif(-2.0f * x, &sn, &cs);
      z[idx] = make_float2(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ACC; ++j) {
      const int t = tid + j * CB_NT;
      if (t >= comps) break;
      const float *p = reinterpret_cast<const float *>(z) + t;
#pragma unroll 8
      for (int i = 0; i < m; ++i) acc[j] += p[(uint32_t)i * 2 * K];
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < ACC; ++j) {
    const int t = tid + j * CB_NT;
    if (t >= comps) break;
    atomicAdd(&P[(uint64_t)cand * 2 * K + t], (double)acc[j]);
  }
}

// A[cand][h - 1] = 2 w_h conj(P_h) / (B n v).
__global__ void __launch_bounds__(CB_NT)
    k_cube_coefficients(const double *__restrict__ P, int K, int entries, double norm,
                        float2 *__restrict__ A) {
  const int i = (int)(blockIdx.x * CB_NT + threadIdx.x);
  if (i >= entries) return;
  const double wk = i % K + 1 < K ? 2.0 : 1.0;
  A[i] = make_float2((float)(2.0 * wk * P[2 * i] / norm), (float)(-2.0 * wk * P[2 * i + 1] / norm));
}

// Gradient: a warp takes 32 rows of a candidate; the lanes split each row's
// harmonics, then lane l adds row l's 32 partial sums (as the tree over lane
// distances 16, 8, 4, 2, 1) and does its f64 terms.
constexpr int CB_GNT = 128;
__global__ void __launch_bounds__(CB_GNT)
    k_cube_grad(const float2 *__restrict__ R, uint32_t rows, int S, int B,
                const double *__restrict__ kc, double Tsub, const float *__restrict__ dsh,
                const __grid_constant__ CandBatch cands, const float2 *__restrict__ A,
                double *__restrict__ grad) {
  __shared__ float part[CB_GNT / 32][32][33];
  __shared__ double red[3][CB_GNT / 32];
  const int cand = (int)blockIdx.y;
  const int K = B / 2;
  const float2 *Ak = A + (uint64_t)cand * K;
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const float twopi_b = 6.283185307179586f / (float)B;
  const uint32_t r0 = (blockIdx.x * (CB_GNT / 32) + warp) * 32;
  const int nr = r0 < rows ? (int)min(32u, rows - r0) : 0;
  const float dl = lane < nr ? dsh[(uint64_t)cand * rows + r0 + lane] : 0.0f;
#pragma unroll 2
  for (int i = 0; i < nr; ++i) {
    const float2 *Rr = R + (uint64_t)(r0 + i) * K;
    const float d = __shfl_sync(0xffffffffu, dl, i);
    float g = 0.0f;
    for (int h = lane + 1; h <= K; h += 32) {
      const float2 v = Rr[h - 1];
      const float x = frac_pos((float)h * d);
      float sn, cs;
      sincospif(-2.0f * x, &sn, &cs);
      // z = R e^(-2 pi i h d) (-2 pi i h / B); contribution Re(A_h z)
      const float zr = v.x * cs - v.y * sn, zi = v.x * sn + v.y * cs;
      const float f = twopi_b * (float)h;
      const float2 a = Ak[h - 1];
      g += a.x * (zi * f) - a.y * (-zr * f);
    }
    part[warp][i][lane] = g;
  }
  __syncwarp();
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  if (lane < nr) {
    const float *p = part[warp][lane];
    float t[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) t[j] = p[j] + p[j + 16];
#pragma unroll
    for (int o = 8; o; o >>= 1)
#pragma unroll
      for (int j = 0; j < o; ++j) t[j] = t[j] + t[j + o];
    const uint32_t r = r0 + (uint32_t)lane;
    const CandDev q = cands.c[cand];
    const double kcc = kc[r / (uint32_t)S], tdq = row_time(r, S, Tsub) - kcc * q.dm;
    const double Bd = (double)B, gg = (double)t[0];
    a0 = gg * Bd * tdq;
    a1 = gg * Bd * 0.5 * tdq * tdq;
    a2 = gg * (-Bd * (q.nu + q.nudot * tdq) * kcc);
  }
  for (int o = 16; o; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
  }
  if (lane == 0) {
    red[0][warp] = a0;
    red[1][warp] = a1;
    red[2][warp] = a2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double x = 0.0;
    for (int w = 0; w < CB_GNT / 32; ++w) x += red[threadIdx.x][w];
    atomicAdd(&grad[(uint64_t)cand * 3 + threadIdx.x], x);
  }
}

// v = sum over channels of each channel's sample variance (the variance of a
// sum of independent channels), from the per-(channel, subint) sums.
__global__ void __launch_bounds__(CB_NT)
    k_cube_var(const double *__restrict__ chsum, uint64_t nch, int S, uint64_t n,
               double *__restrict__ out) {
  __shared__ double red[CB_NT / 32];
  double v = 0.0;
  for (uint64_t c = threadIdx.x; c < nch; c += CB_NT) {
    double s1 = 0.0, s2 = 0.0;
#pragma unroll 8
    for (int s = 0; s < S; ++s) {
      s1 += chsum[(c * S + s) * 2];
      s2 += chsum[(c * S + s) * 2 + 1];
    }
    const double m = s1 / (double)n;
    v += fmax(s2 / (double)n - m * m, 0.0);
  }
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int w = 0; w < CB_NT / 32; ++w) a += red[w];
    out[0] = a;
  }
}

int build_cube(const DeviceObs &o, uint64_t n, int S, int B, double nu, double nudot, double dm,
               CubeWork &w, cudaStream_t st) {
  const uint64_t nch = o.nch;
  double fmax = 0.0;
  for (uint64_t c = 0; c < nch; ++c) fmax = std::fmax(fmax, o.h.fch1 + (double)c * o.h.foff);
  std::vector<double> kc(nch), tau(nch);
  for (uint64_t c = 0; c < nch; ++c) {
    const double f = o.h.fch1 + (double)c * o.h.foff;
    kc[c] = K_DM_C * (1.0 / (f * f) - 1.0 / (fmax * fmax));
    tau[c] = kc[c] * dm;
  }
  w.rows = nch * (uint64_t)S;
  PSR_TRY(w.cube.ensure(w.rows * B * 4));
  PSR_TRY(w.chsum.ensure(w.rows * 2 * 8));
  PSR_TRY(w.tau.ensure(nch * 8));
  PSR_TRY(w.kc.ensure(nch * 8));
  PSR_CUDA(cudaMemcpyAsync(w.tau.p, tau.data(), nch * 8, cudaMemcpyHostToDevice, st));
  PSR_CUDA(cudaMemcpyAsync(w.kc.p, kc.data(), nch * 8, cudaMemcpyHostToDevice, st));
  dim3 grid((unsigned)S, (unsigned)nch);
  PSR_TRY(w.anchors.ensure(w.rows * 5 * 8));
  unsigned long long *ap = w.anchors.as<unsigned long long>();
  const double *tp = w.tau.as<double>();
  float *cp = w.cube.as<float>();
  double *sp = w.chsum.as<double>();
  switch (o.kind) {
    case SAMPLE_U8:
      PSR_TRY(launch_cube_fold(grid, B, st, o.samples.as<uint8_t>(), o.ld, n, S, o.h.tsamp, nu,
                               nudot, tp, ap, cp, sp));
      break;
    case SAMPLE_U16:
      PSR_TRY(launch_cube_fold(grid, B, st, o.samples.as<uint16_t>(), o.ld, n, S, o.h.tsamp, nu,
                               nudot, tp, ap, cp, sp));
      break;
    default:
      PSR_TRY(launch_cube_fold(grid, B, st, o.samples.as<float>(), o.ld, n, S, o.h.tsamp, nu,
                               nudot, tp, ap, cp, sp));
  }
  PSR_CUDA(cudaGetLastError());
  PSR_TRY(w.R.ensure(w.rows * (uint64_t)(B / 2) * sizeof(float2)));
  k_cube_dft<<<(unsigned)((w.rows + CB_ROWS - 1) / CB_ROWS), CB_NT,
               (size_t)cube_dft_group(B) * B * 4, st>>>(
      w.cube.as<float>(), w.rows, B, w.R.as<float2>());
  PSR_CUDA(cudaGetLastError());
  const double Tsub = (double)n * o.h.tsamp / (double)S;
  PSR_TRY(w.ref.ensure(w.rows * 8));
  k_cube_ref<<<(unsigned)((w.rows + CB_NT - 1) / CB_NT), CB_NT, 0, st>>>(
      (uint32_t)w.rows, S, w.kc.as<double>(), Tsub, nu, nudot, dm, w.ref.as<double>());
  PSR_TRY(w.prof.ensure(16));
  k_cube_var<<<1, CB_NT, 0, st>>>(w.chsum.as<double>(), nch, S, n, w.prof.as<double>());
  PSR_CUDA(cudaGetLastError());
  double v = 0.0;
  PSR_CUDA(cudaMemcpyAsync(&v, w.prof.p, 8, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  w.var = v > 0.0 ? v : 1.0;
  return PSR_OK;
}

// J and gradient (in nu, nudot, DM) of every candidate, relative to the
// reference that the cube was built at.  P and the gradients come back in one
// copy.
int eval_cube(const DeviceObs &o, uint64_t n, int S, int B, const std::vector<CandDev> &cand,
              CubeWork &w, std::vector<double> &J, std::vector<double> &grad, cudaStream_t st) {
  const size_t K = cand.size();
  const int H = B / 2;
  const double Tsub = (double)n * o.h.tsamp / (double)S;
  const uint32_t rows = (uint32_t)w.rows;
  const size_t np = K * H * 2, nout = np + K * 3;
  const double norm = (double)B * (double)n * w.var;
  PSR_TRY(w.prof.ensure(nout * 8));
  PSR_TRY(w.g.ensure(std::min<size_t>(K, CB_CANDS) * H * sizeof(float2)));
  PSR_TRY(w.dsh.ensure(std::min<size_t>(K, CB_CANDS) * w.rows * 4));
  PSR_CUDA(cudaMemsetAsync(w.prof.p, 0, nout * 8, st));
  for (size_t c0 = 0; c0 < K; c0 += CB_CANDS) {
    const int nc = (int)std::min<size_t>(CB_CANDS, K - c0);
    CandBatch cb{};
    std::copy_n(cand.begin() + c0, nc, cb.c);
    double *P = w.prof.as<double>() + c0 * H * 2;
    const unsigned gy = (unsigned)nc;
    k_cube_harmonics<<<dim3((rows + CB_HROWS - 1) / CB_HROWS, gy), CB_NT, 0, st>>>(
        w.R.as<float2>(), rows, S, B, w.kc.as<double>(), w.ref.as<double>(), Tsub, cb,
        w.dsh.as<float>(), P);
    k_cube_coefficients<<<(unsigned)((nc * H + CB_NT - 1) / CB_NT), CB_NT, 0, st>>>(
        P, H, nc * H, norm, w.g.as<float2>());
    k_cube_grad<<<dim3((rows + CB_GNT - 1) / CB_GNT, gy), CB_GNT, 0, st>>>(
        w.R.as<float2>(), rows, S, B, w.kc.as<double>(), Tsub, w.dsh.as<float>(), cb,
        w.g.as<float2>(), w.prof.as<double>() + np + c0 * 3);
    PSR_CUDA(cudaGetLastError());
  }
  std::vector<double> out(nout);
  PSR_CUDA(cudaMemcpyAsync(out.data(), w.prof.p, nout * 8, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  J.assign(K, 0.0);
  for (size_t k = 0; k < K; ++k) {
    double j = 0.0;
    for (int h = 1; h <= H; ++h) {
      const double re = out[(k * H + h - 1) * 2], im = out[(k * H + h - 1) * 2 + 1];
      j += (h < H ? 2.0 : 1.0) * (re * re + im * im);
    }
    J[k] = j / norm;
  }
  grad.assign(out.begin() + np, out.end());
  return PSR_OK;
}

// Per-candidate quasi-Newton state (ascent on J in scaled coordinates).
struct Opt {
  double q[3] = {0, 0, 0}, g[3] = {0, 0, 0}, d[3] = {0, 0, 0}, qn[3] = {0, 0, 0};
  double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  double J = 0.0, slope = 0.0, alpha = 1.0, h0 = 1.0;
  int ls = 0;
  bool started = false, done = false;
  uint64_t evals = 0;
};

void set_direction(Opt &s) {
  for (int i = 0; i < 3; ++i)
    s.d[i] = s.H[i][0] * s.g[0] + s.H[i][1] * s.g[1] + s.H[i][2] * s.g[2];
  s.slope = s.d[0] * s.g[0] + s.d[1] * s.g[1] + s.d[2] * s.g[2];
  if (!(s.slope > 0.0)) {
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) s.H[i][j] = i == j ? s.h0 : 0.0;
    for (int i = 0; i < 3; ++i) s.d[i] = s.h0 * s.g[i];
    s.slope = s.h0 * (s.g[0] * s.g[0] + s.g[1] * s.g[1] + s.g[2] * s.g[2]);
  }
  s.alpha = 1.0;
  s.ls = 0;
  if (!(s.slope > 0.0)) s.done = true;
}

}  // namespace

int cube_objective(const DeviceObs &o, uint64_t n, const psr_timing &ref, const psr_timing *theta,
                   uint64_t K, const RefineOptions &opt, double *Jout, double *gout,
                   cudaStream_t st) {
  const int B = (int)opt.bins, S = (int)opt.subints;
  if (B > CB_MAXB || B < 8 || S < 1 || K == 0) {
    set_error("cube_objective: 8..1024 bins, >= 1 subint and >= 1 point required");
    return PSR_EINVAL;
  }
  const double nu_r = 1.0 / ref.period_s, nudot_r = -ref.pdot * nu_r * nu_r;
  CubeWork w;
  PSR_TRY(build_cube(o, n, S, B, nu_r, nudot_r, ref.dm, w, st));
  std::vector<CandDev> cand(K);
  for (uint64_t k = 0; k < K; ++k) {
    cand[k].nu = 1.0 / theta[k].period_s;
    cand[k].nudot = -theta[k].pdot * cand[k].nu * cand[k].nu;
    cand[k].dm = theta[k].dm;
  }
  std::vector<double> J, grad;
  PSR_TRY(eval_cube(o, n, S, B, cand, w, J, grad, st));
  for (uint64_t k = 0; k < K; ++k) {
    Jout[k] = J[k];
    if (gout) {
      gout[3 * k] = grad[3 * k];
      gout[3 * k + 1] = grad[3 * k + 1];
      gout[3 * k + 2] = grad[3 * k + 2];
    }
  }
  return PSR_OK;
}

int refine_cube_group(const DeviceObs &o, uint64_t n, const psr_timing *start, uint64_t K,
                      const RefineOptions &opt, psr_timing *out, double *Jout, uint64_t *evals,
                      CubeCache &cache, cudaStream_t st) {
  if (K == 0) return PSR_OK;
  const int B = (int)opt.bins, S = (int)opt.subints;
  if (B > CB_MAXB) {
    set_error("refine: at most 1024 bins");
    return PSR_EINVAL;
  }
  // Reference: the median start.
  std::vector<double> nus(K), dms(K);
  for (uint64_t k = 0; k < K; ++k) {
    nus[k] = 1.0 / start[k].period_s;
    dms[k] = start[k].dm;
  }
  std::vector<double> sn = nus, sd = dms;
  std::nth_element(sn.begin(), sn.begin() + K / 2, sn.end());
  std::nth_element(sd.begin(), sd.begin() + K / 2, sd.end());
  const double nu_r = sn[K / 2], dm_r = sd[K / 2];
  const double nudot_r = -start[K / 2].pdot * nu_r * nu_r;
  if (!cache.w) cache.w = new CubeWork();
  CubeWork &w = *cache.w;
  PSR_TRY(build_cube(o, n, S, B, nu_r, nudot_r, dm_r, w, st));
  const double T = (double)n * o.h.tsamp;
  double fmax = 0.0, fmin = 1e300;
  for (uint64_t c = 0; c < o.nch; ++c) {
    const double f = o.h.fch1 + (double)c * o.h.foff;
    fmax = std::fmax(fmax, f);
    fmin = std::fmin(fmin, f);
  }
  const double kspan = K_DM_C * (1.0 / (fmin * fmin) - 1.0 / (fmax * fmax));
  // Orthogonal scaled coordinates, as in the filterbank optimiser:
  // dnu = (2 q1 - 4 q2) / (B T), dnudot = 8 q2 / (B T^2), dDM = q3 s3.
  const double Bd = (double)B;
  const double s3 = kspan > 0.0 ? 1.0 / (nu_r * Bd * kspan) : 1.0;
  const double dm_hi = max_dm_for(o, n);
  std::vector<Opt> st8(K);
  auto theta = [&](uint64_t k, const double q[3]) {
    CandDev c;
    const double nu0 = 1.0 / start[k].period_s;
    const double nudot0 = -start[k].pdot * nu0 * nu0;
    c.nu = nu0 + (2.0 * q[0] - 4.0 * q[1]) / (Bd * T);
    c.nudot = nudot0 + 8.0 * q[1] / (Bd * T * T);
    double dm = start[k].dm + q[2] * s3;
    if (opt.dm_window > 0.0)
      dm = std::fmin(std::fmax(dm, start[k].dm - opt.dm_window), start[k].dm + opt.dm_window);
    c.dm = std::fmin(std::fmax(dm, 0.0), dm_hi);
    return c;
  };
  std::vector<double> J, grad;
  for (uint64_t round = 0; round < opt.max_evals; ++round) {
    std::vector<CandDev> batch;
    std::vector<uint64_t> who;
    for (uint64_t k = 0; k < K; ++k) {
      Opt &s = st8[k];
      if (s.done) continue;
      if (!s.started) {
        batch.push_back(theta(k, s.q));
      } else {
        for (int i = 0; i < 3; ++i) s.qn[i] = s.q[i] + s.alpha * s.d[i];
        batch.push_back(theta(k, s.qn));
      }
      who.push_back(k);
    }
    if (batch.empty()) break;
    PSR_TRY(eval_cube(o, n, S, B, batch, w, J, grad, st));
    for (size_t i = 0; i < who.size(); ++i) {
      Opt &s = st8[who[i]];
      ++s.evals;
      const double gq[3] = {grad[i * 3] * 2.0 / (Bd * T),
                            grad[i * 3] * (-4.0 / (Bd * T)) + grad[i * 3 + 1] * 8.0 / (Bd * T * T),
                            grad[i * 3 + 2] * s3};
      if (!s.started) {
        s.started = true;
        s.J = J[i];
        for (int j = 0; j < 3; ++j) s.g[j] = gq[j];
        const double gn = std::sqrt(gq[0] * gq[0] + gq[1] * gq[1] + gq[2] * gq[2]);
        s.h0 = gn > 0.0 ? 1.0 / gn : 1.0;
        for (int a = 0; a < 3; ++a)
          for (int b = 0; b < 3; ++b) s.H[a][b] = a == b ? s.h0 : 0.0;
        set_direction(s);
        continue;
      }
      if (J[i] >= s.J + 1e-4 * s.alpha * s.slope) {
        double sv[3], yv[3], maxstep = 0.0;
        for (int j = 0; j < 3; ++j) {
          sv[j] = s.qn[j] - s.q[j];
          yv[j] = -(gq[j] - s.g[j]);
          maxstep = std::fmax(maxstep, std::fabs(sv[j]));
        }
        const double sy = sv[0] * yv[0] + sv[1] * yv[1] + sv[2] * yv[2];
        if (sy > 1e-12) {
          double Hy[3], yHy = 0.0;
          for (int a = 0; a < 3; ++a)
            Hy[a] = s.H[a][0] * yv[0] + s.H[a][1] * yv[1] + s.H[a][2] * yv[2];
          for (int a = 0; a < 3; ++a) yHy += yv[a] * Hy[a];
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b)
              s.H[a][b] += (sy + yHy) * sv[a] * sv[b] / (sy * sy) -
                           (Hy[a] * sv[b] + sv[a] * Hy[b]) / sy;
        }
        for (int j = 0; j < 3; ++j) {
          s.q[j] = s.qn[j];
          s.g[j] = gq[j];
        }
        s.J = J[i];
        if (maxstep < opt.tol) s.done = true;
        else set_direction(s);
      } else {
        s.alpha *= 0.5;
        if (++s.ls >= 12) s.done = true;
      }
    }
  }
  for (uint64_t k = 0; k < K; ++k) {
    const CandDev c = theta(k, st8[k].q);
    out[k].period_s = 1.0 / c.nu;
    out[k].pdot = -c.nudot / (c.nu * c.nu);
    out[k].dm = c.dm;
    if (Jout) Jout[k] = st8[k].J;
    if (evals) evals[k] = st8[k].evals;
  }
  return PSR_OK;
}

}  // namespace psr
