// K5 power normalisation + birdies, K6 harmonic sums + peaks, K7 per-trial
// sort/dedupe (search/src/lib.rs:45-144).
//
// Normalisation: every 64-bin block b is divided by
//   scale_b = max(max(median(raw[lo..hi]) / ln2, floor), 1e-20),
//   lo = max(64b-128, 1), hi = min(64b+192, len), floor = 1e-6 * mean(raw).
// The median is exact: each 64-bin chunk is sorted once per CTA (a register
// bitonic network per thread; non-negative floats order like their bit
// patterns), elements
// provably below the window's rank-(cnt/2) element are skipped with binary
// searches, and a 5-way merge walk over the sorted chunks finds it.  Normalised power is never
// stored: pw(i) = raw[i] / scale[i>>6], zero for i == 0 and birdie bins.
//
// Harmonic sums follow the reference's f64 arithmetic exactly.  The f64 work
// is only done where it can matter: h = 1 scores are pw(k) or pw(k+1) minus 1,
// so a bin whose larger neighbour cannot reach the threshold is skipped
// before the parabolic offset is computed; h >= 2 scores exist only where
// pw(k) >= 4 (search/src/lib.rs:85-87).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "psr_internal.h"

namespace psr {
namespace {

constexpr int SC_NT = 256;               // threads per CTA, one chunk sort each
constexpr int SC_CH = SC_NT;             // chunks staged per CTA
constexpr int SC_G = SC_CH - 4;          // blocks per CTA (chunks b-2 .. b+2 each)
constexpr float LN2F = 0.693147180559945309f;

__device__ __forceinline__ uint32_t fbits(float f) { return __float_as_uint(f); }

// Number of elements <= key in a sorted chunk of 64 keys (invalid slots hold
// 0xffffffff, above every finite float pattern).  Branchless, 7 probes.
__device__ __forceinline__ int count_le64(const uint32_t *a, uint32_t key) {
  int pos = (a[31] <= key) ? 32 : 0;
  pos += (a[pos + 15] <= key) ? 16 : 0;
  pos += (a[pos + 7] <= key) ? 8 : 0;
  pos += (a[pos + 3] <= key) ? 4 : 0;
  pos += (a[pos + 1] <= key) ? 2 : 0;
  pos += (a[pos] <= key) ? 1 : 0;
  pos += (a[pos] <= key) ? 1 : 0;
  return pos;
}

// Sorted chunks are stored with a 65-word stride so that threads probing the
// same index of different chunks hit different banks; unsorted ones with a
// 68-word stride, for 16-byte accesses (8 lanes' quads fill the 32 banks).
constexpr int SC_STRIDE = 65;
constexpr int SC_RAW = 68;

struct RawCand {
  double score;
  double freq;
  uint32_t k;
  uint32_t h;
};

struct HarmArgs {
  const float *power;
  uint64_t ldp;
  uint64_t plen;
  const float *scale;
  uint64_t lds;
  const double *birdies;
  int nbirdies;
  double bin_hz;
  double threshold;
  float t1;  // smallest float v with (double)v - 1.0 >= threshold
  float lim[6];  // harm_maybe: h + threshold sqrt(h), lowered (-inf: always exact)
  uint64_t first;
  uint64_t end[6];  // end_h for h = 1,2,4,8,16,32 (0 when the h loop is skipped)
  RawCand *raw;
  unsigned *raw_count;
  uint64_t raw_cap;
  unsigned *overflow;
};

__device__ __forceinline__ float pw(const HarmArgs &a, const float *raw, const float *sc,
                                    uint64_t i) {
  if (i == 0) return 0.0f;
  float v = __fdiv_rn(raw[i], sc[i >> 6]);
  if (a.nbirdies) {
    const double f = (double)i * a.bin_hz;
    for (int q = 0; q < a.nbirdies; ++q)
      if (fabs(__dsub_rn(f, a.birdies[2 * q])) <= a.birdies[2 * q + 1]) return 0.0f;
  }
  return v;
}

// Parabolic offset (search/src/lib.rs:91-96).
__device__ __forceinline__ double offset_at(const float *raw, uint64_t k) {
  const double a = (double)raw[k - 1], b = (double)raw[k], c = (double)raw[k + 1];
  const double curv = __dadd_rn(__dsub_rn(a, __dmul_rn(2.0, b)), c);
  if (curv < 0.0) {
    const double o = __ddiv_rn(__dmul_rn(0.5, __dsub_rn(a, c)), curv);
    return fmin(fmax(o, -0.5), 0.5);
  }
  return 0.0;
}

__device__ __forceinline__ double inv_sqrt_div(double x, int hi) {
  // (sum - h) / sqrt(h): sqrt(h) correctly rounded as in Rust's f64::sqrt.
  switch (hi) {
    case 0: return x;
    case 1: return __ddiv_rn(x, 1.4142135623730951);
    case 2: return __dmul_rn(x, 0.5);
    case 3: return __ddiv_rn(x, 2.8284271247461903);
    case 4: return __dmul_rn(x, 0.25);
    default: return __ddiv_rn(x, 5.656854249492381);
  }
}

// round(RN(kf * j)) for a positive normal double kf and 1 <= j <= 32, in
// exact 64-bit integer arithmetic: kf = m * 2^E (53-bit m), the product m*j
// is exact in 58 bits, rounded to 53 bits (nearest, ties to even) as the FPU
// would, then rounded to an integer half away from zero as f64::round does.
// Bit-identical to (uint64_t)round(__dmul_rn(kf, (double)j)).
__device__ __forceinline__ uint64_t round_mul(double kf, uint32_t j) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(kf);
  const int E = (int)((bits >> 52) & 0x7ff) - 1075;
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  unsigned long long q = m * (unsigned long long)j;
  int F = E;
  const int nb = 64 - __clzll((long long)q);
  if (nb > 53) {
    const int sh = nb - 53;
    const unsigned long long rem = q & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
    q >>= sh;
    F += sh;
    if (rem > half || (rem == half && (q & 1ull))) ++q;
    if (q >> 53) {
      q >>= 1;
      ++F;
    }
  }
  if (F >= 0) return q << F;
  const int s = -F;
  if (s >= 64) return 0;
  const unsigned long long ip = q >> s, fr = q & ((1ull << s) - 1ull);
  return ip + (fr >= (1ull << (s - 1)) ? 1ull : 0ull);
}

// Full score of harmonic level hi (h = 1 << hi) at bin k (k in [first, end]);
// kf = k + the parabolic offset.
__device__ double score_at(const HarmArgs &a, const float *raw, const float *sc, uint64_t k,
                           int hi, double &kf) {
  const int h = 1 << hi;
  kf = __dadd_rn((double)k, offset_at(raw, k));
  if (h > 1 && pw(a, raw, sc, k) < 4.0f) return -INFINITY;
  double sum = -0.0;
  for (int j0 = 1; j0 <= h; j0 += 8) {  // gathers in flight, then the sums in order
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      v[u] = 0.0f;
      if (j0 + u <= h) {
        uint64_t idx = round_mul(kf, (uint32_t)(j0 + u));
        if (idx > a.plen - 1) idx = a.plen - 1;
        v[u] = pw(a, raw, sc, idx);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + u <= h) sum = __dadd_rn(sum, (double)v[u]);
  }
  return inv_sqrt_div(__dsub_rn(sum, (double)h), hi);
}

// Appends a raw candidate.  The lanes of a warp that emit together (all for
// the CTA's one trial) take consecutive slots: a ballot of the converged
// lanes, one atomic by the lowest, the base broadcast by a shuffle and each
// lane's rank among them.  The order of the raw list does not matter:
// k_select orders it by (score, h, k).
__device__ void emit(const HarmArgs &a, uint64_t trial, uint64_t k, int hi, double score,
                     double kf) {
  const unsigned mask = __activemask();
  const int lane = (int)(threadIdx.x & 31);
  const int leader = __ffs(mask) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(&a.raw_count[trial], (unsigned)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  const unsigned slot = base + (unsigned)__popc(mask & ((1u << lane) - 1u));
  if (slot >= a.raw_cap) {
    atomicOr(a.overflow, OVERFLOW_RAW);
    return;
  }
  RawCand c;
  c.score = score;
  c.freq = __dmul_rn(kf, a.bin_hz);
  c.k = (uint32_t)k;
  c.h = (uint32_t)hi;
  a.raw[trial * a.raw_cap + slot] = c;
}

// Gate queues: per trial the bins that pass the h = 1 gate (q1) and the
// h >= 2 gate (q2); capacity qcap each, counts n1/n2.  xq: the (bin, level)
// pairs left for exact evaluation, k | level << 25, bit 28 set where both
// neighbours' scores are certainly lower; capacity xcap, count nx.
struct GateArgs {
  uint32_t *q1, *q2, *xq;
  unsigned *n1, *n2, *nx;
  uint64_t qcap, xcap;
};
constexpr uint32_t XQ_PEAK = 1u << 28;

// The floor of every spectrum's scales (search/src/lib.rs:53-54): 1e-6 of its
// mean raw power, from the FFT's partial sums.  One warp per trial, before the
// gate kernel: every CTA of that computed it again, about 1500 cycles of FP64
// (1/64 of the f32 rate) in front of its first barrier.
__global__ void __launch_bounds__(128)
    k_floor(const double *__restrict__ psum, uint32_t npsum, uint64_t ntrials, uint64_t plen,
            float *__restrict__ floor_out) {
  const uint64_t trial = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = (int)(threadIdx.x & 31);
  if (trial >= ntrials) return;
  double s = 0.0;
  for (uint32_t i = lane; i < npsum; i += 32) s += psum[trial * npsum + i];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) floor_out[trial] = (float)(s / (double)plen * 1e-6);
}

constexpr int SCG_OWN = SC_G * 64;  // bins of the CTA's own blocks
constexpr int SCG_LQ = 1024;        // local queue slots (overflow goes to global)
constexpr size_t SCG_SMEM = (size_t)SC_CH * SC_RAW * 4 + (size_t)(SC_G + 4) * 4 +
                            (size_t)SCG_LQ * 2 * 2;

// Normalisation scales of SC_G blocks per CTA, then the harmonic gates on the
// CTA's own bins while they are hot in L2.  An h = 1 peak needs
// max(pw(k), pw(k+1)) >= t1 (t1 = the smallest float whose f64 value minus 1
// reaches the threshold; score_1(k) is pw(k) - 1 or pw(k+1) - 1), and h >= 2
// scores exist only where pw(k) >= 4.  The gates are conservative supersets:
// pw is estimated as raw * (1/scale) and a bin is queued unless the estimate
// is below the threshold by more than 4e-7 relative (the estimate is within
// 2e-7 of the correctly rounded quotient); birdies are ignored and the last
// bin, whose neighbour's scale belongs to the next CTA, is always queued.
// The item kernel evaluates every queued bin exactly.
//
// Median: the rank is counted at a pivot, the mean of the five chunks' own
// medians (7 probes per chunk), then at one moved by the density of exponential
// noise, which on a locally flat spectrum is two or three ranks short; a merge
// walk forwards or backwards over the sorted chunks finishes.  Far pivots fall
// back to rank-bound skips.
// Bound: ALU (the sorting network's 1086 min/max per thread of about 4000
// instructions).  Measured on a GB300, 64 spectra of 2^19 bins: 116 us with up
// to six rounds of skips from rank 0, word-wise staging and one shared atomic
// per queued bin, 114 now.
__global__ void __launch_bounds__(SC_NT)
    k_scales_gate(HarmArgs a, const float *__restrict__ floor_in, uint64_t nblocks,
                  float *__restrict__ scale_out, GateArgs g) {
  extern __shared__ __align__(16) uint32_t dsm[];
  uint32_t *ch = dsm;                                // SC_CH x SC_STRIDE (sorted chunks)
  float *inv_s = reinterpret_cast<float *>(ch + SC_CH * SC_RAW);  // 1/scale per block
  uint16_t *lq1 = reinterpret_cast<uint16_t *>(inv_s + SC_G + 4);
  uint16_t *lq2 = lq1 + SCG_LQ;
  __shared__ int c1, c2;
  __shared__ unsigned base1, base2;
  const uint64_t plen = a.plen;
  const uint64_t trial = blockIdx.y;
  const float *raw = a.power + trial * a.ldp;
  const long long b0 = (long long)blockIdx.x * SC_G;
  const long long c_first = b0 - 2;  // chunk index of local chunk 0
  const float floor_s = __ldg(floor_in + trial);
  if (threadIdx.x == 0) c1 = c2 = 0;
  // Stage the bins of all chunks (16-byte loads, four in flight per thread);
  // out-of-range chunks and bin 0 hold the sentinel 0xffffffff.
  constexpr int NV = SC_CH * 64;
  constexpr int NV4 = NV / 4;
  static_assert(NV4 % (4 * SC_NT) == 0, "staging loop covers the chunks exactly");
  // e = (first bin of the CTA's chunks) + 4 i; 32-bit arithmetic: plen < 2^25
  const int e_first = (int)(c_first * 64), plen_i = (int)plen;
#pragma unroll 1
  for (int base = 0; base < NV4; base += 4 * SC_NT) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e_first + 4 * (base + u * SC_NT + (int)threadIdx.x);
      if (e >= 1 && e + 3 < plen_i) {
        v[u] = *reinterpret_cast<const uint4 *>(raw + e);
      } else {
        uint32_t t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          t[j] = (e + j >= 1 && e + j < plen_i) ? fbits(raw[e + j]) : 0xffffffffu;
        v[u] = make_uint4(t[0], t[1], t[2], t[3]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q = base + u * SC_NT + (int)threadIdx.x;  // quad q of the CTA: chunk q / 16
      *reinterpret_cast<uint4 *>(ch + (q >> 4) * SC_RAW + 4 * (q & 15)) = v[u];
    }
  }
  __syncthreads();
  {
    // Thread t sorts chunk t in registers: Batcher's odd-even merge sort
    // network (543 compare-exchanges for 64 keys), fully unrolled, so every
    // register index is static and there are no shuffles.
    uint32_t x[64];
    {
      const uint4 *row = reinterpret_cast<const uint4 *>(ch + threadIdx.x * SC_RAW);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint4 q = row[i];
        x[4 * i] = q.x;
        x[4 * i + 1] = q.y;
        x[4 * i + 2] = q.z;
        x[4 * i + 3] = q.w;
      }
    }
    __syncthreads();  // the sorted rows overlay the unsorted ones
    uint32_t *row = ch + threadIdx.x * SC_STRIDE;
    // (merge step (p, k) compares a with a + k for every a >= k % p with
    // (a - k % p) mod 2k < k, both in one block of 2p)
#pragma unroll
    for (int p = 1; p < 64; p <<= 1)
#pragma unroll
      for (int k = p; k >= 1; k >>= 1)
#pragma unroll
        for (int a = 0; a < 64; ++a) {
          const int c = a + k, j0 = k % p;
          if (c < 64 && a >= j0 && (a - j0) % (2 * k) < k && a / (2 * p) == c / (2 * p)) {
            const uint32_t p0 = x[a], p1 = x[c];
            x[a] = min(p0, p1);
            x[c] = max(p0, p1);
          }
        }
#pragma unroll
    for (int i = 0; i < 64; ++i) row[i] = x[i];
  }
  __syncthreads();
  const long long b = b0 + threadIdx.x;
  if (threadIdx.x < SC_G && b < (long long)nblocks) {
    const long long center = b * 64;
    const long long lo = max(center - 128, 1ll);
    const long long hi = min(center + 192, (long long)plen);
    const int r = (int)(hi - lo) / 2;
    // The window is local chunks threadIdx.x .. threadIdx.x + 4 (chunks
    // b-2..b+2), each sorted and padded with sentinels above every value.
    const uint32_t *w = ch + threadIdx.x * SC_STRIDE;
    // Pivot: the mean of the chunks' middle keys (as floats; a chunk that is
    // not full may hold a sentinel there).
    int p[5] = {0, 0, 0, 0, 0};
    int rr = r;
    uint32_t med_k = 0;
    bool found = false;
    {
      float sum = 0.0f;
      int full = 0;
#pragma unroll
      for (int d = 0; d < 5; ++d) {
        const uint32_t m = w[d * SC_STRIDE + 32];
        if (m < 0x7f800000u) {
          sum += __uint_as_float(m);
          ++full;
        }
      }
      uint32_t y = full ? __float_as_uint(__fdividef(sum, (float)full)) : 0u;
      if (y > 0u && y < 0x7f000000u) {
        int c = 0, cnt[5];
        auto count = [&]() {
          c = 0;
#pragma unroll
          for (int d = 0; d < 5; ++d) {
            cnt[d] = count_le64(w + d * SC_STRIDE, y - 1u);  // elements < y
            c += cnt[d];
          }
        };
        count();
        // Second pivot, two ranks short: exponential noise has (hi - lo) ln 2 /
        // 2 y elements per unit around its median y.
        const float step = __fdividef((float)(r - c) - 2.0f, 0.34657f * (float)(hi - lo));
        if (fabsf(step) < 0.3f) {
          y = __float_as_uint(__uint_as_float(y) * (1.0f + step));
          count();
        }
        if (c <= r) {  // forwards: these c elements lie below the target
#pragma unroll
          for (int d = 0; d < 5; ++d) p[d] = cnt[d];
          rr = r - c;
        } else if (c - r <= 24) {
          // backwards: the (c - r)-th largest of the elements below y.  Heads
          // are keys + 1, 0 where a chunk has none left.
          uint32_t hd[5];
#pragma unroll
          for (int d = 0; d < 5; ++d) hd[d] = cnt[d] ? w[d * SC_STRIDE + cnt[d] - 1] + 1u : 0u;
          for (int step = c - r; step > 0; --step) {
            uint32_t m = hd[0];
            int am = 0;
#pragma unroll
            for (int d = 1; d < 5; ++d)
              if (hd[d] > m) {
                m = hd[d];
                am = d;
              }
            med_k = m - 1u;
#pragma unroll
            for (int d = 0; d < 5; ++d)
              if (d == am) {
                --cnt[d];
                hd[d] = cnt[d] ? w[d * SC_STRIDE + cnt[d] - 1] + 1u : 0u;
              }
          }
          found = true;
        }
      }
    }
    if (!found) {
      // Rank-bound skips: with p_d elements of chunk d already known to lie
      // below the target and rr = r - sum(p_d), let y = min_d A_d[p_d + rr/5].
      // Each chunk has at most rr/5 unskipped elements below y, so at most rr
      // elements below y remain and the rank-r element is >= y: skip them.
      // Every round shrinks rr geometrically; a short merge walk finishes.
      for (int round = 0; round < 6; ++round) {
        const int q = rr / 5;
        if (q < 3) break;  // (a walk over up to 14 is cheaper than another round)
        uint32_t y = 0xffffffffu;
#pragma unroll
        for (int d = 0; d < 5; ++d)
          if (p[d] + q < 64) y = min(y, w[d * SC_STRIDE + p[d] + q]);
        if (y == 0u) break;
        int adv = 0;
#pragma unroll
        for (int d = 0; d < 5; ++d) {
          const int np = count_le64(w + d * SC_STRIDE, y - 1u);  // elements < y
          adv += np - p[d];
          p[d] = np;
        }
        rr -= adv;
        if (adv == 0) break;
      }
      // 5-way merge walk over the rest: advance the smallest head rr times; the
      // smallest head is then the rank-r element.
      uint32_t hd[5];
#pragma unroll
      for (int d = 0; d < 5; ++d) hd[d] = p[d] < 64 ? w[d * SC_STRIDE + p[d]] : 0xffffffffu;
      for (int step = 0; step < rr; ++step) {
        uint32_t m = hd[0];
        int am = 0;
#pragma unroll
        for (int d = 1; d < 5; ++d)
          if (hd[d] < m) {
            m = hd[d];
            am = d;
          }
#pragma unroll
        for (int d = 0; d < 5; ++d)
          if (d == am) {
            ++p[d];
            hd[d] = p[d] < 64 ? w[d * SC_STRIDE + p[d]] : 0xffffffffu;
          }
      }
      med_k = hd[0];
#pragma unroll
      for (int d = 1; d < 5; ++d) med_k = min(med_k, hd[d]);
    }
    const float sc = fmaxf(fmaxf(__fdiv_rn(__uint_as_float(med_k), LN2F), floor_s), 1e-20f);
    inv_s[threadIdx.x] = __frcp_rn(sc);
    scale_out[trial * a.lds + b] = sc;
  }
  __syncthreads();
  // Gates on the CTA's own bins (raw values re-read; they are hot in L2).
  const uint64_t kb0 = (uint64_t)b0 * 64;
  const float t1lo = a.t1 > 0.0f ? a.t1 * (1.0f - 4e-7f) : -INFINITY;
  const float t4lo = 4.0f * (1.0f - 4e-7f);
  uint32_t *gq1 = g.q1 + trial * g.qcap, *gq2 = g.q2 + trial * g.qcap;
  // Four consecutive bins per thread (one 16-byte load, one block scale);
  // the fourth bin's neighbour is the next group's first (the next lane's).
  // Bins [ilo, ihi] of the CTA are candidates ([first + 1, end_1 - 1]).
  const int own = SCG_OWN;
  const int ilo = (int)max((long long)(a.first + 1) - (long long)kb0, 0ll);
  const int ihi = (int)min((long long)a.end[0] - 1 - (long long)kb0, (long long)own - 1);
  // About 7% of a noise spectrum's groups hold a gated bin, so nearly every
  // warp does: each lane makes a 4-bit mask per gate, and the warp's lanes
  // take their slots from one atomic and the prefix of their counts (in bit
  // planes of ballots).
  const int lane = (int)(threadIdx.x & 31);
  const unsigned below = (1u << lane) - 1u;
  auto append = [&](unsigned m, int i, int *count, uint16_t *lq, unsigned *gcount, uint32_t *gq) {
    const unsigned cnt = (unsigned)__popc(m);
    const unsigned b0 = __ballot_sync(0xffffffffu, cnt & 1u);
    const unsigned b1 = __ballot_sync(0xffffffffu, cnt & 2u);
    const unsigned b2 = __ballot_sync(0xffffffffu, cnt & 4u);
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2));
    int slot = __shfl_sync(0xffffffffu, base, 0) + __popc(b0 & below) + 2 * __popc(b1 & below) +
               4 * __popc(b2 & below);
    while (m) {
      const int j = __ffs((int)m) - 1;
      m &= m - 1;
      if (slot < SCG_LQ) {
        lq[slot] = (uint16_t)(i + j);
      } else {
        const unsigned gi = atomicAdd(gcount, 1u);
        if (gi < g.qcap) gq[gi] = (uint32_t)(kb0 + (uint64_t)(i + j));
        else atomicOr(a.overflow, OVERFLOW_QUEUE);
      }
      ++slot;
    }
  };
  // (four groups per thread in flight: the queue's stores keep the compiler
  // from moving a later group's load above them)
  constexpr int GU = 4;
  for (int i0 = 0; i0 < own / 4; i0 += GU * SC_NT) {  // (uniform trip count)
    float4 r[GU];
    float edge[GU];  // the bin after the warp's last, in lane 31
#pragma unroll
    for (int u = 0; u < GU; ++u) {
      const int i = 4 * (i0 + u * SC_NT + (int)threadIdx.x);
      r[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      edge[u] = 0.0f;
      // (one bin past the last candidate: the group before it, if full, takes
      // its last bin's neighbour from here; at most bin plen + 1 of the padded row)
      if (i < own && i + 3 >= ilo && i <= ihi + 1) {
        r[u] = *reinterpret_cast<const float4 *>(raw + kb0 + (uint64_t)i);
        if (lane == 31 && i + 4 < own && i + 3 <= ihi) edge[u] = raw[kb0 + (uint64_t)(i + 4)];
      }
    }
#pragma unroll
    for (int u = 0; u < GU; ++u) {
      const int i = 4 * (i0 + u * SC_NT + (int)threadIdx.x);
      const float up = __shfl_down_sync(0xffffffffu, r[u].x, 1);
      const float nr = lane == 31 ? edge[u] : up;
      unsigned m1 = 0, m2 = 0;
      if (i < own && i + 3 >= ilo && i <= ihi) {
        const float inv = inv_s[i >> 6];
        const float e[4] = {r[u].x * inv, r[u].y * inv, r[u].z * inv, r[u].w * inv};
        const float nx = (i + 4 < own && i + 3 <= ihi) ? nr * inv_s[(i + 4) >> 6] : 0.0f;
        unsigned mt = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          m2 |= e[j] >= t4lo ? 1u << j : 0u;
          mt |= fmaxf(e[j], j < 3 ? e[j + 1] : nx) >= t1lo ? 1u << j : 0u;
        }
        m1 = mt | (i + 4 < own ? 0u : 8u);  // the CTA's last bin always
        if (i < ilo || i + 3 > ihi) {
          const unsigned in = (0xfu << max(ilo - i, 0)) & (0xfu >> max(i + 3 - ihi, 0));
          m1 &= in;
          m2 &= in;
        }
      }
      if (__any_sync(0xffffffffu, m2)) append(m2, i, &c2, lq2, &g.n2[trial], gq2);
      if (__any_sync(0xffffffffu, m1)) append(m1, i, &c1, lq1, &g.n1[trial], gq1);
    }
  }
  __syncthreads();
  const int m1 = min(c1, SCG_LQ), m2 = min(c2, SCG_LQ);
  if (threadIdx.x == 0) {
    base1 = atomicAdd(&g.n1[trial], (unsigned)m1);
    base2 = atomicAdd(&g.n2[trial], (unsigned)m2);
  }
  __syncthreads();
  if (threadIdx.x == 0 && (base1 + m1 > g.qcap || base2 + m2 > g.qcap))
    atomicOr(a.overflow, OVERFLOW_QUEUE);
  for (int i = threadIdx.x; i < m1 && base1 + i < g.qcap; i += SC_NT)
    gq1[base1 + i] = (uint32_t)(kb0 + lq1[i]);
  for (int i = threadIdx.x; i < m2 && base2 + i < g.qcap; i += SC_NT)
    gq2[base2 + i] = (uint32_t)(kb0 + lq2[i]);
}

// The f32 side of the harmonic sums.  The positions round((k + off) j) are found
// from the f32 parabolic offset with a bound on its error: off is exactly 0
// where the curvature is certainly not negative, exactly +-1/2 where it is
// certainly clamped, else off +- eps; ok is false where that cannot be told.
struct Off {
  float off, eps;
  bool ok;
};
__device__ __forceinline__ Off off_f32(const float *raw, uint32_t k) {
  const float a = raw[k - 1], b = raw[k], c = raw[k + 1];
  const float curv = fmaf(-2.0f, b, a) + c, size = a + 2.0f * b + c;
  Off o{0.0f, 0.0f, fabsf(curv) > 1.3e-7f * size};  // (false for NaN)
  if (o.ok && curv < 0.0f) {
    const float rel = 1.5e-7f * __fdividef(size, -curv) + 1e-6f;
    if (!(rel <= 0.01f)) o.ok = false;
    o.off = __fdividef(0.5f * (a - c), curv);
    if (fabsf(o.off) > 0.5f + rel) {
      o.off = o.off > 0.0f ? 0.5f : -0.5f;
    } else {
      o.eps = fabsf(o.off) * rel;
      o.off = fminf(fmaxf(o.off, -0.5f), 0.5f);
    }
  }
  return o;
}
// raw / scale at harmonic j of bin k, to within 1e-6; `sure` is cleared where
// the position's rounding is within the offset's error (or the scale is
// extreme).  Birdies are ignored.
__device__ __forceinline__ float harm_f32(const float *raw, const float *sc, uint32_t last,
                                          uint32_t k, const Off &o, int j, bool &sure) {
  const float p = fmaf(o.off, (float)j, 0.5f), fl = floorf(p), fr = p - fl;
  const float ej = o.eps > 0.0f ? fmaf(o.eps, (float)j, 4e-6f) : 0.0f;
  const uint32_t idx = min(k * (uint32_t)j + (uint32_t)(int)fl, last);
  const float s = sc[idx >> 6];
  sure &= fr >= ej && fr <= 1.0f - ej && s < 1e30f;
  return __fdividef(raw[idx], s);
}
// Level hi's sum at a neighbour bin against `sum` at the peak: -1 certainly
// lower, 1 certainly higher, 0 not told.
__device__ __forceinline__ int neighbour_f32(const float *raw, const float *sc, uint32_t last,
                                             uint32_t k, int hi, float sum) {
  const float p = __fdividef(raw[k], sc[k >> 6]);
  if (p < 4.0f * (1.0f - 1e-5f)) return -1;  // no score below 4
  if (!(p > 4.0f * (1.0f + 1e-5f))) return 0;
  const Off o = off_f32(raw, k);
  bool sure = o.ok;
  float t = 0.0f;
  for (int j = 1; j <= (1 << hi); ++j) t += harm_f32(raw, sc, last, k, o, j, sure);
  if (!sure) return 0;
  return t < sum * (1.0f - 2e-5f) ? -1 : t > sum * (1.0f + 2e-5f) ? 1 : 0;
}

// Which (bin, level) pairs of the gated bins need the exact score.  A bin's sum
// at a level is certain to within 1e-5; the pair is passed on unless the sum
// is below the level's limit (h + threshold sqrt(h), lowered by 1e-5; birdies
// only lower a score) or, without birdies, a neighbour's is certainly higher.
// Every h = 1 bin is passed on.
// Bound: the gathers.  FP64 runs at 1/64 of the f32 rate here: with every
// gated bin's levels summed in f64 the items took 155 us for 64 spectra of
// 2^19 bins (76% of the FP64 pipe), filter and exact scores 32 + 47 now.
constexpr int HI_NT = 256;
constexpr int HI_CTAS_PER_TRIAL = 12;
constexpr int HX_NT = 128, HX_CTAS_PER_TRIAL = 4;

template <int NL>
__global__ void __launch_bounds__(HI_NT) k_harm_filter(HarmArgs a, GateArgs g) {
  constexpr int HMAX = 1 << (NL - 1);
  const uint64_t trial = blockIdx.y;
  const float *raw = a.power + trial * a.ldp;
  const float *sc = a.scale + trial * a.lds;
  const unsigned n1 = min(g.n1[trial], (unsigned)g.qcap), n2 = min(g.n2[trial], (unsigned)g.qcap);
  const uint32_t *q1 = g.q1 + trial * g.qcap, *q2 = g.q2 + trial * g.qcap;
  uint32_t *xq = g.xq + trial * g.xcap;
  const int lane = (int)(threadIdx.x & 31);
  const uint32_t last = (uint32_t)a.plen - 1;
  for (unsigned base = (blockIdx.x * HI_NT + threadIdx.x) & ~31u; base < n1 + n2;
       base += gridDim.x * HI_NT) {  // (warp-uniform)
    const unsigned idx = base + lane;
    uint32_t entry[NL];  // per level, ~0: none
#pragma unroll
    for (int hi = 0; hi < NL; ++hi) entry[hi] = 0xffffffffu;
    if (idx < n1) {
      entry[0] = q1[idx];
    } else if (idx < n1 + n2) {
      const uint32_t k = q2[idx - n1];
      int hmax = 0;
#pragma unroll
      for (int hi = 1; hi < NL; ++hi)
        if (a.end[hi] != 0 && k + 1 <= a.end[hi]) hmax = hi;
      if (hmax > 0) {
        const Off o = off_f32(raw, k);
        bool sure = o.ok;
        float v[HMAX];
#pragma unroll
        for (int j = 1; j <= HMAX; ++j)
          v[j - 1] = j <= (1 << hmax) ? harm_f32(raw, sc, last, k, o, j, sure) : 0.0f;
        float sum = v[0];
#pragma unroll
        for (int hi = 1; hi < NL; ++hi) {
#pragma unroll
          for (int j = 1 << (hi - 1); j < (1 << hi); ++j) sum += v[j];
          if (hi > hmax) continue;
          if (!sure) {
            entry[hi] = k | (uint32_t)hi << 25;
          } else if (!(sum < a.lim[hi])) {
            uint32_t x = k | (uint32_t)hi << 25;
            if (!a.nbirdies) {
              const int lo = neighbour_f32(raw, sc, last, k - 1, hi, sum);
              const int up = lo > 0 ? 0 : neighbour_f32(raw, sc, last, k + 1, hi, sum);
              if (lo > 0 || up > 0) x = 0xffffffffu;
              else if (lo < 0 && up < 0) x |= XQ_PEAK;
            }
            entry[hi] = x;
          }
        }
      }
    }
#pragma unroll
    for (int hi = 0; hi < NL; ++hi) {
      const bool take = entry[hi] != 0xffffffffu;
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (!m) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&g.nx[trial], (unsigned)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + (unsigned)__popc(m & ((1u << lane) - 1u));
      if (take) {
        if (at < g.xcap) xq[at] = entry[hi];
        else atomicOr(a.overflow, OVERFLOW_EXACT);
      }
    }
  }
}

// The exact scores (reference f64 arithmetic) of the filtered pairs.
__global__ void __launch_bounds__(HX_NT) k_harm_exact(HarmArgs a, GateArgs g) {
  const uint64_t trial = blockIdx.y;
  const float *raw = a.power + trial * a.ldp;
  const float *sc = a.scale + trial * a.lds;
  const unsigned n = min(g.nx[trial], (unsigned)g.xcap);
  const uint32_t *xq = g.xq + trial * g.xcap;
  for (unsigned i = blockIdx.x * HX_NT + threadIdx.x; i < n; i += gridDim.x * HX_NT) {
    const uint32_t x = xq[i];
    const uint64_t k = x & 0x1ffffffu;
    const int hi = (int)((x >> 25) & 7u);
    double kf, kn;
    const double s = score_at(a, raw, sc, k, hi, kf);
    if (s >= a.threshold) {
      const bool peak = (x & XQ_PEAK) || (s > score_at(a, raw, sc, k - 1, hi, kn) &&
                                          s >= score_at(a, raw, sc, k + 1, hi, kn));
      if (peak) emit(a, trial, k, hi, s, kf);
    }
  }
}

// Orderable key: score descending, then (h, k) ascending = the reference's
// insertion order under its stable sort (search/src/lib.rs:130).
__device__ __forceinline__ unsigned long long score_key_desc(double s) {
  unsigned long long b = (unsigned long long)__double_as_longlong(s);
  unsigned long long asc = (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
  return ~asc;
}

constexpr int SEL_CAP = 2048;
constexpr int SEL_NT = 512;

struct SelArgs {
  const RawCand *raw;
  const unsigned *raw_count;
  uint64_t raw_cap;
  const double *trial_dm;
  double tol;  // 1 / (len * tsamp)
  uint64_t max_candidates;
  psr_candidate *kept;
  unsigned *kept_count;
};

__device__ __forceinline__ bool key_less(unsigned long long ka, uint32_t sa,
                                         unsigned long long kb, uint32_t sb) {
  return ka < kb || (ka == kb && sa < sb);
}

// |a - b| < tol, exactly as the f64 comparison, with f32 copies deciding where
// their rounding (2^-24 of each) cannot matter.
__device__ __forceinline__ bool near_freq(double a, float af, double b, float bf, double tol,
                                          float tolf) {
  const float d = fabsf(af - bf), err = 3e-7f * fmaxf(fabsf(af), fabsf(bf)) + 2e-7f * tolf;
  if (d > tolf + err) return false;
  if (d < tolf - err) return true;
  return fabs(__dsub_rn(a, b)) < tol;
}

// One CTA per trial: the raw candidates in score order, then the reference's
// dedupe.  Bitonic sort of (score, order) keys in shared memory: the steps
// over distances below 64 stay inside a warp's 64-element blocks, so only the
// wider ones need the block's barrier.  Dedupe by one warp, 32 candidates at a
// time: each lane tests its candidate against the kept ones, then the lanes
// left are kept in order, each dropping those near it.
// Measured on a GB300, 64 GBT-shaped trials: 53 us with a barrier per step and
// the dedupe one candidate at a time from global memory, 26 now.
__global__ void __launch_bounds__(SEL_NT) k_select(SelArgs a) {
  __shared__ unsigned long long key[SEL_CAP];
  __shared__ uint32_t seq[SEL_CAP];
  __shared__ uint32_t idx[SEL_CAP];
  __shared__ double kept_f[64];
  __shared__ float kept_s[64];
  __shared__ int nk;
  const uint64_t trial = blockIdx.x;
  const RawCand *rc = a.raw + trial * a.raw_cap;
  const unsigned n = min(a.raw_count[trial], (unsigned)a.raw_cap);
  psr_candidate *out = a.kept + trial * a.max_candidates;
  const double dm = a.trial_dm[trial];
  if (threadIdx.x == 0) nk = 0;
  if (n <= SEL_CAP) {
    const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
    unsigned P = 64;
    while (P < n) P <<= 1;
    for (unsigned i = threadIdx.x; i < P; i += SEL_NT) {
      if (i < n) {
        key[i] = score_key_desc(rc[i].score);
        seq[i] = (rc[i].h << 24) | rc[i].k;
        idx[i] = i;
      } else {
        key[i] = ~0ull;
        seq[i] = 0xffffffffu;
        idx[i] = 0xffffffffu;
      }
    }
    __syncthreads();
    auto exchange = [&](unsigned i, unsigned l, unsigned k) {
      const bool up = (i & k) == 0;
      const unsigned long long ki = key[i], kl = key[l];
      const uint32_t si = seq[i], sl = seq[l];
      if (key_less(kl, sl, ki, si) == up) {
        key[i] = kl;
        key[l] = ki;
        seq[i] = sl;
        seq[l] = si;
        const uint32_t t = idx[i];
        idx[i] = idx[l];
        idx[l] = t;
      }
    };
    for (unsigned k = 2; k <= P; k <<= 1) {
      unsigned j = k >> 1;
      for (; j >= 64; j >>= 1) {
        for (unsigned p = threadIdx.x; p < P / 2; p += SEL_NT) {
          const unsigned i = 2 * j * (p / j) + p % j;
          exchange(i, i + j, k);
        }
        __syncthreads();
      }
      for (unsigned b = warp; b < P / 64; b += SEL_NT / 32)
        for (unsigned q = j; q > 0; q >>= 1) {
          const unsigned i = 64 * b + 2 * q * (lane / q) + lane % q;
          exchange(i, i + q, k);
          __syncwarp();
        }
      if (k >= 64) __syncthreads();  // (below, a block stays with its warp)
    }
    // Dedupe (search/src/lib.rs:131-143) by warp 0.
    if (warp == 0) {
      const float tolf = (float)a.tol;
      unsigned kc = 0;
      for (unsigned i0 = 0; i0 < n && kc < a.max_candidates; i0 += 32) {
        const bool in = i0 + lane < n;
        RawCand c{};
        if (in) c = rc[idx[i0 + lane]];
        const float cf = (float)c.freq;
        bool alive = in;
        for (unsigned q = 0; q < kc; ++q)
          alive = alive && !near_freq(kept_f[q], kept_s[q], c.freq, cf, a.tol, tolf);
        unsigned m = __ballot_sync(0xffffffffu, alive);
        while (m && kc < a.max_candidates) {
          const int w = __ffs((int)m) - 1;
          if (lane == w) {
            kept_f[kc] = c.freq;
            kept_s[kc] = cf;
            psr_candidate o;
            o.frequency_hz = c.freq;
            o.period_s = __ddiv_rn(1.0, c.freq);
            o.dm = dm;
            o.harmonics = 1ull << c.h;
            o.score = c.score;
            out[kc] = o;
            alive = false;
          }
          __syncwarp();
          if (alive) alive = !near_freq(kept_f[kc], kept_s[kc], c.freq, cf, a.tol, tolf);
          ++kc;
          m = __ballot_sync(0xffffffffu, alive);
        }
      }
      if (lane == 0) a.kept_count[trial] = kc;
    }
    return;
  }
  // More raw candidates than fit in shared memory: repeated arg-max over the
  // unsorted list (exact order; only reached by pathological spectra).
  __shared__ unsigned long long best_k[SEL_NT / 32];
  __shared__ uint32_t best_s[SEL_NT / 32], best_i[SEL_NT / 32];
  __shared__ unsigned long long last_k;
  __shared__ uint32_t last_s;
  if (threadIdx.x == 0) {
    last_k = 0;
    last_s = 0;
  }
  __syncthreads();
  bool started = false;
  for (;;) {
    unsigned long long bk = ~0ull;
    uint32_t bs = 0xffffffffu, bi = 0xffffffffu;
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned long long kk = score_key_desc(rc[i].score);
      const uint32_t ss = (rc[i].h << 24) | rc[i].k;
      if (started && !key_less(last_k, last_s, kk, ss)) continue;  // already consumed
      if (key_less(kk, ss, bk, bs)) {
        bk = kk;
        bs = ss;
        bi = i;
      }
    }
    for (int o = 16; o; o >>= 1) {
      unsigned long long ok = __shfl_xor_sync(0xffffffffu, bk, o);
      uint32_t os = __shfl_xor_sync(0xffffffffu, bs, o);
      uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (key_less(ok, os, bk, bs)) {
        bk = ok;
        bs = os;
        bi = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      best_k[threadIdx.x >> 5] = bk;
      best_s[threadIdx.x >> 5] = bs;
      best_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long k0 = ~0ull;
      uint32_t s0 = 0xffffffffu, i0 = 0xffffffffu;
      for (int w = 0; w < SEL_NT / 32; ++w)
        if (key_less(best_k[w], best_s[w], k0, s0)) {
          k0 = best_k[w];
          s0 = best_s[w];
          i0 = best_i[w];
        }
      best_i[0] = i0;
      if (i0 != 0xffffffffu) {
        last_k = k0;
        last_s = s0;
        const RawCand c = rc[i0];
        bool dup = false;
        for (int q = 0; q < nk; ++q) dup |= fabs(__dsub_rn(kept_f[q], c.freq)) < a.tol;
        if (!dup) {
          kept_f[nk] = c.freq;
          psr_candidate o;
          o.frequency_hz = c.freq;
          o.period_s = __ddiv_rn(1.0, c.freq);
          o.dm = dm;
          o.harmonics = 1ull << c.h;
          o.score = c.score;
          out[nk] = o;
          ++nk;
        }
      }
    }
    __syncthreads();
    started = true;
    if (best_i[0] == 0xffffffffu || (uint64_t)nk >= a.max_candidates) break;
    __syncthreads();
  }
  if (threadIdx.x == 0) a.kept_count[trial] = (unsigned)nk;
}

}  // namespace

// Buffers for up to `outer` trials' scales, queues and raw candidates; uploads the
// birdie list.
int spectrum_prepare(const FftPlan &p, const SpecConfig &c, uint64_t outer, SpecWork &w,
                     cudaStream_t st) {
  if (c.max_candidates > 64 || c.max_candidates < 1) {
    set_error("search: 1..64 candidates per trial are supported");
    return PSR_EINVAL;
  }
  const uint64_t plen = p.M + 1;
  const uint64_t nblocks = (plen + 63) / 64;
  w.lds = ((nblocks + 63) / 64) * 64;
  if (w.raw_cap == 0) w.raw_cap = 2048;
  PSR_TRY(w.scale.ensure(outer * w.lds * 4));
  PSR_TRY(w.raw.ensure(outer * w.raw_cap * sizeof(RawCand)));
  PSR_TRY(w.counts.ensure((4 * outer + 4) * 4));
  PSR_TRY(w.floors.ensure(outer * 4));
  // Gated bins are ~2% of a noise spectrum; a quarter of the bins is ample
  // and an overflow (flagged) reruns the chunk with room for every bin.  Raw lists
  // overflow on their own where a bright pulsar peaks in many bins, exact lists
  // where most bins pass the gates.
  const uint64_t quarter = plen / 4 + 1024;
  w.qcap = w.queue_full ? plen : quarter;
  // every level of every bin at most
  w.xcap = std::min(quarter * w.xgrow, (uint64_t)c.levels * plen);
  w.xgroup = std::max<uint64_t>(1, outer * quarter / w.xcap);
  PSR_TRY(w.gq.ensure(2 * outer * w.qcap * 4));
  PSR_TRY(w.xq.ensure(w.xgroup * w.xcap * 4));
  PSR_TRY(w.birdies.ensure(std::max<size_t>(c.birdies.size(), 2) * 8));
  if (!c.birdies.empty())
    PSR_CUDA(cudaMemcpyAsync(w.birdies.p, c.birdies.data(), c.birdies.size() * 8,
                             cudaMemcpyHostToDevice, st));
  return PSR_OK;
}

// counts: overflow word, then raw, q1, q2 and exact-list counts per trial.
int spectrum_reset(SpecWork &w, uint64_t outer_trials, cudaStream_t st) {
  PSR_CUDA(cudaMemsetAsync(w.counts.p, 0, (4 * outer_trials + 4) * 4, st));
  w.outer_trials = outer_trials;
  return PSR_OK;
}

// Normalisation scales and harmonic peaks of `ntrials` spectra; their raw
// candidates go to slots [slot0, slot0 + ntrials) of the outer chunk.
namespace {
HarmArgs harm_args(const FftPlan &p, const SpecConfig &c, const float *d_power, uint64_t ldp,
                   SpecWork &w) {
  const uint64_t plen = p.M + 1;
  // search/src/lib.rs:62, 73-78
  const double bin_hz = 1.0 / ((double)p.N * c.tsamp);
  HarmArgs a{};
  a.power = d_power;
  a.ldp = ldp;
  a.plen = plen;
  a.scale = w.scale.as<float>();
  a.lds = w.lds;
  a.birdies = w.birdies.as<double>();
  a.nbirdies = (int)(c.birdies.size() / 2);
  a.bin_hz = bin_hz;
  a.threshold = c.threshold;
  const double firstf = std::fmax(std::ceil(c.min_hz / bin_hz), 1.0);
  const uint64_t first = (uint64_t)firstf;
  const double lastf = std::floor(std::fmin(c.max_hz, 0.5 / c.tsamp) / bin_hz);
  const uint64_t last = std::min<uint64_t>(lastf <= 0.0 ? 0 : (uint64_t)lastf, plen - 2);
  a.first = first;
  for (int hi = 0; hi < c.levels; ++hi) {
    const uint64_t h = 1ull << hi;
    const uint64_t e = std::min(last, (plen - 2) / h);
    a.end[hi] = (e <= first + 1) ? 0 : e;
  }
  a.raw = w.raw.as<RawCand>();
  a.raw_count = w.counts.as<unsigned>() + 4;
  a.raw_cap = w.raw_cap;
  a.overflow = w.counts.as<unsigned>();
  // exact f32 form of the h = 1 prefilter (double)max(pw) - 1.0 >= threshold
  float v = (float)(c.threshold + 1.0);
  if (std::isnan(v)) v = INFINITY;
  for (int it = 0; it < 64 && (double)v - 1.0 >= c.threshold; ++it)
    v = std::nextafter(v, -INFINITY);
  for (int it = 0; it < 64 && !((double)v - 1.0 >= c.threshold); ++it)
    v = std::nextafter(v, INFINITY);
  a.t1 = v;
  for (int hi = 0; hi < 6; ++hi) {
    const double h = (double)(1 << hi), l = h + c.threshold * std::sqrt(h);
    a.lim[hi] = l > 1e-3 && l < 1e30 ? (float)(l * (1.0 - 1e-5)) : -INFINITY;
  }
  return a;
}
GateArgs gate_args(SpecWork &w, uint64_t slot0) {
  GateArgs g{};
  g.qcap = w.qcap;
  g.q1 = w.gq.as<uint32_t>() + slot0 * w.qcap;
  g.q2 = w.gq.as<uint32_t>() + (w.outer_trials + slot0) * w.qcap;
  g.xq = w.xq.as<uint32_t>() + slot0 * w.xcap;
  g.xcap = w.xcap;
  unsigned *n = w.counts.as<unsigned>() + 4 + slot0;
  g.n1 = n + w.outer_trials;
  g.n2 = n + 2 * w.outer_trials;
  g.nx = n + 3 * w.outer_trials;
  return g;
}
}  // namespace

// Normalisation scales and harmonic gates of the `ntrials` spectra at slots
// [slot0, slot0 + ntrials) of the outer chunk (d_power/d_psum point at slot0).
int spectrum_gate(const FftPlan &p, const SpecConfig &c, const float *d_power, uint64_t ldp,
                  const double *d_psum, uint32_t npsum, uint64_t ntrials, uint64_t slot0,
                  SpecWork &w, cudaStream_t st) {
  const uint64_t plen = p.M + 1;
  const uint64_t nblocks = (plen + 63) / 64;
  HarmArgs a = harm_args(p, c, d_power, ldp, w);
  GateArgs g = gate_args(w, slot0);
  PSR_CUDA(cudaFuncSetAttribute(k_scales_gate, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)SCG_SMEM));
  dim3 grid((unsigned)((nblocks + SC_G - 1) / SC_G), (unsigned)ntrials);
  float *floors = w.floors.as<float>() + slot0;
  k_floor<<<(unsigned)((ntrials + 3) / 4), 128, 0, st>>>(d_psum, npsum, ntrials, plen, floors);
  k_scales_gate<<<grid, SC_NT, SCG_SMEM, st>>>(a, floors, nblocks,
                                               w.scale.as<float>() + slot0 * w.lds, g);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

// Exact evaluation of every queued bin of the outer chunk's `ntrials` spectra,
// as many at a time as the exact lists hold.
int spectrum_items(const FftPlan &p, const SpecConfig &c, const float *d_power, uint64_t ldp,
                   uint64_t ntrials, SpecWork &w, cudaStream_t st) {
  HarmArgs a = harm_args(p, c, d_power, ldp, w);
  if (a.end[0] == 0) return PSR_OK;
  for (uint64_t t = 0; t < ntrials; t += w.xgroup) {
    const unsigned nt = (unsigned)std::min(w.xgroup, ntrials - t);
    GateArgs g = gate_args(w, t);
    g.xq = w.xq.as<uint32_t>();
    const dim3 grid(HI_CTAS_PER_TRIAL, nt);
    if (c.levels == 6) k_harm_filter<6><<<grid, HI_NT, 0, st>>>(a, g);
    else k_harm_filter<5><<<grid, HI_NT, 0, st>>>(a, g);
    k_harm_exact<<<dim3(HX_CTAS_PER_TRIAL, nt), HX_NT, 0, st>>>(a, g);
    a.power += w.xgroup * ldp;
    a.scale += w.xgroup * w.lds;
    a.raw += w.xgroup * w.raw_cap;
    a.raw_count += w.xgroup;
  }
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

// Sort/dedupe the raw candidates of `ntrials` trials into kept[][max_candidates].
int spectrum_select(const FftPlan &p, const SpecConfig &c, const double *d_trial_dm,
                    uint64_t ntrials, SpecWork &w, psr_candidate *d_kept, unsigned *d_kept_count,
                    cudaStream_t st) {
  SelArgs s{};
  s.raw = w.raw.as<RawCand>();
  s.raw_count = w.counts.as<unsigned>() + 4;
  s.raw_cap = w.raw_cap;
  s.trial_dm = d_trial_dm;
  s.tol = 1.0 / ((double)p.len * c.tsamp);
  s.max_candidates = c.max_candidates;
  s.kept = d_kept;
  s.kept_count = d_kept_count;
  k_select<<<(unsigned)ntrials, SEL_NT, 0, st>>>(s);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

}  // namespace psr
