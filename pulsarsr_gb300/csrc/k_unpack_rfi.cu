// K1 unpack (fbank::decode) and K2 RFI masking (rfi::mask) on the device.
//
// Layout: samples are channel-major, row c at c*ld, stored in their integer
// width (u8 for nbits <= 8, u16, f32).  Decisions of rfi::mask depend on the
// reference's sequential f32 sums (rfi/src/lib.rs:35-43, 59-67); every sum
// whose order matters is computed by one thread in reference order, and sums
// that are provably exact (integer samples, total <= 2^24) are computed in
// parallel, which gives the identical f32 value.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "psr_internal.h"

namespace psr {

namespace {

constexpr int UNPACK_TT = 256;  // times per tile (16-bit and f32 samples)
constexpr int UNPACK_TC = 32;   // channels per tile

template <class T>
__global__ void k_unpack(const T *__restrict__ payload, T *__restrict__ out, uint64_t ns,
                         uint64_t nch, uint64_t ld, unsigned long long *err_index) {
  __shared__ T tile[UNPACK_TC][UNPACK_TT + 4];
  const uint64_t t0 = (uint64_t)blockIdx.x * UNPACK_TT;
  const uint64_t c0 = (uint64_t)blockIdx.y * UNPACK_TC;
  for (int idx = threadIdx.x; idx < UNPACK_TT * UNPACK_TC; idx += blockDim.x) {
    int tl = idx / UNPACK_TC, cl = idx % UNPACK_TC;
    uint64_t t = t0 + tl, c = c0 + cl;
    T v = T(0);
    if (t < ns && c < nch) {
      uint64_t i = t * nch + c;
      v = payload[i];  // little endian, as the file
      if constexpr (sizeof(T) == 4) {
        if (!isfinite(v)) atomicMin(err_index, (unsigned long long)i);
      }
    }
    tile[cl][tl] = v;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < UNPACK_TT * UNPACK_TC; idx += blockDim.x) {
    int cl = idx / UNPACK_TT, tl = idx % UNPACK_TT;
    uint64_t t = t0 + tl, c = c0 + cl;
    if (t < ns && c < nch) out[c * ld + t] = tile[cl][tl];
  }
}

// Samples of at most 8 bits: tiles of 128 channels x 128 times.  SIGPROC packs
// low-bit samples LSB first (fbank/src/lib.rs:175-179), so the payload is one
// little-endian bit stream and the samples of four adjacent channels are 4 B
// consecutive bits of it, at any bit offset: two 32-bit loads and a funnel
// shift, spread to a byte each.  A thread turns four times of four channels
// (a 4 x 4 byte block, 8 byte permutes) and stores a word of four times per
// channel; column q of channel ch sits at (q + ch / 32) mod 32 of its 33-word
// row, which keeps the 32 lanes' stores (channels 4 l + i) in 32 banks.
// Bound: HBM, payload read and samples written once.  Measured on a GB300: 512
// 8-bit channels of 1,047,799 samples (1.07 GB moved) 0.86 ms with one byte per
// thread and access, 0.34 with a bit address per word, 0.19 with whole words
// where the channel count is a multiple of 4; 96 4-bit channels of 531,000
// samples 0.100 and 0.037.
constexpr int UP_T = 128, UP_C = 128, UP_NT = 256;

template <int B>
__device__ __forceinline__ uint32_t spread_bits(uint32_t v) {
  if constexpr (B == 8) return v;
  if constexpr (B == 4) {
    v &= 0xffffu;
    v = (v | v << 8) & 0x00ff00ffu;
    return (v | v << 4) & 0x0f0f0f0fu;
  }
  if constexpr (B == 2) {
    v &= 0xffu;
    v = (v | v << 12) & 0x000f000fu;
    return (v | v << 6) & 0x03030303u;
  }
  v &= 0xfu;
  v = (v | v << 14) & 0x00030003u;
  return (v | v << 7) & 0x01010101u;
}

template <int B>
__global__ void __launch_bounds__(UP_NT)
    k_unpack8(const uint32_t *__restrict__ payload, uint8_t *__restrict__ out, uint64_t ns,
              uint64_t nch, uint64_t ld) {
  __shared__ uint32_t tile[UP_C * 33];
  const uint64_t t0 = (uint64_t)blockIdx.x * UP_T, c0 = (uint64_t)blockIdx.y * UP_C;
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  const uint64_t c = c0 + 4 * lane;  // lane's four channels
  // channels past the last are zeroed (their bits belong to the next time)
  const uint32_t cmask = c + 4 <= nch ? 0xffffffffu
                         : c < nch    ? 0xffffffffu >> (8 * (4 - (int)(nch - c)))
                                      : 0u;
  const bool words = nch % 4 == 0;
  const uint64_t step = nch * B, bit0 = ((t0 + 4 * warp) * nch + c) * B;
#pragma unroll
  for (int h = 0; h < UP_T / 4 / (UP_NT / 32); ++h) {
    const int q = warp + h * (UP_NT / 32);
    uint32_t v[4];
    if (B == 8 && words) {  // four channels of a time are a word of the payload
      const uint64_t t = t0 + 4 * q;
      const uint32_t *w = payload + (t * nch + c) / 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[i] = t + i < ns && cmask ? __ldg(w + i * (nch / 4)) : 0u;
    } else
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t t = t0 + 4 * q + i;
      uint32_t x = 0;
      if (t < ns && cmask) {
        const uint64_t bit = bit0 + (uint64_t)(32 * h + i) * step;
        const uint32_t *w = payload + (bit >> 5);
        const unsigned sh = (unsigned)bit & 31u;
        // the second word only where the 4 B bits reach it (it may be the
        // payload's 16 bytes of slack)
        const uint32_t lo = __ldg(w), hi = sh + 4 * B > 32 ? __ldg(w + 1) : 0u;
        x = spread_bits<B>(__funnelshift_r(lo, hi, sh)) & cmask;
      }
      v[i] = x;
    }
    const uint32_t a = __byte_perm(v[0], v[1], 0x5140), b = __byte_perm(v[2], v[3], 0x5140);
    const uint32_t d = __byte_perm(v[0], v[1], 0x7362), e = __byte_perm(v[2], v[3], 0x7362);
    uint32_t *p = tile + 4 * lane * 33 + ((q + (lane >> 3)) & 31);
    p[0] = __byte_perm(a, b, 0x5410);
    p[33] = __byte_perm(a, b, 0x7632);
    p[66] = __byte_perm(d, e, 0x5410);
    p[99] = __byte_perm(d, e, 0x7632);
  }
  __syncthreads();
  // one warp per channel row: 32 words of four times
  const uint64_t t = t0 + 4 * lane;
  for (int ch = warp; ch < UP_C && c0 + ch < nch; ch += UP_NT / 32)
    if (t < ns)  // (a last word's samples past ns are zero, as the row's padding)
      *reinterpret_cast<uint32_t *>(out + (c0 + ch) * ld + t) =
          tile[ch * 33 + ((lane + (ch >> 5)) & 31)];
}

// ------------------------------------------------------------ radix select
// Total-order key of an f32 (Rust f32::total_cmp) as an unsigned integer.
__device__ __forceinline__ uint32_t fkey(float f) {
  uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Block-wide exact selection of the element of rank r (ascending) among n
// keys key(i); top_shift is the shift of the highest non-constant digit.
// Each warp counts digits in its own histogram (hist holds 32 x 256 slots),
// so few-valued data (4-bit samples) does not serialise on a handful of bins.
template <class KeyFn>
__device__ uint32_t block_select(KeyFn key, uint64_t n, uint64_t r, int top_shift,
                                 unsigned *hist, uint32_t *bcast) {
  const int nw = (int)(blockDim.x + 31) / 32;
  unsigned *mine = hist + (threadIdx.x >> 5) * 256;
  uint32_t prefix = 0, mask = 0;
  for (int shift = top_shift; shift >= 0; shift -= 8) {
    for (int d = threadIdx.x; d < nw * 256; d += blockDim.x) hist[d] = 0;
    __syncthreads();
    for (uint64_t i = threadIdx.x; i < n; i += blockDim.x) {
      uint32_t k = key(i);
      if ((k & mask) == prefix) atomicAdd(&mine[(k >> shift) & 255u], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += blockDim.x) {
      unsigned t = 0;
      for (int w = 0; w < nw; ++w) t += hist[w * 256 + d];
      hist[d] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t cum = 0;
      uint32_t digit = 255;
      for (int d = 0; d < 256; ++d) {
        if (cum + hist[d] > r) {
          digit = (uint32_t)d;
          break;
        }
        cum += hist[d];
      }
      r -= cum;
      bcast[0] = digit;
      bcast[1] = (uint32_t)(r & 0xffffffffu);
      bcast[2] = (uint32_t)(r >> 32);
    }
    __syncthreads();
    uint32_t digit = bcast[0];
    r = (uint64_t)bcast[1] | ((uint64_t)bcast[2] << 32);
    prefix |= digit << shift;
    mask |= 255u << shift;
    __syncthreads();
  }
  return prefix;
}

__global__ void k_median_f32(const float *__restrict__ v, uint64_t n, float *out) {
  __shared__ unsigned hist[32 * 256];
  __shared__ uint32_t bc[3];
  if (n == 0) {
    if (threadIdx.x == 0) *out = 0.0f;
    return;
  }
  uint32_t k = block_select([&](uint64_t i) { return fkey(v[i]); }, n, n / 2, 24, hist, bc);
  if (threadIdx.x == 0) *out = fkey_inv(k);
}

// Per-channel exact median of the original row (rfi/src/lib.rs:78) of 16-bit
// and f32 samples: a digit of the keys per launch, highest first.  CTAs of
// MD_PER samples count the digits of the keys that match the digits found so far
// in shared memory (in four copies: the top digit of f32 noise has a few values)
// and add their counts to the channel's; the last CTA of a channel to arrive finds
// the digit that holds the rank and clears the counts for the next launch.
// state[c]: rank left, digits found, CTAs arrived.
// Bound: shared-memory atomics, then the reads (three passes for f32, two for
// 16-bit samples).  Measured on a GB300: 32 f32 channels of 65,536 samples, one
// CTA per channel with four 8-bit digits: 125 us, 28 now; 512 16-bit channels of
// 1,047,799: 1.96 ms, 0.85 now.
constexpr int MD_BITS = 11, MD_NT = 256, MD_COPIES = 4;
constexpr int MD_PER = 16384;
struct MedianState {
  unsigned long long rank;
  uint32_t prefix;
  unsigned arrived;
};
template <class T>
__device__ __forceinline__ uint32_t sample_key(T v) {
  if constexpr (sizeof(T) == 4) return fkey(v);
  else return (uint32_t)v;
}
template <class T>
__global__ void __launch_bounds__(MD_NT)
    k_median_digit(const T *__restrict__ s, uint64_t ns, uint64_t ld, int shift, int bits,
                   unsigned *__restrict__ hist, MedianState *__restrict__ state,
                   float *__restrict__ med) {
  __shared__ unsigned h[(1 << MD_BITS) * MD_COPIES];
  __shared__ unsigned wsum[MD_NT / 32];
  __shared__ int last;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t c = blockIdx.y;
  const int nb = 1 << bits;
  const bool first = shift + bits >= 8 * (int)sizeof(T);
  const unsigned long long rank = first ? ns / 2 : state[c].rank;
  const uint32_t prefix = first ? 0u : state[c].prefix;
  for (int i = tid; i < nb * MD_COPIES; i += MD_NT) h[i] = 0;
  __syncthreads();
  // (rows are 64-element aligned and padded: whole 16-byte loads stay in the row)
  constexpr int PER = 16 / (int)sizeof(T);
  const T *row = s + c * ld;
  const uint64_t a = (uint64_t)blockIdx.x * MD_PER, b = min(ns, a + MD_PER);
  for (uint64_t i = a + (uint64_t)tid * PER; i < b; i += MD_NT * PER) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + i));
    T e[PER];
    memcpy(e, &v, 16);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const uint32_t key = sample_key(e[k]);
      // the digits above this one agree
      if (i + k < b && (first || key >> (shift + bits) == prefix))
        atomicAdd(&h[(key >> shift & (nb - 1)) * MD_COPIES + (lane & (MD_COPIES - 1))], 1u);
    }
  }
  __syncthreads();
  unsigned *hc = hist + c * (1 << MD_BITS);
  for (int i = tid; i < nb; i += MD_NT) {
    unsigned t = 0;
#pragma unroll
    for (int k = 0; k < MD_COPIES; ++k) t += h[i * MD_COPIES + k];
    if (t) atomicAdd(&hc[i], t);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&state[c].arrived, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the first digit at which the running count passes the rank
  const int per = max(nb / MD_NT, 1);
  unsigned t = 0;
  for (int k = 0; k < per; ++k)
    if (tid * per + k < nb) t += __ldcg(&hc[tid * per + k]);
  unsigned inc = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  unsigned long long cum = inc - t;
  for (int w = 0; w < warp; ++w) cum += wsum[w];
  if (rank >= cum && rank < cum + t) {  // one thread
    int d = tid * per;
    for (unsigned n; rank >= cum + (n = __ldcg(&hc[d])); ++d) cum += n;
    const uint32_t found = prefix << bits | (uint32_t)d;
    if (shift == 0) {
      if constexpr (sizeof(T) == 4) med[c] = fkey_inv(found);
      else med[c] = (float)found;
    }
    state[c] = MedianState{rank - cum, found, 0u};
  }
  __syncthreads();
  for (int i = tid; i < nb; i += MD_NT) hc[i] = 0;
}

// 8-bit rows: the median from a 256-bin histogram (one pass).  Each row is
// split over several CTAs; a CTA's table has a column per lane, so that a warp's 32
// counts, shared-memory atomics without a result, always fall in 32 banks.
// Bound: the atomics, one per 32 samples.
// Measured on a GB300: 512 channels of 1,047,799 samples 0.52 ms with 16-bit
// columns per thread, 0.27 with byte columns, read, incremented and written,
// that were added up before they could overflow, 0.21 now; 64 channels of 262,144
// samples 17 us, 11 now.
constexpr int MH_NT = 256, MH_COL = 32;
constexpr uint64_t MH_MIN = 16384, MH_MAX = 131072;  // samples per CTA

__global__ void __launch_bounds__(MH_NT)
    k_chan_hist_u8(const uint8_t *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t per,
                   unsigned *__restrict__ hist) {
  __shared__ unsigned h[256 * MH_COL];
  const int tid = (int)threadIdx.x;
  unsigned *mine = h + (tid & (MH_COL - 1));
  const uint8_t *row = s + (uint64_t)blockIdx.y * ld;
  // this CTA's range [a, b), a a multiple of 16 (rows are 64-byte aligned
  // and padded by >= 64 bytes, so whole 16-byte loads stay in the row)
  const uint64_t a = (uint64_t)blockIdx.x * per, b = min(ns, a + per);
#pragma unroll
  for (int i = tid; i < 256 * MH_COL / 4; i += MH_NT)
    reinterpret_cast<uint4 *>(h)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
#pragma unroll 2
  for (uint64_t i = a + (uint64_t)tid * 16; i < b; i += (uint64_t)MH_NT * 16) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + i));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const int m = (int)min((uint64_t)16, b - i);
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < m) atomicAdd(&mine[((w[k >> 2] >> (8 * (k & 3))) & 255u) * MH_COL], 1u);
  }
  __syncthreads();
  unsigned total = 0;  // of bin tid
#pragma unroll 8
  for (int j = 0; j < MH_COL; ++j) total += h[tid * MH_COL + ((j + tid) & (MH_COL - 1))];
  if (total) atomicAdd(&hist[(uint64_t)blockIdx.y * 256 + tid], total);
}

// Element of rank ns / 2 from each row's histogram: one warp per channel, 8 bins
// per lane, a prefix over the lanes.
__global__ void __launch_bounds__(128)
    k_hist_median(const unsigned *__restrict__ hist, uint64_t nch, uint64_t ns,
                  float *__restrict__ med) {
  const uint64_t c = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (c >= nch) return;
  const int lane = (int)(threadIdx.x & 31);
  const unsigned long long r = ns / 2;
  unsigned h[8];
  unsigned long long t = 0;
  const uint4 *q = reinterpret_cast<const uint4 *>(hist + c * 256 + 8 * lane);
  *reinterpret_cast<uint4 *>(h) = q[0];
  *reinterpret_cast<uint4 *>(h + 4) = q[1];
#pragma unroll
  for (int k = 0; k < 8; ++k) t += h[k];
  unsigned long long cum = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, cum, o);
    if (lane >= o) cum += v;
  }
  const unsigned past = __ballot_sync(0xffffffffu, cum > r);
  if (lane != (past ? __ffs((int)past) - 1 : 31)) return;
  cum -= t;
  int d = 8 * lane + 7;
#pragma unroll
  for (int k = 7; k >= 0; --k) {
    unsigned long long upto = cum;
    for (int j = 0; j <= k; ++j) upto += h[j];
    if (upto > r) d = 8 * lane + k;
  }
  med[c] = (float)d;
}

template <class T>
__device__ __forceinline__ float as_f32(T v) {
  return (float)v;
}

// A sum of f32 samples in the reference's order where it can fall (negative
// samples): the per-sample work is taken off the sequential chain, one CTA
// per channel; warps 1.. write the next segment into a shared-memory double
// buffer while thread 0 adds the current one.  The chain then costs one FADD
// latency per sample.
constexpr int PC_NT = 256;
constexpr int PC_SEG = 2048;

template <class T, class Term>
__device__ float pc_sequential_sum(const T *row, uint64_t ns, float *buf, Term term) {
  const uint64_t nseg = (ns + PC_SEG - 1) / PC_SEG;
  float acc = -0.0f;
  constexpr int NP = PC_NT - 32;                 // producer threads
  constexpr int NI = (PC_SEG + NP - 1) / NP;     // samples per producer thread
  auto produce = [&](uint64_t seg, float *dst) {
    const uint64_t t0 = seg * PC_SEG;
    const int cnt = (int)min((uint64_t)PC_SEG, ns - t0);
    float v[NI];
#pragma unroll
    for (int u = 0; u < NI; ++u) {  // all loads issued before any is used
      const int i = (int)threadIdx.x - 32 + u * NP;
      v[u] = i < cnt ? as_f32(row[t0 + i]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int i = (int)threadIdx.x - 32 + u * NP;
      if (i < cnt) dst[i] = term(v[u]);
    }
  };
  if (threadIdx.x >= 32) produce(0, buf);
  __syncthreads();
  for (uint64_t seg = 0; seg < nseg; ++seg) {
    float *cur = buf + (seg & 1) * PC_SEG;
    if (threadIdx.x >= 32) {
      if (seg + 1 < nseg) produce(seg + 1, buf + ((seg + 1) & 1) * PC_SEG);
    } else if (threadIdx.x == 0) {
      const int cnt = (int)min((uint64_t)PC_SEG, ns - seg * PC_SEG);
      const float4 *c4 = reinterpret_cast<const float4 *>(cur);
      int i = 0;
#pragma unroll 8
      for (; i + 4 <= cnt; i += 4) {
        const float4 q = c4[i >> 2];
        acc = __fadd_rn(acc, q.x);
        acc = __fadd_rn(acc, q.y);
        acc = __fadd_rn(acc, q.z);
        acc = __fadd_rn(acc, q.w);
      }
      for (; i < cnt; ++i) acc = __fadd_rn(acc, cur[i]);
    }
    __syncthreads();
  }
  return acc;  // valid in thread 0
}

// Reference-order f32 sums of non-negative terms, s = RN(...RN(RN(-0 + t0) +
// t1)... + t_{n-1}), bit for bit, in parallel.  While s stays in one binade
// [2^e, 2^(e+1)) every representable value is a multiple of u = 2^(e-23), so
// s = K u (2^23 <= K < 2^24) and RN(s + t) = (K + inc(t)) u with inc(t) =
// t/u rounded to nearest: the integer part q of t/u plus one when its
// fraction exceeds 1/2.  An exact half (a tie) rounds to even: inc = q +
// ((K + q) mod 2), so it depends on the running K through its parity alone.
// A run of terms is therefore a map from K's parity to an increment, (d0, d1),
// and maps compose: after (a0, a1), (b0, b1) adds b0 or b1 by the parity of
// what stands then.  t >= 0 makes K monotone: a run whose increment keeps
// K + d < 2^24 is added at once.
//
// The binade is not known before the sum is, but it can be guessed from plain
// sums of the terms.  So the pass over the samples is parallel over the whole
// card, and only a scan over chunks of 512 terms is left per channel:
//   k_es_sums   plain sums of every chunk's samples and their squares
//   k_es_guess  binades of the mean's running sum at every chunk
//   k_es_maps   the map of every chunk at its guessed binade
//   k_es_scan   one warp per channel: composes 32 chunks' maps at a time;
//               a chunk whose guess is wrong, or that leaves its binade, is
//               taken apart into its lanes' 16 terms (maps again at the true
//               binade, the lane that crosses term by term)
// and the last two again for the variance, whose binades follow from the mean
// and the plain sums.  An infinite or NaN term makes a run special: it is added
// term by term.
constexpr int ES_L = 512;          // terms per chunk, 16 per lane
constexpr int ES_PER = ES_L / 32;
constexpr uint32_t ES_SPECIAL = 0xffffffffu;

// Lane l's 16 consecutive samples of a chunk: aligned 16-byte loads (rows
// start 64-element aligned; only issued for samples below ns, whose 16-sample
// run then ends inside the row's padding).
template <class T>
struct EsRaw {
  static constexpr int W = (int)sizeof(T);
  uint4 r[W];
  __device__ __forceinline__ void load(const T *p, bool ok) {
#pragma unroll
    for (int k = 0; k < W; ++k)
      r[k] = ok ? __ldg(reinterpret_cast<const uint4 *>(p) + k) : make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ uint32_t word(int i) const {
    const uint4 &q = r[i >> 2];
    return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
  }
  __device__ __forceinline__ float at(int j) const {
    // integers exactly: 2^23 + v assembled by a byte permute, less 2^23
    if constexpr (sizeof(T) == 1)
      return __uint_as_float(__byte_perm(word(j >> 2), 0x4B000000u, 0x7540u | (j & 3))) -
             8388608.0f;
    else if constexpr (sizeof(T) == 2)
      return __uint_as_float(
                 __byte_perm(word(j >> 1), 0x4B000000u, (j & 1) ? 0x7532u : 0x7510u)) -
             8388608.0f;
    else return __uint_as_float(word(j));
  }
};

// The map (d0, d1) of N terms >= 0 at the binade with biased exponent be (1 to
// 254); true if the run does not fit it (it adds 2^23 units or more, or a term
// is infinite or NaN).  The f32 unit makes the map: two running sums, from
// the binade's first value (K = 2^23, even) and its second (odd), see the
// roundings of any even and odd K as long as they stay in the binade.
template <int N>
__device__ __forceinline__ bool es_run(const float (&t)[N], int be, uint32_t &d0, uint32_t &d1) {
  const uint32_t k0 = (uint32_t)be << 23;
  float s0 = __uint_as_float(k0), s1 = __uint_as_float(k0 + 1);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    s0 = __fadd_rn(s0, t[j]);
    s1 = __fadd_rn(s1, t[j]);
  }
  const uint32_t b0 = __float_as_uint(s0), b1 = __float_as_uint(s1);
  d0 = b0 - k0;
  d1 = b1 - k0 - 1;
  return (int)(b0 >> 23) != be || (int)(b1 >> 23) != be;
}

// Inclusive scan of the lanes' maps.
__device__ __forceinline__ void es_scan_maps(uint32_t &d0, uint32_t &d1, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a0 = __shfl_up_sync(0xffffffffu, d0, o);
    const uint32_t a1 = __shfl_up_sync(0xffffffffu, d1, o);
    if (lane >= o) {
      const uint32_t b0 = d0, b1 = d1;
      d0 = a0 + ((a0 & 1u) ? b1 : b0);
      d1 = a1 + ((a1 & 1u) ? b0 : b1);
    }
  }
}

// Adds the longest prefix of the lanes [cur, 32) with `valid` maps that keeps
// s in its binade (biased exponent be, normal); returns the first lane left.
__device__ __forceinline__ int es_advance(float &s, int be, bool valid, uint32_t m0, uint32_t m1,
                                          int cur, int lane) {
  const unsigned vm = __ballot_sync(0xffffffffu, valid && lane >= cur) >> cur;
  const int run = vm == 0xffffffffu ? 32 : __ffs(~vm) - 1;
  const bool in = lane >= cur && lane < cur + run;
  uint32_t d0 = in ? m0 : 0u, d1 = in ? m1 : 0u;
  es_scan_maps(d0, d1, lane);
  const uint32_t K = (__float_as_uint(s) & 0x7fffffu) | 0x800000u;
  const uint32_t Kn = K + ((K & 1u) ? d1 : d0);
  const int nok = __popc(__ballot_sync(0xffffffffu, in && Kn < (1u << 24)));
  if (nok) {
    const uint32_t Kl = __shfl_sync(0xffffffffu, Kn, cur + nok - 1);
    s = __uint_as_float((uint32_t)be << 23 | (Kl & 0x7fffffu));
  }
  return cur + nok;
}

// One chunk by a warp: lane l holds terms 16 l .. 16 l + 15 of it (cnt valid
// terms in all); returns s, in every lane.
__device__ __noinline__ float es_chunk(const float (&t)[ES_PER], int cnt, float s, int lane) {
  int cur = 0;
  while (cur < 32) {
    const int be = (int)(__float_as_uint(s) >> 23);
    if (be > 0 && be < 255) {
      uint32_t d0, d1;
      const bool bad = es_run(t, be, d0, d1);
      cur = es_advance(s, be, !bad, d0, d1, cur, lane);
      if (cur == 32) break;
    }
#pragma unroll
    for (int j = 0; j < ES_PER; ++j) {
      const float v = __shfl_sync(0xffffffffu, t[j], cur);
      if (cur * ES_PER + j < cnt) s = __fadd_rn(s, v);
    }
    ++cur;
  }
  return s;
}

// Plain sums per chunk: sum[] exact for integer samples (32 bits hold 512
// 16-bit samples), sq[] and the f32 sums rounded (they only guess binades).
// neg[c] is set when a channel holds a negative (or NaN) f32 sample.
// Bound: HBM, one read of the samples.
constexpr int EK_NT = 256, EK_CPW = 4;  // chunks per warp
template <class T>
__global__ void __launch_bounds__(EK_NT)
    k_es_sums(const T *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t nck,
              uint32_t *__restrict__ sum, float *__restrict__ sq, unsigned *__restrict__ neg) {
  const int lane = (int)(threadIdx.x & 31);
  const T *row = s + (uint64_t)blockIdx.y * ld;
  const uint64_t k0 = ((uint64_t)blockIdx.x * (EK_NT / 32) + (threadIdx.x >> 5)) * EK_CPW;
  EsRaw<T> x[EK_CPW];
#pragma unroll
  for (int i = 0; i < EK_CPW; ++i) {
    const uint64_t p = (k0 + i) * ES_L + (uint64_t)lane * ES_PER;
    x[i].load(row + p, p < ns);
  }
  bool below = false;
#pragma unroll
  for (int i = 0; i < EK_CPW; ++i) {
    const uint64_t k = k0 + i;
    if (k >= nck) break;  // (warp-uniform)
    const uint64_t at = (uint64_t)blockIdx.y * nck + k;  // (samples past ns are zero)
    if constexpr (sizeof(T) == 1) {
      unsigned a = 0, q = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        a = __dp4a(x[i].word(w), 0x01010101u, a);
        q = __dp4a(x[i].word(w), x[i].word(w), q);
      }
      a = __reduce_add_sync(0xffffffffu, a);
      q = __reduce_add_sync(0xffffffffu, q);
      if (lane == 0) {
        sum[at] = a;
        sq[at] = (float)q;
      }
    } else if constexpr (sizeof(T) == 2) {
      unsigned a = 0;
      float q = 0.0f;
#pragma unroll
      for (int j = 0; j < ES_PER; ++j) {
        const float v = x[i].at(j);
        a += (unsigned)v;
        q = __fmaf_rn(v, v, q);
      }
      a = __reduce_add_sync(0xffffffffu, a);
      for (int o = 16; o; o >>= 1) q += __shfl_down_sync(0xffffffffu, q, o);
      if (lane == 0) {
        sum[at] = a;
        sq[at] = q;
      }
    } else {
      float a = 0.0f, q = 0.0f;
#pragma unroll
      for (int j = 0; j < ES_PER; ++j) {
        const float v = x[i].at(j);
        below |= !(v >= 0.0f);
        a += v;
        q = __fmaf_rn(v, v, q);
      }
      for (int o = 16; o; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        q += __shfl_down_sync(0xffffffffu, q, o);
      }
      if (lane == 0) {
        sum[at] = __float_as_uint(a);
        sq[at] = q;
      }
    }
  }
  if (sizeof(T) == 4 && __any_sync(0xffffffffu, below) && lane == 0) atomicOr(&neg[blockIdx.y], 1u);
}

// Plain sums run in integers (exact) for integer samples and in f32 otherwise
// (FP64 runs at 1/64 rate here; only the binade is wanted).
template <class T>
struct EsPlain {
  typedef unsigned long long type;
  static __device__ __forceinline__ type of(uint32_t v) { return v; }
};
template <>
struct EsPlain<float> {
  typedef float type;
  static __device__ __forceinline__ float of(uint32_t v) { return __uint_as_float(v); }
};
// Biased f32 exponent of a prefix (0: no guess).
__device__ __forceinline__ uint8_t es_binade(float p) {
  const uint32_t b = __float_as_uint(p) >> 23;
  return b > 0 && b < 255 ? (uint8_t)b : (uint8_t)0;
}

// Binades at the start of every chunk of one channel's running sum of chunk
// sums f(k), by a CTA of EG_NT threads; returns the total in every thread.
constexpr int EG_NT = 256;
template <class A, class F>
__device__ A es_guess(uint64_t nck, F f, uint8_t *__restrict__ out, A *red) {
  // contiguous chunks per thread: its sum, a scan of the threads' sums, then
  // its running sums
  const uint64_t per = (nck + EG_NT - 1) / EG_NT;
  const uint64_t a = min((uint64_t)threadIdx.x * per, nck), b = min(a + per, nck);
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  A t = 0;
  for (uint64_t k = a; k < b; ++k) t += f(k);
  A inc = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const A v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  __syncthreads();  // red may still be read by an earlier call
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  A p = inc - t, tot = 0;
  for (int i = 0; i < EG_NT / 32; ++i) {
    if (i < warp) p += red[i];
    tot += red[i];
  }
  for (uint64_t k = a; k < b; ++k) {
    out[k] = es_binade((float)p);
    p += f(k);
  }
  return tot;
}

// What a channel's mean needs: 0 its exact integer total (at most 2^24, every
// partial sum exact), 1 the maps, 2 the sequential sum (negative samples).
struct EsChan {
  int mode;
};

template <class T>
__device__ void es_guess_var(const uint32_t *sum, const float *sq, uint64_t nck, uint64_t ns,
                             float m, uint8_t *guess, float *red) {
  es_guess<float>(nck, [&](uint64_t k) {
    const float cnt = (float)min((uint64_t)ES_L, ns - k * ES_L);
    const float a = (float)EsPlain<T>::of(sum[k]);
    return fmaxf(__fmaf_rn(m, __fmaf_rn(cnt, m, -2.0f * a), sq[k]), 0.0f);
  }, guess, red);
}

// One CTA per channel: the mean's binades, or the mean itself where the total
// is exact (then the variance's binades).
template <class T>
__global__ void __launch_bounds__(EG_NT)
    k_es_guess(const uint32_t *__restrict__ sum, const float *__restrict__ sq,
               const unsigned *__restrict__ neg, uint64_t nck, uint64_t ns,
               uint8_t *__restrict__ guess, EsChan *__restrict__ chan,
               float *__restrict__ means) {
  typedef typename EsPlain<T>::type A;
  __shared__ A red[EG_NT / 32];
  __shared__ float redf[EG_NT / 32];
  const uint64_t c = blockIdx.x;
  sum += c * nck;
  sq += c * nck;
  guess += c * nck;
  const A tot = es_guess<A>(nck, [&](uint64_t k) { return EsPlain<T>::of(sum[k]); }, guess, red);
  int mode = 1;
  if (sizeof(T) < 4 && tot <= (A)16777216) mode = 0;
  if (sizeof(T) == 4 && neg[c]) mode = 2;
  const float m = __fdiv_rn((float)tot, (float)ns);
  if (threadIdx.x == 0) {
    chan[c].mode = mode;
    if (mode == 0) means[c] = m;
  }
  if (mode == 0) es_guess_var<T>(sum, sq, nck, ns, m, guess, redf);
}

template <bool VAR>
__device__ __forceinline__ float es_term(float x, float m) {
  if constexpr (!VAR) return x;
  const float d = __fsub_rn(x, m);
  return __fmul_rn(d, d);
}

// The map of every chunk at its guessed binade.
// Bound: issue, about 8 instructions per sample, twice the time of the bytes.
// Measured on a GB300 (512 8-bit channels of 1,047,799 samples, means above
// 2^24): the six kernels 0.59 ms, 0.20 and 0.17 of them in the two passes of
// k_es_maps (0.88 each with the increments computed in integers, bound by the
// half-rate pipe); one CTA per channel that walked its chunks in order took 6.4
// with its totals.
template <class T, bool VAR>
__global__ void __launch_bounds__(EK_NT)
    k_es_maps(const T *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t nck,
              const uint8_t *__restrict__ guess, const EsChan *__restrict__ chan,
              const float *__restrict__ means, uint2 *__restrict__ maps) {
  const uint64_t c = blockIdx.y;
  if (!VAR && chan[c].mode != 1) return;
  const int lane = (int)(threadIdx.x & 31);
  const T *row = s + c * ld;
  const float m = VAR ? means[c] : 0.0f;
  const uint64_t k0 = ((uint64_t)blockIdx.x * (EK_NT / 32) + (threadIdx.x >> 5)) * EK_CPW;
  const uint64_t whole = ns / ES_L;  // chunks of 512 terms
  EsRaw<T> nx;
  {
    const uint64_t p = k0 * ES_L + (uint64_t)lane * ES_PER;
    nx.load(row + p, p < ns);
  }
  for (int i = 0; i < EK_CPW; ++i) {
    const uint64_t k = k0 + i;
    if (k >= nck) break;
    const uint64_t p = k * ES_L + (uint64_t)lane * ES_PER;
    const EsRaw<T> x = nx;
    if (i + 1 < EK_CPW) nx.load(row + p + ES_L, p + ES_L < ns);
    const int be = (int)guess[c * nck + k];
    uint2 out = make_uint2(ES_SPECIAL, ES_SPECIAL);
    if (be) {
      float t[ES_PER];
#pragma unroll
      for (int j = 0; j < ES_PER; ++j) t[j] = es_term<VAR>(x.at(j), m);
      if (k >= whole) {
        const int left = p < ns ? (int)min((uint64_t)ES_PER, ns - p) : 0;
#pragma unroll
        for (int j = 0; j < ES_PER; ++j)
          if (j >= left) t[j] = 0.0f;
      }
      uint32_t d0, d1;
      const bool bad = es_run(t, be, d0, d1);
      if (!__any_sync(0xffffffffu, bad)) {
        if (!__any_sync(0xffffffffu, d0 != d1)) {  // no lane depends on the parity
          d0 = d1 = __reduce_add_sync(0xffffffffu, d0);
        } else {
          es_scan_maps(d0, d1, lane);
          d0 = __shfl_sync(0xffffffffu, d0, 31);
          d1 = __shfl_sync(0xffffffffu, d1, 31);
        }
        if (d0 < (1u << 24) && d1 < (1u << 24)) out = make_uint2(d0, d1);
      }
    }
    if (lane == 0) maps[c * nck + k] = out;
  }
}

// The running sum over a channel's chunks; the mean (then the variance's
// binades) or the variance.  One CTA per channel, the scan by its first warp.
template <class T, bool VAR>
__global__ void __launch_bounds__(EG_NT)
    k_es_scan(const T *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t nck,
              const uint32_t *__restrict__ sum, const float *__restrict__ sq,
              uint8_t *__restrict__ guess, const EsChan *__restrict__ chan,
              const uint2 *__restrict__ maps, float *__restrict__ means,
              float *__restrict__ vars) {
  __shared__ float red[EG_NT / 32];
  __shared__ float mean_s;
  const uint64_t c = blockIdx.x;
  if (!VAR && chan[c].mode == 0) return;
  guess += c * nck;
  maps += c * nck;
  const T *row = s + c * ld;
  if (threadIdx.x < 32 && (VAR || chan[c].mode == 1)) {
    const int lane = (int)threadIdx.x;
    const float m = VAR ? means[c] : 0.0f;
    float acc = -0.0f;
    uint2 nm = make_uint2(ES_SPECIAL, ES_SPECIAL);
    int nb = 0;
    if (lane < (int)min((uint64_t)32, nck)) {
      nm = maps[lane];
      nb = (int)guess[lane];
    }
    for (uint64_t g0 = 0; g0 < nck; g0 += 32) {
      const int cnt = (int)min((uint64_t)32, nck - g0);
      const uint2 mp = nm;
      const int gb = nb;
      if (g0 + 32 + lane < nck) {
        nm = maps[g0 + 32 + lane];
        nb = (int)guess[g0 + 32 + lane];
      }
      int cur = 0;
      while (cur < cnt) {
        const int be = (int)(__float_as_uint(acc) >> 23);
        if (be > 0 && be < 255) {
          const bool valid = lane < cnt && gb == be && mp.x != ES_SPECIAL;
          cur = es_advance(acc, be, valid, mp.x, mp.y, cur, lane);
          if (cur >= cnt) break;
        }
        const uint64_t k = g0 + cur, p = k * ES_L + (uint64_t)lane * ES_PER;
        EsRaw<T> x;
        x.load(row + p, p < ns);
        float t[ES_PER];
#pragma unroll
        for (int j = 0; j < ES_PER; ++j) t[j] = p + j < ns ? es_term<VAR>(x.at(j), m) : 0.0f;
        acc = es_chunk(t, (int)min((uint64_t)ES_L, ns - k * ES_L), acc, lane);
        ++cur;
      }
    }
    if (lane == 0) {
      const float v = __fdiv_rn(acc, (float)ns);
      if (VAR) {
        vars[c] = v;
      } else {
        means[c] = v;
        mean_s = v;
      }
    }
  }
  if constexpr (!VAR) {
    __shared__ __align__(16) float buf[sizeof(T) == 4 ? 2 * PC_SEG : 4];
    if constexpr (sizeof(T) == 4) {
      if (chan[c].mode == 2) {
        const float a = pc_sequential_sum(row, ns, buf, [](float x) { return x; });
        if (threadIdx.x == 0) {
          mean_s = __fdiv_rn(a, (float)ns);
          means[c] = mean_s;
        }
      }
    }
    (void)buf;
    __syncthreads();
    es_guess_var<T>(sum + c * nck, sq + c * nck, nck, ns, mean_s, guess, red);
  }
}

// Per-(channel, block) sequential f32 sums (rfi/src/lib.rs:62-64).
template <class T>
__global__ void k_block_sums(const T *__restrict__ s, uint64_t ns, uint64_t ld,
                             uint64_t nch, uint64_t bs, uint64_t blocks_n,
                             float *__restrict__ bsum) {
  uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= nch * blocks_n) return;
  uint64_t c = id / blocks_n, b = id % blocks_n;
  uint64_t start = b * bs, end = min(start + bs, ns);
  const T *row = s + c * ld;
  float acc = -0.0f;
  for (uint64_t t = start; t < end; ++t) acc = __fadd_rn(acc, as_f32(row[t]));
  bsum[c * blocks_n + b] = acc;
}

// The same for integer samples whose block totals stay at most 2^24 (every
// partial sum exact, so any order): a warp per (block, channel), 16-byte loads
// with the samples outside the block masked.  Measured on a GB300: 512 8-bit
// channels of 1,047,799 samples, blocks of 1000: 0.62 ms with a thread per
// block, 0.165 with 64-bit indices, a division per warp and masks sample by
// sample, 0.108 now.
constexpr int BS_W = 8;  // warps (blocks) per CTA
// The low min(max(x, 0), 4) bytes of a word.
__device__ __forceinline__ uint32_t low_bytes(int x) {
  return x >= 4 ? 0xffffffffu : x <= 0 ? 0u : 0xffffffffu >> (32 - 8 * x);
}
template <class T>
__global__ void __launch_bounds__(32 * BS_W)
    k_block_sums_int(const T *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t bs,
                     uint64_t blocks_n, float *__restrict__ bsum) {
  const uint64_t b = (uint64_t)blockIdx.x * BS_W + (threadIdx.x >> 5), c = blockIdx.y;
  if (b >= blocks_n) return;
  const int lane = (int)(threadIdx.x & 31);
  constexpr int PER = 16 / (int)sizeof(T);
  const uint64_t start = b * bs, base = start & ~(uint64_t)(PER - 1);
  const T *p = s + c * ld + base;
  // samples [head, stop) from base: a block is at most 2^24 samples
  const int head = (int)(start - base), stop = head + (int)min(bs, ns - start);
  unsigned acc = 0;
  for (int i = lane * PER; i < stop; i += 32 * PER) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p + i));
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
    if (i < head || i + PER > stop) {
      const int lo = (head - i) * (int)sizeof(T), hi = (stop - i) * (int)sizeof(T);
#pragma unroll
      for (int u = 0; u < 4; ++u) w[u] &= low_bytes(hi - 4 * u) & ~low_bytes(lo - 4 * u);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if constexpr (sizeof(T) == 1) acc = __dp4a(w[u], 0x01010101u, acc);
      else acc += (w[u] & 0xffffu) + (w[u] >> 16);
    }
  }
  acc = __reduce_add_sync(0xffffffffu, acc);
  if (lane == 0) bsum[c * blocks_n + b] = (float)acc;
}

// Counters of NW warps that select together.
struct RankShared {
  uint32_t lo, hi;
  unsigned below[32];
};
template <int NW>
__device__ __forceinline__ void rank_sync() {
  if constexpr (NW > 1) __syncthreads();
  else __syncwarp();
}

// The element of rank r among n keys, key 32 NW i + tid in k[i] of the group's
// thread tid (padded with 0xffffffff, above all others): the largest value with at
// most r keys below it, bit by bit below the bits that all keys share, one warp
// reduction (and, for a group of warps, one barrier) per bit.
template <int N, int NW>
__device__ uint32_t group_rank(const uint32_t (&k)[N], int n, int r, int tid, RankShared &sh) {
  uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (32 * NW * i + tid < n) {
      lo = min(lo, k[i]);
      hi = max(hi, k[i]);
    }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if constexpr (NW > 1) {
    if (tid < 32) sh.below[tid] = 0;
    if (tid == 0) {
      sh.lo = 0xffffffffu;
      sh.hi = 0;
    }
    __syncthreads();
    if ((tid & 31) == 0) {
      atomicMin(&sh.lo, lo);
      atomicMax(&sh.hi, hi);
    }
    __syncthreads();
    lo = sh.lo;
    hi = sh.hi;
  }
  uint32_t p = lo;
  if (lo != hi) {
    const int top = 31 - __clz((int)(lo ^ hi));  // highest bit in which keys differ
    p = top == 31 ? 0u : lo >> (top + 1) << (top + 1);
    for (int bit = top; bit >= 0; --bit) {
      const uint32_t cand = p | (1u << bit);
      unsigned b0 = 0, b1 = 0;
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        b0 += k[i] < cand ? 1u : 0u;
        if (i + 1 < N) b1 += k[i + 1] < cand ? 1u : 0u;
      }
      unsigned below = __reduce_add_sync(0xffffffffu, b0 + b1);
      if constexpr (NW > 1) {
        if ((tid & 31) == 0) atomicAdd(&sh.below[bit], below);
        __syncthreads();
        below = sh.below[bit];
      }
      if ((int)below <= r) p = cand;
    }
  }
  rank_sync<NW>();
  return p;
}

// rfi::outliers (rfi/src/lib.rs:13-22) for n <= 32 NW N values by NW warps, the
// keys in registers through both selections.  A radix selection's four rounds
// over 32 histograms took about 13 us in a 1024-thread block whatever n is; the
// channel and block decisions of 512 channels and 1048 blocks took 35 and 21 us
// with two selections by one warp of a block and scratch in between, 13 and 9 now.
template <int N, int NW>
__device__ void group_outliers(const float *v, int n, float threshold, unsigned char *flags,
                               int tid, RankShared &sh) {
  uint32_t k[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int j = 32 * NW * i + tid;
    k[i] = j < n ? fkey(v[j]) : 0xffffffffu;
  }
  const float center = n > 0 ? fkey_inv(group_rank<N, NW>(k, n, n / 2, tid, sh)) : 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (32 * NW * i + tid < n) k[i] = fkey(fabsf(__fsub_rn(fkey_inv(k[i]), center)));
  const float mad = n > 0 ? fkey_inv(group_rank<N, NW>(k, n, n / 2, tid, sh)) : 0.0f;
  const float scale =
      fmaxf(fmaxf(__fmul_rn(1.4826f, mad), __fmul_rn(fabsf(center), 1e-4f)), 1e-6f);
  const float lim = __fmul_rn(threshold, scale);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int j = 32 * NW * i + tid;
    if (j < n) flags[j] = fkey_inv(k[i]) > lim ? 1 : 0;
  }
}
constexpr int CH_RANK_MAX = 1024;   // channels: a warp per vector
constexpr int BL_RANK_MAX = 2048, BL_NW = 4;  // blocks: four warps

// The same for any n, by one block; hist holds 32 x 256 words.
__device__ void block_outliers(const float *v, uint64_t n, float threshold,
                               float *dev_scratch, unsigned char *flags,
                               unsigned *hist, uint32_t *bc) {
  float center = 0.0f;
  if (n > 0) {
    auto key = [&](uint64_t i) { return fkey(v[i]); };
    center = fkey_inv(block_select(key, n, n / 2, 24, hist, bc));
  }
  for (uint64_t i = threadIdx.x; i < n; i += blockDim.x)
    dev_scratch[i] = fabsf(__fsub_rn(v[i], center));
  __syncthreads();
  float mad = 0.0f;
  if (n > 0) {
    auto key = [&](uint64_t i) { return fkey(dev_scratch[i]); };
    mad = fkey_inv(block_select(key, n, n / 2, 24, hist, bc));
  }
  float scale = fmaxf(fmaxf(__fmul_rn(1.4826f, mad), __fmul_rn(fabsf(center), 1e-4f)), 1e-6f);
  float lim = __fmul_rn(threshold, scale);
  for (uint64_t i = threadIdx.x; i < n; i += blockDim.x)
    flags[i] = fabsf(__fsub_rn(v[i], center)) > lim ? 1 : 0;
  __syncthreads();
}

// Channel decision (rfi/src/lib.rs:44-48); writes chbad[] and active count.
constexpr int DEC_NT = 512;
__global__ void __launch_bounds__(DEC_NT) k_channel_decide(const float *means, const float *vars, uint64_t nch,
                                 float threshold, float *scratch, unsigned char *f1,
                                 unsigned char *f2, unsigned char *chbad,
                                 unsigned long long *active) {
  __shared__ unsigned hist[32 * 256];
  __shared__ uint32_t bc[3];
  if (nch <= CH_RANK_MAX) {
    __shared__ RankShared sh;  // (not used by one warp)
    const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    if (warp < 2) {
      const float *v = warp ? vars : means;
      unsigned char *f = warp ? f2 : f1;
      if (nch <= 256) group_outliers<8, 1>(v, (int)nch, threshold, f, lane, sh);
      else if (nch <= 512) group_outliers<16, 1>(v, (int)nch, threshold, f, lane, sh);
      else group_outliers<CH_RANK_MAX / 32, 1>(v, (int)nch, threshold, f, lane, sh);
    }
    __syncthreads();
  } else {
    block_outliers(means, nch, threshold, scratch, f1, hist, bc);
    block_outliers(vars, nch, threshold, scratch, f2, hist, bc);
  }
  __shared__ unsigned good;
  if (threadIdx.x == 0) good = 0;
  __syncthreads();
  for (uint64_t c = threadIdx.x; c < nch; c += blockDim.x) {
    const bool bad = f1[c] || f2[c] || vars[c] < 1e-12f;
    chbad[c] = bad ? 1 : 0;
    if (!bad) atomicAdd(&good, 1u);
  }
  __syncthreads();
  if (threadIdx.x == 0) *active = good;
}

// Block means over good channels in channel order (rfi/src/lib.rs:55-69): a CTA
// takes 32 blocks; its other warps load tiles of 64 channels (double buffered,
// masked channels as zeros, which change no sum) while warp 0 adds in order,
// so the chain is one FADD per channel (one thread per block that loads as it
// adds took 130 us at 512 channels, with warp 0 loading too and a test per
// channel 38, 17 now).
constexpr int BM_L = 8, BM_C = 64;  // loading warps, channels of a tile
constexpr int BM_NT = 32 * (1 + BM_L);
__global__ void __launch_bounds__(BM_NT)
    k_block_means(const float *bsum, const unsigned char *chbad, uint64_t nch, uint64_t ns,
                  uint64_t bs, uint64_t blocks_n, const unsigned long long *active,
                  float *bmeans) {
  __shared__ float tile[2][BM_C][32];
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  const uint64_t b = (uint64_t)blockIdx.x * 32 + lane;
  auto load = [&](uint64_t c0, int k) {  // warps 1 and up
    constexpr int R = BM_C / BM_L;
    float v[R];
    bool use[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint64_t c = c0 + (warp - 1) * R + i;
      use[i] = c < nch && !chbad[c];
      v[i] = c < nch && b < blocks_n ? bsum[c * blocks_n + b] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) tile[k][(warp - 1) * R + i][lane] = use[i] ? v[i] : 0.0f;
  };
  if (warp) load(0, 0);
  __syncthreads();
  float sum = 0.0f;
  int k = 0;
  for (uint64_t c0 = 0; c0 < nch; c0 += BM_C, k ^= 1) {
    if (warp) {
      if (c0 + BM_C < nch) load(c0 + BM_C, k ^ 1);
    } else {
#pragma unroll
      for (int r = 0; r < BM_C; ++r) sum = __fadd_rn(sum, tile[k][r][lane]);
    }
    __syncthreads();
  }
  if (warp != 0 || b >= blocks_n) return;
  uint64_t start = b * bs, end = min(start + bs, ns);
  unsigned long long a = *active;
  if (a < 1) a = 1;
  bmeans[b] = __fdiv_rn(sum, (float)((end - start) * a));
}

__global__ void __launch_bounds__(DEC_NT)
    k_block_decide(const float *bmeans, uint64_t blocks_n, float threshold, float *scratch,
                   unsigned char *blkbad) {
  __shared__ unsigned hist[32 * 256];
  __shared__ uint32_t bc[3];
  block_outliers(bmeans, blocks_n, threshold, scratch, blkbad, hist, bc);
}
// The same for at most BL_RANK_MAX blocks.
__global__ void __launch_bounds__(32 * BL_NW)
    k_block_decide_few(const float *bmeans, int blocks_n, float threshold,
                       unsigned char *blkbad) {
  __shared__ RankShared sh;
  const int tid = (int)threadIdx.x;
  if (blocks_n <= 64 * BL_NW) group_outliers<2, BL_NW>(bmeans, blocks_n, threshold, blkbad, tid, sh);
  else if (blocks_n <= 256 * BL_NW)
    group_outliers<8, BL_NW>(bmeans, blocks_n, threshold, blkbad, tid, sh);
  else
    group_outliers<BL_RANK_MAX / (32 * BL_NW), BL_NW>(bmeans, blocks_n, threshold, blkbad, tid, sh);
}

// Replace masked samples with the channel median (rfi/src/lib.rs:76-89): CTA
// (group of FILL_B blocks, channel) writes the masked blocks of its group, a warp
// per block in 16-byte stores, and leaves at once where there are none.
// Testing every sample's block took 0.64 ms on 512 channels of 1,047,799
// samples (GB300), this 0.022; 64 channels of 262,144 samples 27 us with sample
// stores, 4 now.
constexpr int FILL_B = 64, FILL_NT = 256;
template <class T>
__global__ void __launch_bounds__(FILL_NT)
    k_fill(T *__restrict__ s, uint64_t ns, uint64_t ld, uint64_t bs, uint64_t blocks_n,
           const unsigned char *__restrict__ chbad, const unsigned char *__restrict__ blkbad,
           const float *__restrict__ med) {
  const uint64_t c = blockIdx.y, b0 = (uint64_t)blockIdx.x * FILL_B;
  const uint64_t b1 = min(b0 + FILL_B, blocks_n);
  const bool whole = chbad[c] != 0;
  const uint64_t mine = b0 + threadIdx.x;
  if (!__syncthreads_or(whole || (mine < b1 && blkbad[mine]))) return;
  constexpr uint64_t PER = 16 / sizeof(T);
  const T typical = (T)med[c];
  T same[PER];
#pragma unroll
  for (int i = 0; i < (int)PER; ++i) same[i] = typical;
  uint4 v;
  memcpy(&v, same, 16);
  T *row = s + c * ld;  // 16-byte aligned, as is every PER-th sample
  const uint64_t lane = threadIdx.x & 31;
  for (uint64_t b = b0 + (threadIdx.x >> 5); b < b1; b += FILL_NT / 32) {
    if (!whole && !blkbad[b]) continue;
    const uint64_t t0 = b * bs, t1 = min(t0 + bs, ns);
    const uint64_t a0 = min((t0 + PER - 1) / PER * PER, t1), a1 = max(t1 / PER * PER, a0);
    if (t0 + lane < a0) row[t0 + lane] = typical;  // (fewer than PER <= 16 samples)
    for (uint64_t t = a0 + PER * lane; t < a1; t += 32 * PER)
      *reinterpret_cast<uint4 *>(row + t) = v;
    if (a1 + lane < t1) row[a1 + lane] = typical;
  }
}

}  // namespace

int DeviceObs::alloc(cudaStream_t st) {
  ld = ((ns + 64 + 63) / 64) * 64;
  size_t bytes = (size_t)ld * nch * sample_bytes(kind) + 256;
  PSR_TRY(samples.ensure(bytes));
  // on the stream that fills the samples next: a plain cudaMemset runs on the
  // legacy default stream, which does not order against non-blocking streams
  PSR_CUDA(cudaMemsetAsync(samples.p, 0, bytes, st));
  return PSR_OK;
}

int launch_unpack(const DeviceObs &o, unsigned long long *d_err, cudaStream_t st) {
  if (o.kind == SAMPLE_U8) {
    const dim3 grid((unsigned)((o.ns + UP_T - 1) / UP_T), (unsigned)((o.nch + UP_C - 1) / UP_C));
    const uint32_t *p = o.payload.as<uint32_t>();
    uint8_t *x = o.samples.as<uint8_t>();
    switch (o.h.nbits) {
      case 1: k_unpack8<1><<<grid, UP_NT, 0, st>>>(p, x, o.ns, o.nch, o.ld); break;
      case 2: k_unpack8<2><<<grid, UP_NT, 0, st>>>(p, x, o.ns, o.nch, o.ld); break;
      case 4: k_unpack8<4><<<grid, UP_NT, 0, st>>>(p, x, o.ns, o.nch, o.ld); break;
      default: k_unpack8<8><<<grid, UP_NT, 0, st>>>(p, x, o.ns, o.nch, o.ld);
    }
  } else {
    const dim3 grid((unsigned)((o.ns + UNPACK_TT - 1) / UNPACK_TT),
                    (unsigned)((o.nch + UNPACK_TC - 1) / UNPACK_TC));
    if (o.kind == SAMPLE_U16)
      k_unpack<uint16_t><<<grid, 256, 0, st>>>(o.payload.as<uint16_t>(), o.samples.as<uint16_t>(),
                                               o.ns, o.nch, o.ld, d_err);
    else
      k_unpack<float><<<grid, 256, 0, st>>>(o.payload.as<float>(), o.samples.as<float>(), o.ns,
                                            o.nch, o.ld, d_err);
  }
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

int launch_median_f32(const float *d_vals, uint64_t n, float *d_out, unsigned int *,
                      cudaStream_t st) {
  k_median_f32<<<1, 1024, 0, st>>>(d_vals, n, d_out);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

// Channel means and variances (rfi/src/lib.rs:35-43) into w.means and w.vars.
template <class T>
static int enqueue_mean_var(const T *s, uint64_t nch, uint64_t ns, uint64_t ld, RfiWork &w,
                            cudaStream_t st) {
  const uint64_t nck = (ns + ES_L - 1) / ES_L;
  PSR_TRY(w.es_sum.ensure(nch * nck * 4));
  PSR_TRY(w.es_sq.ensure(nch * nck * 4));
  PSR_TRY(w.es_guess.ensure(nch * nck));
  PSR_TRY(w.es_maps.ensure(nch * nck * sizeof(uint2)));
  PSR_TRY(w.es_chan.ensure(nch * sizeof(EsChan)));
  PSR_TRY(w.es_neg.ensure(nch * 4));
  uint32_t *sum = w.es_sum.as<uint32_t>();
  float *sq = w.es_sq.as<float>(), *means = w.means.as<float>(), *vars = w.vars.as<float>();
  uint8_t *guess = w.es_guess.as<uint8_t>();
  EsChan *chan = w.es_chan.as<EsChan>();
  uint2 *maps = w.es_maps.as<uint2>();
  if (sizeof(T) == 4) PSR_CUDA(cudaMemsetAsync(w.es_neg.p, 0, nch * 4, st));
  constexpr uint64_t per = (EK_NT / 32) * EK_CPW;
  const dim3 grid((unsigned)((nck + per - 1) / per), (unsigned)nch);
  k_es_sums<T><<<grid, EK_NT, 0, st>>>(s, ns, ld, nck, sum, sq, w.es_neg.as<unsigned>());
  k_es_guess<T><<<(unsigned)nch, EG_NT, 0, st>>>(sum, sq, w.es_neg.as<unsigned>(), nck, ns, guess,
                                                 chan, means);
  k_es_maps<T, false><<<grid, EK_NT, 0, st>>>(s, ns, ld, nck, guess, chan, means, maps);
  k_es_scan<T, false><<<(unsigned)nch, EG_NT, 0, st>>>(s, ns, ld, nck, sum, sq, guess, chan, maps,
                                                       means, vars);
  k_es_maps<T, true><<<grid, EK_NT, 0, st>>>(s, ns, ld, nck, guess, chan, means, maps);
  k_es_scan<T, true><<<(unsigned)nch, EG_NT, 0, st>>>(s, ns, ld, nck, sum, sq, guess, chan, maps,
                                                      means, vars);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

template <class T>
static int rfi_enqueue_t(DeviceObs &o, uint64_t bs, float thr, RfiWork &w, cudaStream_t st) {
  const uint64_t nch = o.nch, ns = o.ns;
  const uint64_t blocks_n = (ns + bs - 1) / bs;
  w.blocks_n = blocks_n;
  PSR_TRY(w.means.ensure(nch * 4));
  PSR_TRY(w.vars.ensure(nch * 4));
  PSR_TRY(w.med.ensure(nch * 4));
  PSR_TRY(w.bsum.ensure(nch * blocks_n * 4));
  PSR_TRY(w.bmeans.ensure(blocks_n * 4));
  PSR_TRY(w.bad.ensure(nch + blocks_n));  // of the channels, then of the blocks
  unsigned char *chbad = w.bad.as<unsigned char>(), *blkbad = chbad + nch;
  PSR_TRY(w.scratch.ensure(std::max(nch, blocks_n) * 4));
  PSR_TRY(w.flags.ensure(2 * nch));
  PSR_TRY(w.active.ensure(8));
  T *s = o.samples.as<T>();
  PSR_TRY(enqueue_mean_var<T>(s, nch, ns, o.ld, w, st));
  if constexpr (sizeof(T) < 4) {
    if (bs <= (1u << 24) / (sizeof(T) == 1 ? 255u : 65535u))
      k_block_sums_int<T><<<dim3((unsigned)((blocks_n + BS_W - 1) / BS_W), (unsigned)nch),
                            32 * BS_W, 0, st>>>(s, ns, o.ld, bs, blocks_n, w.bsum.as<float>());
  }
  if (sizeof(T) == 4 || bs > (1u << 24) / (sizeof(T) == 1 ? 255u : 65535u))
    k_block_sums<T><<<(unsigned)((nch * blocks_n + 127) / 128), 128, 0, st>>>(
        s, ns, o.ld, nch, bs, blocks_n, w.bsum.as<float>());
  if constexpr (sizeof(T) == 1) {
    // long shares (a table is cleared and added up per CTA), but enough CTAs for
    // every SM
    const uint64_t share = std::min(MH_MAX, std::max(MH_MIN, ns * nch / 1200));
    const uint64_t per = (share + 15) / 16 * 16;
    PSR_TRY(w.mhist.ensure(nch * 256 * 4));
    PSR_CUDA(cudaMemsetAsync(w.mhist.p, 0, nch * 256 * 4, st));
    k_chan_hist_u8<<<dim3((unsigned)((ns + per - 1) / per), (unsigned)nch), MH_NT, 0, st>>>(
        s, ns, o.ld, per, w.mhist.as<unsigned>());
    k_hist_median<<<(unsigned)((nch + 3) / 4), 128, 0, st>>>(w.mhist.as<unsigned>(), nch, ns,
                                                                 w.med.as<float>());
  } else {
    const size_t hb = nch * sizeof(unsigned) << MD_BITS;
    PSR_TRY(w.mhist.ensure(hb + nch * sizeof(MedianState)));
    PSR_CUDA(cudaMemsetAsync(w.mhist.p, 0, hb + nch * sizeof(MedianState), st));
    MedianState *state = reinterpret_cast<MedianState *>(w.mhist.as<char>() + hb);
    const dim3 grid((unsigned)((ns + MD_PER - 1) / MD_PER), (unsigned)nch);
    for (int top = 8 * (int)sizeof(T); top > 0;) {
      const int bits = std::min(MD_BITS, top);
      top -= bits;
      k_median_digit<T><<<grid, MD_NT, 0, st>>>(s, ns, o.ld, top, bits, w.mhist.as<unsigned>(),
                                                state, w.med.as<float>());
    }
  }
  unsigned char *fl = w.flags.as<unsigned char>();
  k_channel_decide<<<1, DEC_NT, 0, st>>>(w.means.as<float>(), w.vars.as<float>(), nch, thr,
                                       w.scratch.as<float>(), fl, fl + nch,
                                       chbad, w.active.as<unsigned long long>());
  k_block_means<<<(unsigned)((blocks_n + 31) / 32), BM_NT, 0, st>>>(
      w.bsum.as<float>(), chbad, nch, ns, bs, blocks_n,
      w.active.as<unsigned long long>(),
      w.bmeans.as<float>());
  if (blocks_n <= (uint64_t)BL_RANK_MAX)
    k_block_decide_few<<<1, 32 * BL_NW, 0, st>>>(w.bmeans.as<float>(), (int)blocks_n, thr,
                                                 blkbad);
  else
    k_block_decide<<<1, DEC_NT, 0, st>>>(w.bmeans.as<float>(), blocks_n, thr,
                                         w.scratch.as<float>(), blkbad);
  k_fill<T><<<dim3((unsigned)((blocks_n + FILL_B - 1) / FILL_B), (unsigned)nch), FILL_NT, 0, st>>>(
      s, ns, o.ld, bs, blocks_n, chbad, blkbad,
      w.med.as<float>());
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

int rfi_channel_stats(const DeviceObs &o, float *means, float *variances, cudaStream_t st) {
  RfiWork w;
  PSR_TRY(w.means.ensure(o.nch * 4));
  PSR_TRY(w.vars.ensure(o.nch * 4));
  switch (o.kind) {
    case SAMPLE_U8: PSR_TRY(enqueue_mean_var(o.samples.as<uint8_t>(), o.nch, o.ns, o.ld, w, st)); break;
    case SAMPLE_U16: PSR_TRY(enqueue_mean_var(o.samples.as<uint16_t>(), o.nch, o.ns, o.ld, w, st)); break;
    default: PSR_TRY(enqueue_mean_var(o.samples.as<float>(), o.nch, o.ns, o.ld, w, st));
  }
  PSR_CUDA(cudaMemcpyAsync(means, w.means.p, o.nch * 4, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaMemcpyAsync(variances, w.vars.p, o.nch * 4, cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  return PSR_OK;
}

int rfi_enqueue(DeviceObs &o, uint64_t bs, float thr, RfiWork &w, cudaStream_t st) {
  if (bs == 0 || !(thr > 0.0f) || !std::isfinite(thr)) {
    set_error("rfi::mask: block_samples > 0 and a finite positive threshold are required");
    return PSR_EINVAL;
  }
  switch (o.kind) {
    case SAMPLE_U8: return rfi_enqueue_t<uint8_t>(o, bs, thr, w, st);
    case SAMPLE_U16: return rfi_enqueue_t<uint16_t>(o, bs, thr, w, st);
    default: return rfi_enqueue_t<float>(o, bs, thr, w, st);
  }
}

int rfi_collect(const DeviceObs &o, uint64_t bs, RfiWork &w, cudaStream_t st, RfiResult &res) {
  std::vector<unsigned char> ch(o.nch + w.blocks_n);
  PSR_CUDA(cudaMemcpyAsync(ch.data(), w.bad.p, ch.size(), cudaMemcpyDeviceToHost, st));
  PSR_CUDA(cudaStreamSynchronize(st));
  const unsigned char *bl = ch.data() + o.nch;
  res.channels.clear();
  res.blocks.clear();
  for (uint64_t c = 0; c < o.nch; ++c)
    if (ch[c]) res.channels.push_back(c);
  for (uint64_t b = 0; b < w.blocks_n; ++b)
    if (bl[b]) res.blocks.push_back(b);
  // rfi/src/lib.rs:75-94
  uint64_t count = res.channels.size() * o.ns;
  uint64_t good = o.nch - res.channels.size();
  for (uint64_t b : res.blocks) {
    uint64_t start = b * bs, end = std::min(start + bs, o.ns);
    count += (end - start) * good;
  }
  res.masked_fraction = (double)count / (double)(o.nch * o.ns);
  return PSR_OK;
}

}  // namespace psr
