// K3 incoherent dedispersion (dedisperse::apply, dedisperse/src/lib.rs:61-90,
// run for many trials as in the CLI loop cli/src/main.rs:462-469).
//
// out[trial][t] = sum_c data[c][t + delay[trial][c]],  t in [0, n).
//
// Integer samples (u8): every partial sum is an integer below 2^16, so the
// reference's channel-ordered f32 sum is exact and any summation order gives
// the bit-identical value.  The fast kernel stages a tile of every channel
// row into shared memory with TMA bulk copies (cp.async.bulk + mbarrier,
// double buffered), and each thread accumulates four sample words (16
// samples, words tl + 256 k of the tile) for a block of trials in packed
// 2 x u16 lanes (samples of <= 4 bits first in 4 x u8 lanes, widened once per
// group of channels).  Consecutive trials whose delay for a channel falls in
// the same aligned word reuse the loaded words (CTA-uniform test) and only
// shift them again.
//
// Everything else (f32 samples, or integer sums that could exceed 2^16) uses
// a kernel that adds channels in reference order in f32.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <type_traits>
#include <vector>

#include "psr_internal.h"

namespace psr {
namespace {

constexpr int DD_NT = 256;              // threads per CTA
constexpr int DD_TPT = 16;              // samples per thread
constexpr int DD_TT = DD_NT * DD_TPT;   // samples per tile (4096)
constexpr int DD_DB = 8;                // trials per CTA (16-bit lanes only)
constexpr int DD_DB8 = 8;               // trials per CTA with 8-bit lanes (128 registers)
constexpr int DD_MAXCC = 32;            // rows per stage (one issuing lane each)
constexpr long long DD_SPIN_LIMIT = 1ll << 26;  // try_wait polls before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false (and the error word set) if the phase never completes.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity,
                                                  unsigned *err, long long limit) {
  for (long long i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicOr(err, 1u);
  return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

struct StageInfo {
  long long base[DD_MAXCC];    // absolute sample index of the staged row start
  int off[DD_MAXCC][DD_DB];    // tile start + delay - staged row start, per trial
};

// Issue the TMA copies of rows [c0, c0+cc) for trials [d0, d0+DB) of tile t0.
// Run by warp 0: lane i stages row c0+i.  The delay of trial d0 + d and
// channel c is delays[min(d0 + d, ntrials - 1) * dstride + c] (global memory,
// or the CTA's block preloaded in shared memory with d0 = 0, ntrials = DB).
template <int DB>
__device__ void issue_stage(const uint8_t *__restrict__ s, uint64_t ld, uint64_t ns,
                            uint64_t nch, uint64_t dstride, const uint32_t *__restrict__ delays,
                            uint64_t ntrials, uint64_t d0, uint64_t t0, uint64_t c0, int cc,
                            uint8_t *buf, int rowcap, StageInfo *info, uint64_t *bar,
                            int arm_only) {
  const int lane = threadIdx.x & 31;
  unsigned bytes = 0;
  if (lane < cc && c0 + lane < nch) {
    const uint64_t c = c0 + lane;
    uint32_t dmin = 0xffffffffu, dmax = 0;
    for (int d = 0; d < DB; ++d) {
      uint64_t tr = d0 + d < ntrials ? d0 + d : ntrials - 1;
      uint32_t v = delays[tr * dstride + c];
      dmin = min(dmin, v);
      dmax = max(dmax, v);
    }
    long long a = (long long)((t0 + dmin) & ~(uint64_t)15);
    long long rowend = (long long)((ns + 15) & ~(uint64_t)15);
    long long b = (long long)((t0 + dmax + DD_TT + 15) & ~(uint64_t)15);
    if (b > rowend) b = rowend;
    if (b > a + rowcap) b = a + rowcap;
    info->base[lane] = a;
    for (int d = 0; d < DB; ++d) {
      uint64_t tr = d0 + d < ntrials ? d0 + d : ntrials - 1;
      info->off[lane][d] = (int)((long long)t0 - a) + (int)delays[tr * dstride + c];
    }
    if (b > a) {
      bytes = (unsigned)(b - a);
      mbar_expect_tx(bar, bytes);
    }
    __syncwarp(__activemask());
    // arm_only (a test of the bounded wait): the barrier expects the bytes
    // but no copy is issued, so its phase never completes and nothing is in
    // flight when the CTA gives up.
    if (bytes && !arm_only) bulk_g2s(buf + (size_t)lane * rowcap, s + c * ld + a, bytes, bar);
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// BYTE_LANES: samples are at most (255 / group), so `group` channels can be
// summed in the four 8-bit lanes of a 32-bit word with a plain IADD (no lane
// overflows, so no carry crosses a byte); the byte lanes are widened into the
// 16-bit lanes once per group.  Without BYTE_LANES every channel is widened.
template <bool BYTE_LANES, int DB, bool PRELOAD>
__global__ void __launch_bounds__(DD_NT, 2)
    k_dedisp_u8(const uint8_t *__restrict__ s, uint64_t ld, uint64_t ns, uint64_t nch,
                uint64_t dstride, const uint32_t *__restrict__ delays, uint64_t ntrials,
                uint64_t n, float *__restrict__ out, uint64_t ldo, double *__restrict__ part,
                uint64_t ntiles, int cc, int rowcap, int group, int accumulate, unsigned *err,
                long long spin_limit, int arm_only) {
  extern __shared__ __align__(128) uint8_t smem[];
  const size_t bstride = (size_t)cc * rowcap;  // buffer b at smem + b * bstride
  __shared__ uint64_t bars[2];
  __shared__ StageInfo info[2];
  __shared__ unsigned long long wsum[DD_NT / 32][DB];

  const uint64_t t0 = (uint64_t)blockIdx.x * DD_TT;
  const uint64_t d0 = (uint64_t)blockIdx.y * DB;
  const int tl = threadIdx.x;
  const int nchunks = (int)((nch + cc - 1) / cc);

  // preload: the CTA's [DB][nch] block of delays is copied once into shared
  // memory after the row buffers, so that issuing a stage (between chunks,
  // while the other warps wait at the barrier) reads no global memory.
  auto issue = [&](int k, int b) {
    if constexpr (PRELOAD)
      issue_stage<DB>(s, ld, ns, nch, nch,
                      reinterpret_cast<const uint32_t *>(smem + 2 * bstride), DB, 0, t0,
                      (uint64_t)k * cc, cc, smem + b * bstride, rowcap, &info[b], &bars[b],
                      arm_only);
    else
      issue_stage<DB>(s, ld, ns, nch, dstride, delays, ntrials, d0, t0, (uint64_t)k * cc, cc,
                      smem + b * bstride, rowcap, &info[b], &bars[b], arm_only);
  };
  if constexpr (PRELOAD) {
    uint32_t *dly = reinterpret_cast<uint32_t *>(smem + 2 * bstride);
    const unsigned nc = (unsigned)nch;  // DB * nch <= 4096 (16 KB) when preloaded
    for (unsigned i = tl; i < DB * nc; i += DD_NT) {
      const unsigned d = i / nc, c = i - d * nc;
      const uint64_t tr = d0 + d < ntrials ? d0 + d : ntrials - 1;
      dly[i] = delays[tr * dstride + c];
    }
  }
  if (tl == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tl < 32) {
    issue(0, 0);
    if (nchunks > 1) issue(1, 1);
  }

  uint32_t acc[DB][8];
#pragma unroll
  for (int d = 0; d < DB; ++d)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[d][i] = 0;
  uint32_t acc8[BYTE_LANES ? DB : 1][4];
#pragma unroll
  for (int d = 0; d < (BYTE_LANES ? DB : 1); ++d)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc8[d][i] = 0;
  int gcount = 0;
  auto widen = [&]() {
    if constexpr (BYTE_LANES) {
#pragma unroll
      for (int d = 0; d < DB; ++d)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[d][2 * i] += __byte_perm(acc8[d][i], 0, 0x4140);
          acc[d][2 * i + 1] += __byte_perm(acc8[d][i], 0, 0x4342);
          acc8[d][i] = 0;
        }
    }
  };

  // Chunk k is staged in buffer k & 1, in that barrier's phase (k >> 1).
  // A wait that gives up ends the whole CTA: the decision is made uniform
  // by __syncthreads_or before any thread reads the buffer or reaches a
  // later barrier, so no thread is left waiting on one that left.
  int failed = -1;
  for (int k = 0; k < nchunks; ++k) {
    const int b = k & 1;
    const bool ok = mbar_wait_bounded(&bars[b], (unsigned)((k >> 1) & 1), err, spin_limit);
    if (__syncthreads_or(!ok)) {
      failed = k;
      break;
    }
    const uint64_t c0 = (uint64_t)k * cc;
    const int rows = (int)min((uint64_t)cc, (uint64_t)(nch - c0));
    const uint8_t *buf = smem + b * bstride;
    for (int r = 0; r < rows; ++r) {
      // Thread tl owns words tl + 256 k (k < 4) of the tile.  A trial's row
      // offset `off` (bytes, CTA-uniform) selects words w = off >> 2 onward,
      // shifted right by (off & 3) bytes.  Delays grow by 0 or 1 sample from
      // one trial to the next, so consecutive trials mostly share w: the
      // loaded words are kept and only re-shifted.  Lane d < DB reads trial
      // d's offset; the ballots of "offset changed" and "word changed"
      // against trial d - 1 are warp-uniform bit masks and the offsets are
      // broadcast by shuffles, so every branch below is uniform by
      // construction.
      const uint32_t *row = reinterpret_cast<const uint32_t *>(buf + (size_t)r * rowcap) + tl;
      const int lane = tl & 31;
      const int myoff = info[b].off[r][lane < DB ? lane : DB - 1];
      const int prevoff = __shfl_up_sync(0xffffffffu, myoff, 1);
      const unsigned chg =
          __ballot_sync(0xffffffffu, lane < DB && (lane == 0 || myoff != prevoff));
      const unsigned wchg =
          __ballot_sync(0xffffffffu, lane < DB && (lane == 0 || (myoff >> 2) != (prevoff >> 2)));
      uint32_t a0 = 0, a1 = 0, a2 = 0, a3 = 0, b0 = 0, b1 = 0, b2 = 0, b3 = 0;
      uint32_t x0 = 0, x1 = 0, x2 = 0, x3 = 0;
      // 16-bit lanes: the shifted words split into sample pairs once per
      // offset change, not once per trial
      uint32_t y[BYTE_LANES ? 1 : 8];
#pragma unroll
      for (int i = 0; i < (BYTE_LANES ? 1 : 8); ++i) y[i] = 0;
#pragma unroll
      for (int d = 0; d < DB; ++d) {
        if (chg & (1u << d)) {
          const int off = __shfl_sync(0xffffffffu, myoff, d);
          if (wchg & (1u << d)) {
            const uint32_t *p = row + (off >> 2);
            a0 = p[0];
            b0 = p[1];
            a1 = p[256];
            b1 = p[257];
            a2 = p[512];
            b2 = p[513];
            a3 = p[768];
            b3 = p[769];
          }
          const unsigned sh = (unsigned)(off & 3) * 8u;
          x0 = __funnelshift_r(a0, b0, sh);
          x1 = __funnelshift_r(a1, b1, sh);
          x2 = __funnelshift_r(a2, b2, sh);
          x3 = __funnelshift_r(a3, b3, sh);
          if constexpr (!BYTE_LANES) {
            y[0] = __byte_perm(x0, 0, 0x4140);
            y[1] = __byte_perm(x0, 0, 0x4342);
            y[2] = __byte_perm(x1, 0, 0x4140);
            y[3] = __byte_perm(x1, 0, 0x4342);
            y[4] = __byte_perm(x2, 0, 0x4140);
            y[5] = __byte_perm(x2, 0, 0x4342);
            y[6] = __byte_perm(x3, 0, 0x4140);
            y[7] = __byte_perm(x3, 0, 0x4342);
          }
        }
        if constexpr (BYTE_LANES) {
          acc8[d][0] += x0;
          acc8[d][1] += x1;
          acc8[d][2] += x2;
          acc8[d][3] += x3;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[d][i] += y[i];
        }
      }
      if (BYTE_LANES && ++gcount == group) {
        widen();
        gcount = 0;
      }
    }
    __syncthreads();  // every thread is done reading buffer b
    if (tl < 32 && k + 2 < nchunks) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(k + 2, b);
    }
  }
  widen();
  if (failed >= 0) {
    // Before leaving, wait (bounded) for the copies still outstanding: chunk
    // `failed` in its buffer and, if it was issued, chunk failed + 1 in the
    // other, each in the phase it was issued in.
    if (tl == 0) {
      mbar_wait_bounded(&bars[failed & 1], (unsigned)((failed >> 1) & 1), err, spin_limit);
      if (failed + 1 < nchunks)
        mbar_wait_bounded(&bars[(failed + 1) & 1], (unsigned)(((failed + 1) >> 1) & 1), err,
                          spin_limit);
    }
    return;
  }

  // Word k of this thread holds samples t0 + 4 (tl + 256 k) + {0, 1, 2, 3}:
  // acc[d][2k] their first two (16-bit lanes), acc[d][2k + 1] the last two.
#pragma unroll
  for (int d = 0; d < DB; ++d) {
    const uint64_t tr = d0 + d;
    unsigned long long local = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint64_t tb = t0 + 4 * ((uint64_t)tl + 256 * k);
      const uint32_t p = acc[d][2 * k], q = acc[d][2 * k + 1];
      const float v[4] = {(float)(p & 0xffffu), (float)(p >> 16), (float)(q & 0xffffu),
                          (float)(q >> 16)};
      if (tb + 4 <= n) {
        local += (p & 0xffffu) + (p >> 16) + (q & 0xffffu) + (q >> 16);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (tb + i < n) local += (unsigned)v[i];
      }
      if (tr < ntrials) {
        // Channel groups after the first add their (integer) partial sums to
        // the earlier groups' in f32: exact while every sum stays below 2^24.
        float *dst = out + tr * ldo + tb;
        if (tb + 4 <= n) {
          float4 w = make_float4(v[0], v[1], v[2], v[3]);
          if (accumulate) {
            const float4 o = *reinterpret_cast<const float4 *>(dst);
            w.x += o.x;
            w.y += o.y;
            w.z += o.z;
            w.w += o.w;
          }
          *reinterpret_cast<float4 *>(dst) = w;
        } else {
          for (int i = 0; i < 4; ++i)
            if (tb + i < n) dst[i] = accumulate ? dst[i] + v[i] : v[i];
        }
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
    if ((tl & 31) == 0) wsum[tl >> 5][d] = local;
  }
  __syncthreads();
  if (tl < DB && d0 + tl < ntrials) {
    unsigned long long t = 0;
    for (int w = 0; w < DD_NT / 32; ++w) t += wsum[w][tl];
    double *pp = &part[(d0 + tl) * ntiles + blockIdx.x];
    *pp = accumulate ? *pp + (double)t : (double)t;
  }
}

// ---------------------------------------------------------------------------
// Two-level dedispersion of u8 samples.  Channels are taken in subbands of G
// adjacent channels.  A trial's delays inside a subband, relative to the
// subband's smallest delay, form a pattern; over a chunk of trials the same
// patterns come back (DM plans of about one sample per trial have 4 to 30 of
// them per subband and 256 trials), so
//   k_sub_part  sums each pattern's G channels once per chunk, over the whole
//               series (16-bit sums, rows of a scratch buffer), and
//   k_sub_sum   adds, for every trial, one row per subband at the trial's
//               shift.
// Every sum is an integer (below 2^16 in its lane, below 2^24 in all), so
// the result is bit-identical to the reference's channel-ordered f32 sum.
constexpr int SUB_GMAX = 8;
constexpr int SP_NT = 256;              // k_sub_part: threads
constexpr int SP_TT = SP_NT * 16;       // and samples per tile (4 words of 4 per thread)
constexpr int SS_TB = 16;               // k_sub_sum: trials per CTA, one warp each
constexpr int SS_K = 16;                // 32-bit words (sample pairs) per lane
constexpr int SS_TT = 32 * SS_K * 2;    // samples per tile (1024)
constexpr int SS_NT = 32 * (SS_TB + 1); // and a warp that issues the copies
constexpr int SS_MAXROWS = 64;          // rows of a stage (two per issuing lane)
constexpr int SS_MAXBUF = 4;            // stage buffers
constexpr int SS_MAXSTAGES = 1024;      // stages of a trial block

// A subband of one chunk: its patterns are rows [row0, row0 + npat) of the
// chunk's scratch; row sample i is series time i + seg0 of a trial whose
// smallest subband delay is dmin.
struct SubBand {
  int32_t dmin, spread, row0, npat, relmax, pad;
};
// A stage of k_sub_sum, packed: the next nrows (bits 0-7) rows of the trial
// block's row list, the next nsubs (bits 8-15) subbands, and a flush after it
// (bit 16).
constexpr uint32_t sub_stage(int nrows, int nsubs, int flush) {
  return (uint32_t)nrows | (uint32_t)nsubs << 8 | (uint32_t)flush << 16;
}
// A staged row: a scratch row and the first sample copied.
struct SubRow {
  uint32_t row, start;  // start: a multiple of 8 samples (16 bytes)
};

// Bound: shared memory and issue, about 22 instructions per 16 samples of a
// pattern's channel (8 word loads, 4 funnel shifts, then 4 byte-lane adds or,
// above 255, per word one full add and one add of the odd bytes: with
// T = sum of the words mod 2^32 and O = sum of the odd bytes in 16-bit lanes,
// the even bytes' sum is T - (O << 8)).
// Measured on a GB300 with k_sub_sum below, against the channel-by-channel
// kernel (and, at 4096 channels, the subband kernel that summed patterns per
// 8 trials in shared memory): 96 4-bit channels, 2000 trials of 263,500
// samples 0.60 + 1.58 ms against 3.22; 512 8-bit channels, 700 trials of
// 523,500 samples 0.63 + 4.17 against 12.95; 4096 8-bit channels, 300 trials
// of 1,045,000 samples 6.9 + 27.9 against 124 (118).
template <int G, bool BYTE>
__global__ void __launch_bounds__(SP_NT)
    k_sub_part(const uint8_t *__restrict__ s, uint64_t ld, uint64_t ns, uint64_t nch,
               const SubBand *__restrict__ subs, const uint16_t *__restrict__ rel,
               uint64_t seg0, uint64_t seglen, uint16_t *__restrict__ scratch, uint64_t ldp,
               int rowcap, unsigned *err, long long spin_limit) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bar;
  const SubBand sb = subs[blockIdx.y];
  const uint64_t i0 = (uint64_t)blockIdx.x * SP_TT;
  if (i0 >= seglen + (uint64_t)sb.spread + 2) return;  // (uniform) past every trial's last sample
  const int tl = threadIdx.x;
  const uint64_t c0 = (uint64_t)blockIdx.y * G;
  const int gr = (int)min((uint64_t)G, nch - c0);
  const uint64_t abs0 = seg0 + i0 + (uint64_t)sb.dmin;
  const uint64_t a = abs0 & ~15ull;
  if (tl == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tl < 32) {
    const uint64_t rowend = (ns + 15) & ~15ull;
    // + 4: the last word's funnel shift reads one word on
    uint64_t b = (abs0 + SP_TT + (uint64_t)sb.relmax + 4 + 15) & ~15ull;
    b = min(min(b, rowend), a + (uint64_t)rowcap);
    if (tl < gr && b > a) mbar_expect_tx(&bar, (unsigned)(b - a));
    __syncwarp();
    if (tl < gr && b > a)
      bulk_g2s(smem + (size_t)tl * rowcap, s + (c0 + tl) * ld + a, (unsigned)(b - a), &bar);
    __syncwarp();
    if (tl == 0) mbar_arrive(&bar);
  }
  const bool ok = mbar_wait_bounded(&bar, 0, err, spin_limit);
  if (__syncthreads_or(!ok)) {
    if (tl == 0) mbar_wait_bounded(&bar, 0, err, spin_limit);
    return;
  }
  const uint16_t *rp = rel + (size_t)sb.row0 * G;
  uint16_t *dst = scratch + (uint64_t)sb.row0 * ldp + i0 + 4 * tl;
  const int base = (int)(abs0 - a);
  uint16_t rn[G];
  auto load_rel = [&](const uint16_t *q) {  // rows of the table are 2 G bytes, aligned
    if constexpr (G == 8) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(q));
      memcpy(rn, &v, 16);
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2 *>(q));
      memcpy(rn, &v, 8);
    }
  };
  load_rel(rp);
  for (int p = 0; p < sb.npat; ++p) {
    int off[G];
#pragma unroll
    for (int r = 0; r < G; ++r) off[r] = base + (int)rn[r];
    if (p + 1 < sb.npat) load_rel(rp + (size_t)(p + 1) * G);
    uint32_t T[4] = {0, 0, 0, 0}, O[4] = {0, 0, 0, 0};
#pragma unroll
    for (int r = 0; r < G; ++r) {
      if (r < gr) {
        const uint32_t *q =
            reinterpret_cast<const uint32_t *>(smem + (size_t)r * rowcap) + tl + (off[r] >> 2);
        const unsigned sh = (unsigned)(off[r] & 3) * 8u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t x = __funnelshift_r(q[256 * k], q[256 * k + 1], sh);
          T[k] += x;
          if constexpr (!BYTE) O[k] += __byte_perm(x, 0, 0x4341);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint2 w;
      if constexpr (BYTE) {
        w.x = __byte_perm(T[k], 0, 0x4140);
        w.y = __byte_perm(T[k], 0, 0x4342);
      } else {
        const uint32_t E = T[k] - (O[k] << 8);  // samples 0 and 2; O: samples 1 and 3
        w.x = __byte_perm(E, O[k], 0x5410);
        w.y = __byte_perm(E, O[k], 0x7632);
      }
      *reinterpret_cast<uint2 *>(dst + 1024 * k) = w;
    }
    dst += ldp;
  }
}

// One warp per trial: lane l owns the sample pairs (words) l + 32 k of the
// tile.  A row at an even shift adds its words as they lie (E).  At an odd
// shift 2 m + 1 the words from m on are added as they lie too, into O: a
// pair's odd-shift sum is the high half of O's word and the low half of the
// next, so the odd shifts cost one realignment per trial (or flush) instead
// of one per row.  FLUSH: the sums pass 16 bits; stages marked by the plan
// add the lanes to 32-bit sums.
// The rows arrive in a ring of nbuf stage buffers: the last warp issues the
// bulk copies of a stage once all trial warps have left its buffer, with the
// row list read two stages ahead.  Waits are bounded; one that gives up sets
// the error word and `dead`, on which every warp leaves, the issuing warp
// last, after the copies it has in flight.
// Bound: shared-memory loads, 2 bytes per (trial, subband, sample) in two
// instructions per word: two thirds of the wavefronts and of the issue slots at
// 512 channels, with 16 trial warps per SM to hide the rest (the copies out of L2 take
// a tenth of the crossbar; a row serves the trials of its block that share the
// pattern, 4 to 5 of 16 at G = 4).  With the copies issued by a trial warp between
// two CTA barriers and two buffers the 4096-channel case took 50.5 ms, with the ring
// 27.9; with 24 trials per CTA 33.8 (72 registers leave fewer loads in flight),
// with two trials per warp on one window of words 56.5, with several tiles per CTA
// 32.3 (CTAs of one tile no longer run side by side, and rows miss L2).
template <bool FLUSH>
__global__ void __launch_bounds__(SS_NT, FLUSH ? 1 : 2)
    k_sub_sum(const uint16_t *__restrict__ scratch, uint64_t ldp,
              const uint32_t *__restrict__ stage0, const uint32_t *__restrict__ row0,
              const uint32_t *__restrict__ stages, const SubRow *__restrict__ rows,
              const uint32_t *__restrict__ info, uint64_t nsub, uint64_t ntrials, uint64_t seg0,
              uint64_t segend, float *__restrict__ out, uint64_t ldo, double *__restrict__ part,
              uint64_t ntiles, int rowcap, int bufbytes, int nbuf, unsigned *err,
              long long spin_limit) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[SS_MAXBUF], empty[SS_MAXBUF];
  __shared__ uint32_t desc[SS_MAXSTAGES];
  __shared__ volatile int dead;
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  const uint64_t tb = blockIdx.x;
  const uint64_t tile0 = (uint64_t)blockIdx.y * SS_TT;  // from seg0
  const uint32_t st0 = stage0[tb];
  const int nst = (int)(stage0[tb + 1] - st0);
  for (int i = threadIdx.x; i < nst; i += SS_NT) desc[i] = stages[st0 + i];
  if (threadIdx.x == 0) {
    dead = 0;
    for (int i = 0; i < nbuf; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], SS_TB);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto wait = [&](uint64_t *bar, unsigned parity) -> bool {
    for (long long i = 0; i < spin_limit; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if ((i & 63) == 63 && dead) return false;
    }
    atomicOr(err, 1u);
    dead = 1;
    return false;
  };

  if (warp == SS_TB) {
    // lane i copies rows i and i + 32 of every stage
    const SubRow *rl = rows + row0[tb];
    const uint16_t *src = scratch + tile0;
    constexpr int H = SS_MAXROWS / 32;
    SubRow r[2][H];  // the rows of stages k and k + 1
    int ahead = 0;   // first row of the stage to read next
    auto fetch = [&](int k, SubRow *x) {
      const int nr = k < nst ? (int)(desc[k] & 255u) : 0;
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (lane + 32 * h < nr) x[h] = rl[ahead + lane + 32 * h];
      ahead += nr;
    };
    fetch(0, r[0]);
    fetch(1, r[1]);
    int b = 0;
    unsigned turn = 0;
    int issued = 0;
    auto one = [&](int k, SubRow *x) -> bool {
      if (turn && !__all_sync(0xffffffffu, wait(&empty[b], (turn - 1) & 1))) return false;
      const int nr = (int)(desc[k] & 255u);
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (lane + 32 * h < nr) {
          mbar_expect_tx(&full[b], (unsigned)rowcap);
          bulk_g2s(smem + (size_t)b * bufbytes + (size_t)(lane + 32 * h) * rowcap,
                   src + (uint64_t)x[h].row * ldp + x[h].start, (unsigned)rowcap, &full[b]);
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[b]);
      ++issued;
      fetch(k + 2, x);
      if (++b == nbuf) {
        b = 0;
        ++turn;
      }
      return true;
    };
    for (int k = 0; k < nst; k += 2) {
      if (!one(k, r[0])) break;
      if (k + 1 < nst && !one(k + 1, r[1])) break;
    }
    // leave after the copies of the last nbuf stages issued
    for (int k = max(0, issued - nbuf); k < issued; ++k)
      for (long long i = 0; i < spin_limit; ++i)
        if (mbar_try_wait(&full[k % nbuf], (unsigned)(k / nbuf) & 1)) break;
    return;
  }

  const uint32_t *inf = info + (tb * SS_TB + warp) * nsub;
  const uint64_t tr = tb * SS_TB + warp;
  const bool live = tr < ntrials;
  uint32_t E[SS_K], O[SS_K + 1];
  uint32_t acc[FLUSH ? 2 * SS_K : 1];
#pragma unroll
  for (int i = 0; i < SS_K; ++i) E[i] = O[i] = 0;
  O[SS_K] = 0;
#pragma unroll
  for (int i = 0; i < (FLUSH ? 2 * SS_K : 1); ++i) acc[i] = 0;
  // Sums of word k's two samples: E's word plus O's realigned by one sample
  // (the next word is the next lane's; lane 31's is lane 0's of k + 1).
  auto merged = [&](int k, uint32_t &v0, uint32_t &v1) {
    const uint32_t up = __shfl_down_sync(0xffffffffu, O[k], 1);
    const uint32_t wrap = __shfl_sync(0xffffffffu, O[k + 1], 0);
    const uint32_t nx = lane == 31 ? wrap : up;
    v0 = (E[k] & 0xffffu) + (O[k] >> 16);
    v1 = (E[k] >> 16) + (nx & 0xffffu);
  };
  // This trial's words in the stage's buffer: byte offset, bit 0 an odd
  // shift; lane j holds the stage's subband j.
  uint32_t nextinf = lane < (int)((desc[0] >> 8) & 255u) ? __ldg(inf + lane) : 0u;
  int b = 0;
  unsigned turn = 0;
  for (int k = 0; k < nst; ++k) {
    const uint32_t d = desc[k];
    const int nsubs = (int)((d >> 8) & 255u);
    const uint32_t myinf = nextinf;
    inf += nsubs;
    if (k + 1 < nst && lane < (int)((desc[k + 1] >> 8) & 255u)) nextinf = __ldg(inf + lane);
    if (!__all_sync(0xffffffffu, wait(&full[b], turn & 1))) return;
    if (live) {
      const uint8_t *buf = smem + (size_t)b * bufbytes;
      for (int j = 0; j < nsubs; ++j) {
        const uint32_t w = __shfl_sync(0xffffffffu, myinf, j);
        const uint32_t *q = reinterpret_cast<const uint32_t *>(buf + (w & ~1u));
        if (w & 1u) {
#pragma unroll
          for (int i = 0; i < SS_K; ++i) O[i] += q[lane + 32 * i];
          O[SS_K] += q[32 * SS_K];
        } else {
#pragma unroll
          for (int i = 0; i < SS_K; ++i) E[i] += q[lane + 32 * i];
        }
      }
      if constexpr (FLUSH) {
        if (d >> 16) {
#pragma unroll
          for (int i = 0; i < SS_K; ++i) {
            uint32_t v0, v1;
            merged(i, v0, v1);
            acc[2 * i] += v0;
            acc[2 * i + 1] += v1;
          }
#pragma unroll
          for (int i = 0; i < SS_K; ++i) E[i] = O[i] = 0;
          O[SS_K] = 0;
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[b]);
    if (++b == nbuf) {
      b = 0;
      ++turn;
    }
  }
  if (!live) return;
  const uint64_t t0 = seg0 + tile0;
  float *dst = out + tr * ldo + t0;
  uint32_t local = 0;  // at most 2 SS_K sums below 2^24
#pragma unroll
  for (int k = 0; k < SS_K; ++k) {
    uint32_t v0, v1;
    merged(k, v0, v1);
    if constexpr (FLUSH) {
      v0 += acc[2 * k];
      v1 += acc[2 * k + 1];
    }
    const int e = 2 * (lane + 32 * k);
    if (t0 + e + 2 <= segend) {
      *reinterpret_cast<float2 *>(dst + e) = make_float2((float)v0, (float)v1);
      local += v0 + v1;
    } else if (t0 + e < segend) {
      dst[e] = (float)v0;
      local += v0;
    }
  }
  unsigned long long sum = local;
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if (lane == 0) part[tr * ntiles + t0 / SS_TT] = (double)sum;
}

// Reference-order f32 accumulation (one output per thread per trial).
constexpr int DG_TPT = 4;
constexpr int DG_NT = 256;
constexpr int DG_TT = DG_NT * DG_TPT;
constexpr int DG_DB = 4;

template <class T>
__global__ void __launch_bounds__(DG_NT)
    k_dedisp_generic(const T *__restrict__ s, uint64_t ld, uint64_t nch,
                     const uint32_t *__restrict__ delays, uint64_t ntrials, uint64_t n,
                     float *__restrict__ out, uint64_t ldo, double *__restrict__ part,
                     uint64_t ntiles) {
  __shared__ double wsum[DG_NT / 32][DG_DB];
  __shared__ double wabs[DG_NT / 32][DG_DB];
  __shared__ int wq[DG_NT / 32][DG_DB];
  const uint64_t t0 = (uint64_t)blockIdx.x * DG_TT;
  const uint64_t d0 = (uint64_t)blockIdx.y * DG_DB;
  float acc[DG_DB][DG_TPT];
#pragma unroll
  for (int d = 0; d < DG_DB; ++d)
#pragma unroll
    for (int i = 0; i < DG_TPT; ++i) acc[d][i] = 0.0f;
  for (uint64_t c = 0; c < nch; ++c) {
    const T *row = s + c * ld;
#pragma unroll
    for (int d = 0; d < DG_DB; ++d) {
      uint64_t tr = d0 + d < ntrials ? d0 + d : ntrials - 1;
      const uint64_t dl = __ldg(&delays[tr * nch + c]);
#pragma unroll
      for (int i = 0; i < DG_TPT; ++i) {
        uint64_t t = t0 + (uint64_t)i * DG_NT + threadIdx.x;
        float v = t < n ? (float)row[t + dl] : 0.0f;
        acc[d][i] = __fadd_rn(acc[d][i], v);
      }
    }
  }
  // Non-integer samples: besides the sum, each tile records the sum of |x|
  // and the finest binary quantum among its outputs, from which
  // k_reduce_parts decides whether every partial sum is exact in f64.
  constexpr bool kFloat = std::is_same<T, float>::value;
#pragma unroll
  for (int d = 0; d < DG_DB; ++d) {
    double local = 0.0, labs = 0.0;
    int lq = kNoQuantum;
    const uint64_t tr = d0 + d;
#pragma unroll
    for (int i = 0; i < DG_TPT; ++i) {
      uint64_t t = t0 + (uint64_t)i * DG_NT + threadIdx.x;
      if (t < n) {
        if (tr < ntrials) out[tr * ldo + t] = acc[d][i];
        local += (double)acc[d][i];
        if (kFloat) {
          labs += fabs((double)acc[d][i]);
          lq = min(lq, quantum_exponent(acc[d][i]));
        }
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      local += __shfl_down_sync(0xffffffffu, local, o);
      if (kFloat) {
        labs += __shfl_down_sync(0xffffffffu, labs, o);
        lq = min(lq, __shfl_down_sync(0xffffffffu, lq, o));
      }
    }
    if ((threadIdx.x & 31) == 0) {
      wsum[threadIdx.x >> 5][d] = local;
      if (kFloat) {
        wabs[threadIdx.x >> 5][d] = labs;
        wq[threadIdx.x >> 5][d] = lq;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < DG_DB && d0 + threadIdx.x < ntrials) {
    double t = 0.0, a = 0.0;
    int q = kNoQuantum;
    for (int w = 0; w < DG_NT / 32; ++w) {
      t += wsum[w][threadIdx.x];
      if (kFloat) {
        a += wabs[w][threadIdx.x];
        q = min(q, wq[w][threadIdx.x]);
      }
    }
    const uint64_t at = (d0 + threadIdx.x) * ntiles + blockIdx.x;
    part[at] = t;
    if (kFloat) {
      part[ntrials * ntiles + at] = a;
      part[2 * ntrials * ntiles + at] = (double)q;
    }
  }
}

// ---------------------------------------------------------------------------
// The same for blocks of trials, from staged rows: f32 and 16-bit samples.
// One warp per trial, DR_TB trials and a tile of DR_TT samples per CTA; the rows
// arrive in a ring of stage buffers of `stage` channels that a warp of its own
// fills (as k_sub_sum's), and every trial adds its shifted words in channel
// order.  A pair of 16-bit samples at an odd shift is put together from two
// words.
// Bound: shared-memory loads, one word per f32 addition (or pair), of which
// an SM does 32 per clock.  The tile's sum takes no f64 work per sample (1/64
// rate, half of the time of short series before): the values are integers of their
// finest quantum, summed in 64 bits; the sum is only used where it stays
// below 2^53 of it, and sum |x|, which decides that, is rounded up.
// Measured on a GB300 against k_dedisp_generic, 512 channels, 256 trials of
// 260,000 samples: f32 6.64 ms, 4.09 now (90% of the loads' rate); 16-bit
// 7.45, 4.60.
constexpr int DR_TB = 16;
constexpr int DR_NT = 32 * (DR_TB + 1);
constexpr int DR_K = 32;            // samples per lane
constexpr int DR_TT = 32 * DR_K;    // and per tile
static_assert(DR_TT == DG_TT, "part[] counts tiles of DG_TT samples");
constexpr int DR_MAXBUF = 4;
constexpr int DR_SMEM = 106 * 1024;  // two CTAs per SM

// Sum of a lane's values x[i] (those with valid(i)) over its warp: S in units of
// 2^q, exact while sum |x| < 2^(53 + q); A >= sum |x|; q their finest quantum.
template <class Valid>
__device__ __forceinline__ void quantum_sum(const float (&x)[DR_K], Valid valid, double &S,
                                            double &A, int &q) {
  q = kNoQuantum;
  float a = 0.0f;
#pragma unroll
  for (int i = 0; i < DR_K; ++i)
    if (valid(i)) {
      q = min(q, quantum_exponent(x[i]));
      a = __fadd_ru(a, fabsf(x[i]));
    }
  q = __reduce_min_sync(0xffffffffu, q);
#pragma unroll
  for (int o = 16; o; o >>= 1) a = __fadd_ru(a, __shfl_xor_sync(0xffffffffu, a, o));
  long long t = 0;
#pragma unroll
  for (int i = 0; i < DR_K; ++i)
    if (valid(i)) {
      const uint32_t b = __float_as_uint(x[i]);
      const int e = (int)(b >> 23 & 255u);
      const long long m = (long long)(e ? (b & 0x7fffffu) | 0x800000u : b & 0x7fffffu);
      // (a value past 2^54 quanta makes the sum unused: any shift will do)
      const int sh = (e ? e : 1) - 150 - q;
      const long long v = sh >= 0 ? m << min(sh, 30) : m >> min(-sh, 31);
      t += (int)b < 0 ? -v : v;
    }
#pragma unroll
  for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  S = q >= kNoQuantum ? 0.0
                      : (double)t * __longlong_as_double((long long)(1023 + q) << 52);
  A = (double)a;
}

template <class T>
__global__ void __launch_bounds__(DR_NT, 2)
    k_dedisp_rows(const T *__restrict__ s, uint64_t ld, uint64_t nch,
                  const uint32_t *__restrict__ delays, uint64_t ntrials, uint64_t n,
                  float *__restrict__ out, uint64_t ldo, double *__restrict__ part,
                  uint64_t ntiles, int stage, int rowcap, int nbuf, unsigned *err,
                  long long spin_limit) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[DR_MAXBUF], empty[DR_MAXBUF];
  __shared__ uint32_t start[DR_MAXBUF][32];  // first sample staged, from the tile's
  __shared__ volatile int dead;
  constexpr bool kFloat = std::is_same<T, float>::value;
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  const uint64_t t0 = (uint64_t)blockIdx.x * DR_TT;
  const uint64_t d0 = (uint64_t)blockIdx.y * DR_TB;
  const int nst = (int)((nch + stage - 1) / stage);
  const size_t bufbytes = (size_t)stage * rowcap;
  if (threadIdx.x == 0) {
    dead = 0;
    for (int i = 0; i < nbuf; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], DR_TB);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto wait = [&](uint64_t *bar, unsigned parity) -> bool {
    for (long long i = 0; i < spin_limit; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if ((i & 63) == 63 && dead) return false;
    }
    atomicOr(err, 1u);
    dead = 1;
    return false;
  };

  if (warp == DR_TB) {
    // lane i copies channel i of every stage, from the smallest delay of the
    // block's trials on
    auto first = [&](int k) -> uint32_t {
      const uint64_t c = (uint64_t)k * stage + lane;
      uint32_t m = 0xffffffffu;
      if (k < nst && lane < stage && c < nch)
        for (int d = 0; d < DR_TB; ++d)
          m = min(m, __ldg(&delays[min(d0 + d, ntrials - 1) * nch + c]));
      return m & ~(uint32_t)(16 / sizeof(T) - 1);
    };
    uint32_t ahead = first(0);
    int b = 0, issued = 0;
    unsigned turn = 0;
    for (int k = 0; k < nst; ++k) {
      const uint32_t at = ahead;
      ahead = first(k + 1);
      if (turn && !__all_sync(0xffffffffu, wait(&empty[b], (turn - 1) & 1))) break;
      const uint64_t c = (uint64_t)k * stage + lane;
      if (lane < stage && c < nch) {
        start[b][lane] = at;
        // (the row ends at ld; what lies past it belongs to samples past n)
        const uint64_t left = (ld - (t0 + at)) * sizeof(T);
        const unsigned bytes = (unsigned)min((uint64_t)rowcap, left);
        mbar_expect_tx(&full[b], bytes);
        bulk_g2s(smem + (size_t)b * bufbytes + (size_t)lane * rowcap, s + c * ld + t0 + at, bytes,
                 &full[b]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[b]);
      ++issued;
      if (++b == nbuf) {
        b = 0;
        ++turn;
      }
    }
    // leave after the copies of the last nbuf stages issued
    for (int k = max(0, issued - nbuf); k < issued; ++k)
      for (long long i = 0; i < spin_limit; ++i)
        if (mbar_try_wait(&full[k % nbuf], (unsigned)(k / nbuf) & 1)) break;
    return;
  }

  const uint64_t tr = d0 + warp;
  const bool live = tr < ntrials;
  const uint32_t *dl = delays + min(tr, ntrials - 1) * nch;
  float acc[DR_K];
#pragma unroll
  for (int i = 0; i < DR_K; ++i) acc[i] = 0.0f;
  uint32_t next = lane < stage && (uint64_t)lane < nch ? __ldg(dl + lane) : 0u;
  int b = 0;
  unsigned turn = 0;
  for (int k = 0; k < nst; ++k) {
    const uint64_t c0 = (uint64_t)k * stage;
    const int nc = (int)min((uint64_t)stage, nch - c0);
    uint32_t mine = next;
    if (lane < stage && c0 + stage + lane < nch) next = __ldg(dl + c0 + stage + lane);
    if (!__all_sync(0xffffffffu, wait(&full[b], turn & 1))) return;
    if (live) {
      if (lane < nc) mine -= start[b][lane];
      const uint8_t *buf = smem + (size_t)b * bufbytes;
      for (int j = 0; j < nc; ++j, buf += rowcap) {
        const uint32_t o = __shfl_sync(0xffffffffu, mine, j);
        if constexpr (kFloat) {
          const float *q = reinterpret_cast<const float *>(buf) + o + lane;
#pragma unroll
          for (int i = 0; i < DR_K; ++i) acc[i] = __fadd_rn(acc[i], q[32 * i]);
        } else {
          const uint32_t *q = reinterpret_cast<const uint32_t *>(buf) + (o >> 1) + lane;
          auto add = [&](int i, uint32_t x) {  // 2^23 + v by a byte permute, less 2^23
            acc[2 * i] = __fadd_rn(
                acc[2 * i],
                __fsub_rn(__uint_as_float(__byte_perm(x, 0x4B000000u, 0x7510u)), 8388608.0f));
            acc[2 * i + 1] = __fadd_rn(
                acc[2 * i + 1],
                __fsub_rn(__uint_as_float(__byte_perm(x, 0x4B000000u, 0x7532u)), 8388608.0f));
          };
          if (o & 1u) {
#pragma unroll
            for (int i = 0; i < DR_K / 2; ++i)
              add(i, __byte_perm(q[32 * i], q[32 * i + 1], 0x5432u));
          } else {
#pragma unroll
            for (int i = 0; i < DR_K / 2; ++i) add(i, q[32 * i]);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[b]);
    if (++b == nbuf) {
      b = 0;
      ++turn;
    }
  }
  if (!live) return;
  const int m = (int)min((uint64_t)DR_TT, n - t0);  // samples of the tile
  auto sample = [&](int i) { return kFloat ? lane + 32 * i : 2 * (lane + 32 * (i >> 1)) + (i & 1); };
  float *dst = out + tr * ldo + t0;
#pragma unroll
  for (int i = 0; i < DR_K; ++i)
    if (sample(i) < m) dst[sample(i)] = acc[i];
  const uint64_t at = tr * ntiles + blockIdx.x;
  if constexpr (kFloat) {
    double S, A;
    int q;
    quantum_sum(acc, [&](int i) { return sample(i) < m; }, S, A, q);
    if (lane == 0) {
      part[at] = S;
      part[ntrials * ntiles + at] = A;
      part[2 * ntrials * ntiles + at] = (double)q;
    }
  } else {
    unsigned long long t = 0;  // sums below 2^32 each
#pragma unroll
    for (int i = 0; i < DR_K; ++i)
      if (sample(i) < m) t += __float2uint_rz(acc[i]);
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) part[at] = (double)t;
  }
}

// The plan of k_dedisp_rows for sample type T: false where its rows do not fit
// (delays that spread far over 16 trials) or the trials are too few to share
// them (below 8 its warps idle).
template <class T>
bool rows_plan(uint64_t nch, uint64_t ntrials, uint64_t max_spread, int &stage, int &rowcap,
               int &nbuf) {
  if (ntrials < 8 || (sizeof(T) == 2 && nch > 65536) || max_spread > DR_SMEM) return false;
  // 16 trials lie in three windows of 8 that overlap
  const uint64_t cap =
      ((DR_TT + 3 * max_spread + 16 / sizeof(T) + 2) * sizeof(T) + 15) & ~(uint64_t)15;
  if (cap * 2 > DR_SMEM) return false;
  const uint64_t rows = DR_SMEM / cap;
  stage = (int)std::min<uint64_t>({32, nch, std::max<uint64_t>(1, rows / DR_MAXBUF)});
  nbuf = (int)std::min<uint64_t>(DR_MAXBUF, rows / stage);
  rowcap = (int)cap;
  return true;
}

// ---------------------------------------------------------------------------
// The series sum per trial and the f32 mean the FFT subtracts
// (search/src/lib.rs:36-40).  The reference's mean is a sequential f64 sum
// starting from -0.0.  Integer samples make every partial sum an exact integer
// below 2^53, so any order gives it.  Otherwise the series is taken in segments
// of which the sum, sum |x| and the finest quantum 2^q among the values are
// known.  A running sum s that is a multiple of 2^qs stays exact through a
// segment, in any order inside it, while |s| + sum |x| < 2^(53 + min(q, qs))
// (with a margin for the rounding of sum |x|): every partial sum is a multiple
// of that quantum below 2^53 of it.  Such segments are added at once, 32 at a
// time where that holds for all of them together; the others sample by sample
// in order.

// 2^(53 + q) (q within f32 exponents' reach; larger: no limit).
__device__ __forceinline__ double exact_limit(int q) {
  return q > 200 ? INFINITY : __longlong_as_double((long long)(53 + q + 1023) << 52);
}
// Quantum exponent of a finite f64 (zero constrains nothing).
__device__ __forceinline__ int quantum_exponent64(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & ~(1ull << 63);
  if (b == 0) return kNoQuantum;
  const int e = (int)(b >> 52);
  unsigned long long m = b & 0xFFFFFFFFFFFFFull;
  if (e) m |= 1ull << 52;
  return (e ? e : 1) - 1075 + (__ffsll((long long)m) - 1);
}
// Whether s passes exactly through values of magnitude sum `mag` and quantum q.
__device__ __forceinline__ bool passes(double s, double mag, int q) {
  const int qs = quantum_exponent64(s);
  return fabs(s) + mag * (1.0 + 0x1p-20) < exact_limit(min(q, qs));
}

// The sequential sum s + x[..] over segments [g0, g1) by one warp; segment i
// covers samples [i len, (i + 1) len) of x[0, n) and seg(i, S, A, q) gives its
// sum, sum |x| and quantum.  All lanes hold s and return the sum.
template <class Seg>
__device__ double sequential_sum(const float *__restrict__ x, uint64_t n, uint64_t len,
                                 uint64_t g0, uint64_t nseg, Seg seg, int lane, double s) {
  for (uint64_t g = g0; g < nseg; g += 32) {
    double S = 0.0, A = 0.0;
    int q = kNoQuantum;
    if (g + lane < nseg) seg(g + lane, S, A, q);
    double St = S, At = A;
    int qt = q;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      St += __shfl_xor_sync(0xffffffffu, St, o);
      At += __shfl_xor_sync(0xffffffffu, At, o);
      qt = min(qt, __shfl_xor_sync(0xffffffffu, qt, o));
    }
    if (passes(s, At, qt)) {
      s += St;
      continue;
    }
    const int cnt = (int)min((uint64_t)32, nseg - g);
    for (int i = 0; i < cnt; ++i) {
      const double Si = __shfl_sync(0xffffffffu, S, i), Ai = __shfl_sync(0xffffffffu, A, i);
      const int qi = __shfl_sync(0xffffffffu, q, i);
      if (passes(s, Ai, qi)) {
        s += Si;
        continue;
      }
      const uint64_t a = (g + i) * len, b = min(a + len, n);
      for (uint64_t t0 = a; t0 < b; t0 += 32) {
        const float v = t0 + lane < b ? x[t0 + lane] : 0.0f;
        const int m = (int)min((uint64_t)32, b - t0);
        for (int u = 0; u < m; ++u) s += (double)__shfl_sync(0xffffffffu, v, u);
      }
    }
  }
  return s;
}

// Per-tile partial sums into sums and means: one warp per trial.  Integer
// samples: the tiles' sums added 32 lanes wide.  f32 samples (check): the
// sequential sum, tiles of 1024 samples as segments (the one-thread re-addition
// that inexact series took before costs about 30 us per 1000 samples).
constexpr int RP_NT = 128;
__global__ void __launch_bounds__(RP_NT)
    k_reduce_parts(const double *part, uint64_t ntiles, uint64_t ntrials, uint64_t n,
                   double *sums, float *means, const float *series, uint64_t ldo, int check) {
  const uint64_t tr = (uint64_t)blockIdx.x * (RP_NT / 32) + (threadIdx.x >> 5);
  const int lane = (int)(threadIdx.x & 31);
  if (tr >= ntrials) return;
  double s = 0.0;
  if (check) {
    const double *ps = part + tr * ntiles, *pa = ps + ntrials * ntiles,
                 *pq = pa + ntrials * ntiles;
    s = sequential_sum(series + tr * ldo, n, DG_TT, 0, ntiles,
                       [&](uint64_t i, double &S, double &A, int &q) {
                         S = ps[i];
                         A = pa[i];
                         q = (int)pq[i];
                       }, lane, -0.0);
  } else {
    for (uint64_t i = lane; i < ntiles; i += 32) s += part[tr * ntiles + i];
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  }
  if (lane != 0) return;
  sums[tr] = s;
  means[tr] = (float)(s / (double)n);
}

// launch_series_mean: segments of SM_SEG samples, one warp each, and blocks of
// SM_B segments, one CTA each; then one warp over 32 blocks at a time, which
// opens a block that does not pass into its segments.  Measured on a GB300:
// 3,000,001 samples 2.56 ms by one CTA that read the series, 0.02 + 0.01 now.
constexpr int SM_SEG = 256, SM_B = 32, SM_NT = 32 * SM_B;
struct SegSum {
  double S, A;
  int q, pad;
};
__global__ void __launch_bounds__(SM_NT)
    k_series_segs(const float *__restrict__ x, uint64_t n, uint64_t nseg,
                  SegSum *__restrict__ seg, SegSum *__restrict__ blk) {
  __shared__ SegSum sh[SM_B];
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  const uint64_t i = (uint64_t)blockIdx.x * SM_B + warp;
  float v[SM_SEG / 32];
#pragma unroll
  for (int u = 0; u < SM_SEG / 32; ++u) {
    const uint64_t t = i * SM_SEG + 32 * u + lane;
    v[u] = t < n ? x[t] : 0.0f;
  }
  double S = 0.0;
  float A = 0.0f;  // an upper bound is all it is used for
  int q = kNoQuantum;
#pragma unroll
  for (int u = 0; u < SM_SEG / 32; ++u) {
    S += (double)v[u];
    A = __fadd_ru(A, fabsf(v[u]));
    q = min(q, quantum_exponent(v[u]));
  }
  // (where S itself is inexact, A and q make passes() fail for any s)
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      S += __shfl_xor_sync(0xffffffffu, S, o);
      A = __fadd_ru(A, __shfl_xor_sync(0xffffffffu, A, o));
    }
    q = __reduce_min_sync(0xffffffffu, q);
  };
  reduce();
  if (lane == 0) {
    sh[warp] = SegSum{S, (double)A, q, 0};
    if (i < nseg) seg[i] = sh[warp];
  }
  __syncthreads();
  if (warp != 0) return;
  S = sh[lane].S;
  A = (float)sh[lane].A;  // (was a float)
  q = sh[lane].q;
  reduce();
  if (lane == 0) blk[blockIdx.x] = SegSum{S, (double)A, q, 0};
}
__global__ void __launch_bounds__(32)
    k_series_mean(const float *__restrict__ x, uint64_t n, const SegSum *__restrict__ seg,
                  uint64_t nseg, const SegSum *__restrict__ blk, uint64_t nblk, double *sum_out,
                  float *mean_out) {
  const int lane = (int)threadIdx.x;
  double s = -0.0;
  for (uint64_t g = 0; g < nblk; g += 32) {
    SegSum b{0.0, 0.0, kNoQuantum, 0};
    if (g + lane < nblk) b = blk[g + lane];
    double St = b.S, At = b.A;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      St += __shfl_xor_sync(0xffffffffu, St, o);
      At += __shfl_xor_sync(0xffffffffu, At, o);
    }
    if (passes(s, At, __reduce_min_sync(0xffffffffu, b.q))) {
      s += St;
      continue;
    }
    const int cnt = (int)min((uint64_t)32, nblk - g);
    for (int i = 0; i < cnt; ++i) {
      const double Si = __shfl_sync(0xffffffffu, b.S, i), Ai = __shfl_sync(0xffffffffu, b.A, i);
      if (passes(s, Ai, __shfl_sync(0xffffffffu, b.q, i))) {
        s += Si;
        continue;
      }
      s = sequential_sum(x, n, SM_SEG, (g + i) * SM_B, min((g + i + 1) * SM_B, nseg),
                         [&](uint64_t j, double &S, double &A, int &q) {
                           const SegSum e = seg[j];
                           S = e.S;
                           A = e.A;
                           q = e.q;
                         }, lane, s);
    }
  }
  if (lane != 0) return;
  if (sum_out) *sum_out = s;
  *mean_out = (float)(s / (double)n);
}

}  // namespace

size_t series_mean_scratch(uint64_t n) {
  const uint64_t nseg = (n + SM_SEG - 1) / SM_SEG;
  return (size_t)(nseg + (nseg + SM_B - 1) / SM_B) * sizeof(SegSum);
}

int launch_series_mean(const float *d_x, uint64_t n, double *d_sum, float *d_mean,
                       void *d_scratch, cudaStream_t st) {
  const uint64_t nseg = (n + SM_SEG - 1) / SM_SEG, nblk = (nseg + SM_B - 1) / SM_B;
  SegSum *seg = static_cast<SegSum *>(d_scratch), *blk = seg + nseg;
  k_series_segs<<<(unsigned)nblk, SM_NT, 0, st>>>(d_x, n, nseg, seg, blk);
  k_series_mean<<<1, 32, 0, st>>>(d_x, n, seg, nseg, blk, nblk, d_sum, d_mean);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

uint64_t series_ld(uint64_t n) { return ((n + 63) / 64) * 64; }

namespace {
int reduce_parts(const double *d_part, uint64_t ntiles, uint64_t ntrials, uint64_t n,
                 double *d_sums, float *d_means, const float *d_series, uint64_t ldo, int check,
                 cudaStream_t st) {
  constexpr uint64_t per = RP_NT / 32;
  k_reduce_parts<<<(unsigned)((ntrials + per - 1) / per), RP_NT, 0, st>>>(
      d_part, ntiles, ntrials, n, d_sums, d_means, d_series, ldo, check);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}
}  // namespace

namespace {
std::atomic<int> g_subbands{-1};

// Dynamic shared memory of k_sub_sum's stage buffers: two CTAs per SM without
// FLUSH, one with it.
constexpr int SS_SMEM = 106 * 1024, SS_SMEM_FLUSH = 216 * 1024;
constexpr int SP_MAXSMEM = 72 * 1024;       // k_sub_part: three CTAs per SM

// A subband's delays relative to its smallest, 16 bits each.
struct RelKey {
  uint64_t a = 0, b = 0;
  bool operator==(const RelKey &o) const { return a == o.a && b == o.b; }
};

// The patterns of every subband over one chunk of trials.
struct ChunkPatterns {
  std::vector<SubBand> subs;
  std::vector<RelKey> keys;     // rows, in subband order
  std::vector<uint16_t> pat;    // [subband][trial of the chunk]
  std::vector<uint32_t> ref;    // [subband][trial]: smallest delay
  bool ok = true;
};

void chunk_patterns(const std::vector<uint32_t> &tab, uint64_t nch, uint64_t ta, uint64_t tz,
                    int G, ChunkPatterns &cp) {
  const uint64_t nt = tz - ta, nsub = (nch + G - 1) / G;
  cp = ChunkPatterns();
  cp.subs.reserve(nsub);
  cp.pat.resize(nsub * nt);
  cp.ref.resize(nsub * nt);
  uint32_t hsize = 64;
  while (hsize < 4 * nt) hsize <<= 1;
  std::vector<uint32_t> slot(hsize, 0);  // 1 + row of the subband's pattern, by generation
  std::vector<uint32_t> gen(hsize, 0);
  // The table's rows are nch apart: a strip of 64 channels is copied first.
  constexpr uint64_t STRIP = 64;
  std::vector<uint32_t> strip(nt * STRIP);
  for (uint64_t j = 0; j < nsub && cp.ok; ++j) {
    const uint64_t ca = j * G;
    const int ge = (int)std::min<uint64_t>(G, nch - ca);
    if (ca % STRIP == 0) {
      const uint64_t w = std::min<uint64_t>(STRIP, nch - ca);
      for (uint64_t t = 0; t < nt; ++t)
        std::copy_n(&tab[(ta + t) * nch + ca], w, &strip[t * STRIP]);
    }
    SubBand sb{};
    sb.row0 = (int32_t)cp.keys.size();
    uint32_t dmin = 0xffffffffu, dmax = 0;
    RelKey last;
    for (uint64_t t = 0; t < nt && cp.ok; ++t) {
      const uint32_t *d = &strip[t * STRIP + ca % STRIP];
      uint32_t m = d[0], mx = d[0];
      for (int c = 1; c < ge; ++c) {
        m = std::min(m, d[c]);
        mx = std::max(mx, d[c]);
      }
      if (mx - m > 4095u || mx > (uint32_t)INT32_MAX) {  // SubBand holds 31 bits
        cp.ok = false;
        break;
      }
      sb.relmax = std::max(sb.relmax, (int32_t)(mx - m));
      dmin = std::min(dmin, m);
      dmax = std::max(dmax, m);
      RelKey k;
      for (int c = 0; c < ge; ++c) {
        const uint64_t r = d[c] - m;
        if (c < 4) k.a |= r << (16 * c);
        else k.b |= r << (16 * (c - 4));
      }
      cp.ref[j * nt + t] = m;
      if (t && k == last) {  // as the trial before
        cp.pat[j * nt + t] = cp.pat[j * nt + t - 1];
        continue;
      }
      last = k;
      uint64_t h = (k.a ^ (k.b * 0x9E3779B97F4A7C15ull)) * 0xD6E8FEB86659FD93ull;
      uint32_t q = (uint32_t)(h >> 40) & (hsize - 1);
      for (;;) {
        if (gen[q] != j + 1) {
          gen[q] = (uint32_t)j + 1;
          slot[q] = (uint32_t)cp.keys.size();
          cp.keys.push_back(k);
          break;
        }
        if (cp.keys[slot[q]] == k) break;
        q = (q + 1) & (hsize - 1);
      }
      cp.pat[j * nt + t] = (uint16_t)(slot[q] - (uint32_t)sb.row0);
    }
    sb.dmin = (int32_t)dmin;
    sb.spread = (int32_t)(dmax - dmin);
    sb.npat = (int32_t)(cp.keys.size() - (size_t)sb.row0);
    if (sb.npat > 65535) cp.ok = false;  // pat[] holds 16 bits
    cp.subs.push_back(sb);
  }
}

// The two-level kernels against the channel-by-channel one on a chunk of nt
// trials, per 512 samples, in SM issue slots fitted to times on a GB300 (96,
// 512 and 4096 channels, 64 to 256 trials, both widths): a channel of a trial
// costs the channel-by-channel kernel 38 (<= 4-bit samples) or 62; a pattern
// costs k_sub_part 80 + 50 G or 310 + 38 G (the write of its row included);
// k_sub_sum 280 per row it stages, or 32 per (trial, subband), whichever is more.
double direct_cost(uint64_t nch, uint64_t nt, double maxv) {
  return (maxv * 2.0 <= 255.0 ? 38.0 : 62.0) * (double)nch * (double)nt;
}
double two_level_cost(const ChunkPatterns &cp, uint64_t nt, int G, double maxv) {
  const double part = maxv * SUB_GMAX <= 255.0 ? 80.0 + 50.0 * G : 310.0 + 38.0 * G;
  const uint64_t nsub = cp.subs.size();
  std::vector<uint32_t> seen(65536, 0);
  uint32_t gen = 0;
  uint64_t staged = 0;
  for (uint64_t j = 0; j < nsub; ++j)
    for (uint64_t t = 0; t < nt; ++t) {
      if (t % SS_TB == 0) ++gen;
      uint32_t &s = seen[cp.pat[j * nt + t]];
      staged += s != gen;
      s = gen;
    }
  return part * (double)cp.keys.size() +
         std::max(280.0 * (double)staged, 32.0 * (double)nt * (double)nsub);
}
}  // namespace

int dedisp_subbands_default() {
  return g_subbands.load();
}

namespace {
// A plan's tables on the host, and the shape that the plan takes from them.
struct SubbandTables {
  SubbandPlan::Shape shape;
  std::vector<SubBand> subs;
  std::vector<uint16_t> rel;
  std::vector<uint32_t> stage0, rowlist0, stages, info;
  std::vector<SubRow> rows;
  std::vector<SubbandPlan::Chunk> chunks;
};
constexpr uint64_t SUB_GRID = 65535;  // tiles of a segment: grid.y
static_assert(32 * SS_MAXSTAGES <= SUB_GRID, "as do the subbands of any plan that fits");

// The tables at width G; false when the plan does not fit.  `known`: the
// patterns of chunk known_ci at this width, or null.
bool subband_tables(const std::vector<uint32_t> &tab, uint64_t nch, uint64_t n, double maxv,
                    const std::vector<uint64_t> &cstart, int G, uint64_t scratch,
                    SubbandTables &out, const ChunkPatterns *known = nullptr,
                    size_t known_ci = 0) {
  const bool flush = (double)nch * maxv > 65535.0;
  const size_t nchunks = cstart.size() - 1;
  const uint64_t nsub = (nch + G - 1) / G;
  out = SubbandTables();
  auto &[shape, subs, rel, stage0, rowlist0, stages, info, rows, chunks] = out;
  struct Win {  // a row a trial block uses: offsets [lo, hi] of its trials
    uint32_t row, lo, hi;
  };
  std::vector<Win> wins;
  std::vector<uint32_t> winpos;     // first window of each (trial block, subband)
  std::vector<uint8_t> slotof;      // [trial block][subband][16]
  std::vector<uint32_t> offof;
  uint64_t max_rows = 0, max_spread = 0;
  int relmax = 0;
  uint32_t maxwin = 0;
  size_t most = 0;
  for (size_t ci = 0; ci < nchunks; ++ci) {
    const uint64_t ta = cstart[ci], nt = cstart[ci + 1] - ta;
    if (nt == 0) return false;
    ChunkPatterns own;
    const bool have = known && ci == known_ci;
    if (!have) chunk_patterns(tab, nch, ta, ta + nt, G, own);
    const ChunkPatterns &cp = have ? *known : own;
    if (!cp.ok) return false;
    SubbandPlan::Chunk c;
    c.sub0 = subs.size();
    c.rel0 = rel.size();
    c.block0 = 0;
    c.nblocks = (nt + SS_TB - 1) / SS_TB;
    c.spread = 0;
    slotof.reserve(slotof.size() + c.nblocks * nsub * SS_TB);
    offof.reserve(offof.size() + c.nblocks * nsub * SS_TB);
    for (const SubBand &sb : cp.subs) {
      c.spread = std::max<uint64_t>(c.spread, (uint64_t)sb.spread);
      relmax = std::max(relmax, sb.relmax);
      subs.push_back(sb);
    }
    max_spread = std::max(max_spread, c.spread);
    max_rows = std::max<uint64_t>(max_rows, cp.keys.size());
    for (const RelKey &k : cp.keys)
      for (int r = 0; r < G; ++r)
        rel.push_back((uint16_t)((r < 4 ? k.a >> (16 * r) : k.b >> (16 * (r - 4))) & 0xffffu));
    for (uint64_t tb = 0; tb < c.nblocks; ++tb) {
      for (uint64_t j = 0; j < nsub; ++j) {
        const SubBand &sb = cp.subs[j];
        winpos.push_back((uint32_t)wins.size());
        const size_t w0 = wins.size();
        for (int d = 0; d < SS_TB; ++d) {
          // slots past the chunk's trials repeat its last one
          const uint64_t t = std::min<uint64_t>(tb * SS_TB + d, nt - 1);
          const uint32_t row = (uint32_t)sb.row0 + cp.pat[j * nt + t];
          const uint32_t off = cp.ref[j * nt + t] - (uint32_t)sb.dmin;
          size_t w = w0;
          while (w < wins.size() && wins[w].row != row) ++w;
          if (w == wins.size()) wins.push_back(Win{row, off, off});
          wins[w].lo = std::min(wins[w].lo, off);
          wins[w].hi = std::max(wins[w].hi, off);
          slotof.push_back((uint8_t)(w - w0));
          offof.push_back(off);
        }
        for (size_t w = w0; w < wins.size(); ++w)
          maxwin = std::max(maxwin, wins[w].hi - (wins[w].lo & ~7u));
        most = std::max(most, wins.size() - w0);
      }
    }
    chunks.push_back(c);
  }
  winpos.push_back((uint32_t)wins.size());
  // A staged row: the tile, its trials' offsets, and the word past the tile
  // that an odd shift reads.
  const uint64_t rowcap = (((uint64_t)SS_TT + maxwin + 2) * 2 + 15) & ~15ull;
  const uint64_t room = flush ? SS_SMEM_FLUSH : SS_SMEM;
  const int maxrows = (int)std::min<uint64_t>(
      SS_MAXROWS, std::max<uint64_t>(most, room / (SS_MAXBUF * rowcap)));
  const uint64_t bufbytes = ((uint64_t)maxrows * rowcap + 127) & ~127ull;
  const int nbuf = (int)std::min<uint64_t>(SS_MAXBUF, room / bufbytes);
  const uint64_t prowcap = ((uint64_t)SP_TT + relmax + 36 + 15) & ~15ull;
  if (nbuf < 2 || prowcap * G > SP_MAXSMEM) return false;
  // Segments of the series: the rows of one stay within `scratch`, its tiles
  // within a grid.
  const uint64_t tail = max_spread + rowcap / 2 + 16;
  uint64_t seg = std::min((n + SS_TT - 1) / SS_TT, SUB_GRID) * SS_TT;
  auto stride = [&](uint64_t sg) { return ((sg + tail + SP_TT - 1) / SP_TT) * SP_TT; };
  if (max_rows * stride(seg) * 2 > scratch) {
    const uint64_t per = scratch / (2 * max_rows);
    seg = per > tail + SP_TT ? ((per - tail - SP_TT) / SS_TT) * SS_TT : 0;
    if (seg < 16 * SS_TT) return false;  // rows too many to reuse
  }
  const uint64_t ldp = stride(seg);
  // Stages: subbands in order while their rows fit the buffer; a stage after
  // which the next could pass 16 bits is marked to flush.
  size_t wi = 0, si = 0;
  uint64_t blk = 0;
  for (size_t ci = 0; ci < nchunks; ++ci) {
    chunks[ci].block0 = blk;
    for (uint64_t tb = 0; tb < chunks[ci].nblocks; ++tb, ++blk) {
      stage0.push_back((uint32_t)stages.size());
      rowlist0.push_back((uint32_t)rows.size());
      int nrows = 0, nsubs = 0;
      double held = 0.0;  // largest sum the 16-bit lanes can hold so far
      const size_t inf0 = info.size();
      info.resize(inf0 + SS_TB * nsub);
      for (uint64_t j = 0; j < nsub; ++j, ++wi) {
        const int nw = (int)(winpos[wi + 1] - winpos[wi]);
        const double add = maxv * (double)std::min<uint64_t>(G, nch - j * G);
        const bool over = held + add > 65535.0;
        if (nsubs && (nrows + nw > maxrows || nsubs == 32 || over)) {
          stages.push_back(sub_stage(nrows, nsubs, over ? 1 : 0));
          if (over) held = 0.0;
          nrows = nsubs = 0;
        }
        held += add;
        for (int w = 0; w < nw; ++w) {
          const Win &x = wins[winpos[wi] + w];
          rows.push_back(SubRow{x.row, x.lo & ~7u});
        }
        for (int d = 0; d < SS_TB; ++d, ++si) {
          const Win &x = wins[winpos[wi] + slotof[si]];
          const uint32_t o = offof[si] - (x.lo & ~7u);
          info[inf0 + (size_t)d * nsub + j] =
              (uint32_t)(nrows + slotof[si]) * (uint32_t)rowcap + (o >> 1) * 4u + (o & 1u);
        }
        nrows += nw;
        nsubs += 1;
      }
      stages.push_back(sub_stage(nrows, nsubs, 0));
      if (stages.size() - stage0.back() > SS_MAXSTAGES) return false;
    }
  }
  stage0.push_back((uint32_t)stages.size());
  shape.G = G;
  shape.nsub = nsub;
  shape.byte_part = maxv * SUB_GMAX <= 255.0;
  shape.flush = flush;
  shape.seg = seg;
  shape.ldp = ldp;
  shape.scratch_bytes = max_rows * ldp * 2 + 256;
  shape.rowcap = (int)rowcap;
  shape.prowcap = (int)prowcap;
  shape.bufbytes = (int)bufbytes;
  shape.nbuf = nbuf;
  return true;
}

// The tables at width G (4 or 8), or at the cheapest that pays (-1); shape.G is 0
// where there is no plan.
void choose_subband_tables(const std::vector<uint32_t> &tab, uint64_t nch, uint64_t n, double maxv,
                           const std::vector<uint64_t> &cstart, int G, bool once,
                           uint64_t scratch, SubbandTables &t) {
  t = SubbandTables();
  if (G == 0 || cstart.size() < 2 || !(maxv > 0.0) || maxv > 255.0 ||
      (double)nch * maxv >= 16777216.0 || n < 2)
    return;
  auto take = [&](int g, const ChunkPatterns *known, size_t known_ci) {
    const bool fits = subband_tables(tab, nch, n, maxv, cstart, g, scratch, t, known, known_ci);
    if (!fits) t = SubbandTables();
    return fits;
  };
  if (G == 4 || G == 8) {
    take(G, nullptr, 0);
    return;
  }
  // A plan for one pass has to save more than it takes to make: 25 ns per
  // channel and trial, 150 us for its buffers and copies (299 channels, 59 trials
  // of 131,000 to 400,000 samples: 0.3 to 0.5 ms, the kernels saved 0.1).  Seconds
  // per unit of the costs below, which are fitted to a GB300: 512 samples, four
  // issue slots a clock of 152 SMs at 1.9 GHz.
  const double unit = (double)n / 512.0 / 1.155e12;
  const uint64_t total = cstart.back() - cstart.front();
  const double making = once ? 150e-6 + 25e-9 * (double)(nch * total) : 0.0;
  if (once && 0.8 * unit * direct_cost(nch, total, maxv) < making) return;
  // The widths that are cheaper than the channel-by-channel kernel on the
  // middle chunk, cheapest first.
  const size_t mid = (cstart.size() - 2) / 2;
  const uint64_t nt = cstart[mid + 1] - cstart[mid];
  std::vector<std::pair<double, int>> pick;
  ChunkPatterns cp[2];  // at widths 8, 4
  for (int g : {8, 4}) {
    ChunkPatterns &p = cp[g == 4];
    chunk_patterns(tab, nch, cstart[mid], cstart[mid + 1], g, p);
    if (!p.ok) continue;
    const double c = two_level_cost(p, nt, g, maxv);
    const double saved = direct_cost(nch, nt, maxv) - c;
    if (saved > 0.0 && unit * saved * (double)total / (double)nt > making) pick.emplace_back(c, g);
  }
  std::sort(pick.begin(), pick.end());
  for (const auto &p : pick)
    if (take(p.second, &cp[p.second == 4], mid)) return;
}

}  // namespace

int build_subband_plan(const std::vector<uint32_t> &tab, uint64_t nch, uint64_t n, double maxv,
                       const std::vector<uint64_t> &cstart, int G, SubbandPlan &plan,
                       cudaStream_t st, bool once, uint64_t scratch) {
  SubbandTables t;
  choose_subband_tables(tab, nch, n, maxv, cstart, G, once, scratch, t);
  static_cast<SubbandPlan::Shape &>(plan) = SubbandPlan::Shape();
  plan.chunks.clear();
  if (t.shape.G == 0) {
    plan.release();
    return PSR_OK;
  }
  auto up = [&](DevBuf &b, const auto &v) -> int {
    PSR_TRY(b.ensure(v.size() * sizeof(v[0])));
    PSR_CUDA(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice, st));
    return PSR_OK;
  };
  auto all = [&]() -> int {
    PSR_TRY(plan.scratch.ensure(t.shape.scratch_bytes));
    PSR_TRY(up(plan.subs, t.subs));
    PSR_TRY(up(plan.rel, t.rel));
    PSR_TRY(up(plan.stage0, t.stage0));
    PSR_TRY(up(plan.stages, t.stages));
    PSR_TRY(up(plan.rowlist0, t.rowlist0));
    PSR_TRY(up(plan.rows, t.rows));
    PSR_TRY(up(plan.info, t.info));
    PSR_CUDA(cudaStreamSynchronize(st));
    return PSR_OK;
  };
  if (all() != PSR_OK) {  // no memory for it: channel by channel
    cudaGetLastError();
    plan.release();
    return PSR_OK;
  }
  static_cast<SubbandPlan::Shape &>(plan) = t.shape;
  plan.chunks = std::move(t.chunks);
  return PSR_OK;
}

namespace {
template <int G, bool BYTE>
int run_part(const DeviceObs &o, const SubbandPlan &sb, const SubbandPlan::Chunk &c,
             uint64_t seg0, uint64_t seglen, unsigned *d_err, cudaStream_t st, long long spin) {
  const size_t smem = (size_t)G * sb.prowcap;
  PSR_CUDA(cudaFuncSetAttribute(k_sub_part<G, BYTE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                SP_MAXSMEM));
  dim3 grid((unsigned)((seglen + c.spread + 2 + SP_TT - 1) / SP_TT), (unsigned)sb.nsub);
  k_sub_part<G, BYTE><<<grid, SP_NT, smem, st>>>(
      o.samples.as<uint8_t>(), o.ld, o.ns, o.nch, sb.subs.as<SubBand>() + c.sub0,
      sb.rel.as<uint16_t>() + c.rel0, seg0, seglen, sb.scratch.as<uint16_t>(), sb.ldp, sb.prowcap,
      d_err, spin);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

int launch_dedisperse_sub(const DeviceObs &o, uint64_t ntrials, uint64_t n, float *d_out,
                          uint64_t ldo, double *d_part, unsigned *d_err, cudaStream_t st,
                          long long spin, const SubbandPlan &sb, uint64_t chunk_index) {
  const SubbandPlan::Chunk &c = sb.chunks[chunk_index];
  const uint64_t ntiles = (n + SS_TT - 1) / SS_TT;
  auto kern = sb.flush ? k_sub_sum<true> : k_sub_sum<false>;
  PSR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                sb.flush ? SS_SMEM_FLUSH : SS_SMEM));
  for (uint64_t seg0 = 0; seg0 < n; seg0 += sb.seg) {
    const uint64_t len = std::min(sb.seg, n - seg0);
    if (sb.G == 8)
      PSR_TRY(sb.byte_part ? (run_part<8, true>(o, sb, c, seg0, len, d_err, st, spin))
                           : (run_part<8, false>(o, sb, c, seg0, len, d_err, st, spin)));
    else
      PSR_TRY(sb.byte_part ? (run_part<4, true>(o, sb, c, seg0, len, d_err, st, spin))
                           : (run_part<4, false>(o, sb, c, seg0, len, d_err, st, spin)));
    dim3 grid((unsigned)c.nblocks, (unsigned)((len + SS_TT - 1) / SS_TT));
    kern<<<grid, SS_NT, (size_t)sb.nbuf * sb.bufbytes, st>>>(
        sb.scratch.as<uint16_t>(), sb.ldp, sb.stage0.as<uint32_t>() + c.block0,
        sb.rowlist0.as<uint32_t>() + c.block0, sb.stages.as<uint32_t>(), sb.rows.as<SubRow>(),
        sb.info.as<uint32_t>() + c.block0 * SS_TB * sb.nsub, sb.nsub, ntrials, seg0, seg0 + len,
        d_out, ldo, d_part, ntiles, sb.rowcap, sb.bufbytes, sb.nbuf, d_err, spin);
    PSR_CUDA(cudaGetLastError());
  }
  return PSR_OK;
}
}  // namespace

int launch_dedisperse_ex(const DeviceObs &o, const uint32_t *d_delays, uint64_t ntrials,
                         uint64_t n, float *d_out, uint64_t ldo, double *d_part,
                         double *d_sums, float *d_means, uint64_t max_spread, unsigned *d_err,
                         cudaStream_t st, long long spin_limit, int arm_only, bool want_means,
                         const SubbandPlan *sb, uint64_t chunk_index) {
  const long long spin = spin_limit > 0 ? spin_limit : DD_SPIN_LIMIT;
  if (sb && sb->G && !arm_only && o.kind == SAMPLE_U8 && chunk_index < sb->chunks.size()) {
    PSR_TRY(launch_dedisperse_sub(o, ntrials, n, d_out, ldo, d_part, d_err, st, spin, *sb,
                                  chunk_index));
    if (want_means)
      PSR_TRY(reduce_parts(d_part, (n + SS_TT - 1) / SS_TT, ntrials, n, d_sums, d_means, d_out,
                           ldo, 0, st));
    return PSR_OK;
  }
  // Integer samples: channel groups small enough that a group's sum fits the
  // 16-bit lanes (nch * max <= 65535 when there is one group); the groups'
  // sums are added in f32, exact while the total stays below 2^24.
  const double maxv = o.kind == SAMPLE_U8 ? o.max_value() : 0.0;
  const uint64_t gch = maxv > 0.0 ? (uint64_t)(65535.0 / maxv) : 0;
  const bool packed = o.kind == SAMPLE_U8 && gch >= 1 && (double)o.nch * maxv < 16777216.0;
  if (packed) {
    const uint64_t ntiles = (n + DD_TT - 1) / DD_TT;
    int rowcap = (int)(((uint64_t)DD_TT + max_spread + 32 + 15) & ~(uint64_t)15);
    int dev = 0;
    PSR_CUDA(cudaGetDevice(&dev));
    int smax = 0;
    PSR_CUDA(cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    // two CTAs per SM: each gets half of the SM's shared memory
    int smsm = 0;
    PSR_CUDA(cudaDeviceGetAttribute(&smsm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    size_t budget = std::min((size_t)smax, (size_t)smsm / 2) - 4096;
    const uint64_t glen = std::min<uint64_t>(gch, o.nch);
    // The CTA's delay block ([trials per CTA][channels of the group], u32) is
    // preloaded into shared memory when it takes at most 16 KB.
    const int group = (int)(255.0 / maxv);
    // (one trial takes a kernel for one: the block of 8 would add it 8 times)
    const bool one = ntrials == 1;
    const size_t dly_bytes = (size_t)(one ? 1 : group >= 2 ? DD_DB8 : DD_DB) * glen * 4;
    const int preload = dly_bytes <= 16384 && dly_bytes + 2 * (size_t)rowcap <= budget;
    if (preload) budget -= dly_bytes;
    int cc = (int)std::min<uint64_t>({(uint64_t)DD_MAXCC, glen, budget / (2 * (size_t)rowcap)});
    if (cc >= 1) {
      size_t smem = 2 * (size_t)cc * rowcap + (preload ? dly_bytes : 0);
      for (uint64_t c0 = 0; c0 < o.nch; c0 += glen) {
        const uint64_t ng = std::min(glen, o.nch - c0);
        const uint8_t *sg = o.samples.as<uint8_t>() + c0 * o.ld;
        const uint32_t *dg = d_delays + c0;
        const int acc = c0 > 0 ? 1 : 0;
        const int ccg = (int)std::min<uint64_t>((uint64_t)cc, ng);
        auto run = [&](auto kern, int db, int grp) -> int {
          dim3 grid((unsigned)ntiles, (unsigned)((ntrials + db - 1) / db));
          PSR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
          kern<<<grid, DD_NT, smem, st>>>(sg, o.ld, o.ns, ng, o.nch, dg, ntrials, n, d_out, ldo,
                                          d_part, ntiles, ccg, rowcap, grp, acc, d_err, spin,
                                          arm_only);
          return PSR_OK;
        };
        int rc;
        if (one && group >= 2)
          rc = preload ? run(k_dedisp_u8<true, 1, true>, 1, group)
                       : run(k_dedisp_u8<true, 1, false>, 1, group);
        else if (one)
          rc = preload ? run(k_dedisp_u8<false, 1, true>, 1, 1)
                       : run(k_dedisp_u8<false, 1, false>, 1, 1);
        else if (group >= 2)
          rc = preload ? run(k_dedisp_u8<true, DD_DB8, true>, DD_DB8, group)
                       : run(k_dedisp_u8<true, DD_DB8, false>, DD_DB8, group);
        else
          rc = preload ? run(k_dedisp_u8<false, DD_DB, true>, DD_DB, 1)
                       : run(k_dedisp_u8<false, DD_DB, false>, DD_DB, 1);
        if (rc != PSR_OK) return rc;
        PSR_CUDA(cudaGetLastError());
      }
      if (want_means)
        PSR_TRY(reduce_parts(d_part, ntiles, ntrials, n, d_sums, d_means, d_out, ldo, 0, st));
      return PSR_OK;
    }
  }
  const uint64_t ntiles = (n + DG_TT - 1) / DG_TT;
  auto rows = [&](const auto *x, int &rc) -> bool {
    using T = std::remove_cv_t<std::remove_reference_t<decltype(*x)>>;
    int stage, rowcap, nbuf;
    if (arm_only || !rows_plan<T>(o.nch, ntrials, max_spread, stage, rowcap, nbuf)) return false;
    rc = [&]() -> int {
      PSR_CUDA(cudaFuncSetAttribute(k_dedisp_rows<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    DR_SMEM));
      k_dedisp_rows<T><<<dim3((unsigned)ntiles, (unsigned)((ntrials + DR_TB - 1) / DR_TB)), DR_NT,
                         (size_t)nbuf * stage * rowcap, st>>>(
          x, o.ld, o.nch, d_delays, ntrials, n, d_out, ldo, d_part, ntiles, stage, rowcap, nbuf,
          d_err, spin);
      return PSR_OK;
    }();
    return true;
  };
  dim3 grid((unsigned)ntiles, (unsigned)((ntrials + DG_DB - 1) / DG_DB));
  int rc = PSR_OK;
  switch (o.kind) {
    case SAMPLE_U8:
      k_dedisp_generic<uint8_t><<<grid, DG_NT, 0, st>>>(o.samples.as<uint8_t>(), o.ld, o.nch,
                                                        d_delays, ntrials, n, d_out, ldo,
                                                        d_part, ntiles);
      break;
    case SAMPLE_U16:
      if (rows(o.samples.as<const uint16_t>(), rc)) break;
      k_dedisp_generic<uint16_t><<<grid, DG_NT, 0, st>>>(o.samples.as<uint16_t>(), o.ld,
                                                         o.nch, d_delays, ntrials, n, d_out,
                                                         ldo, d_part, ntiles);
      break;
    default:
      if (rows(o.samples.as<const float>(), rc)) break;
      k_dedisp_generic<float><<<grid, DG_NT, 0, st>>>(o.samples.as<float>(), o.ld, o.nch,
                                                      d_delays, ntrials, n, d_out, ldo, d_part,
                                                      ntiles);
  }
  PSR_TRY(rc);
  PSR_CUDA(cudaGetLastError());
  if (want_means)
    PSR_TRY(reduce_parts(d_part, ntiles, ntrials, n, d_sums, d_means, d_out, ldo,
                         o.kind == SAMPLE_F32 ? 1 : 0, st));
  return PSR_OK;
}

uint64_t dedisperse_part_count(const DeviceObs &o, uint64_t n) {
  // f32 samples: sums, sums of |x| and quanta per tile
  const uint64_t per = o.kind == SAMPLE_F32 ? 3 : 1;
  return per * std::max((n + DD_TT - 1) / DD_TT, (n + DG_TT - 1) / DG_TT);
}

}  // namespace psr

extern "C" int psr_test_subband_plan(const uint32_t *delays, uint64_t nch, uint64_t ntrials,
                                     uint64_t chunk, uint64_t n, double max_value, int subbands,
                                     int once, uint64_t *info) {
  if (!delays || !info || nch == 0 || ntrials == 0 || chunk == 0) {
    psr::set_error("test_subband_plan: a delay table and room for the result");
    return PSR_EINVAL;
  }
  std::vector<uint64_t> cstart;
  for (uint64_t t = 0; t < ntrials; t += chunk) cstart.push_back(t);
  cstart.push_back(ntrials);
  psr::SubbandTables t;
  psr::choose_subband_tables(std::vector<uint32_t>(delays, delays + nch * ntrials), nch, n,
                             max_value, cstart, subbands, once != 0, psr::SUB_SCRATCH, t);
  const psr::SubbandPlan::Shape &p = t.shape;
  info[0] = (uint64_t)p.G;
  info[1] = p.flush;
  info[2] = p.seg;
  info[3] = p.seg ? (n + p.seg - 1) / p.seg : 0;
  info[4] = p.scratch_bytes;
  return PSR_OK;
}

extern "C" int psr_set_dedisp_subbands(int subbands) {
  if (subbands != -1 && subbands != 0 && subbands != 4 && subbands != 8) {
    psr::set_error("set_dedisp_subbands: -1, 0, 4 or 8");
    return PSR_EINVAL;
  }
  psr::g_subbands.store(subbands);
  return PSR_OK;
}
