// K4 real FFT + raw power (search/src/lib.rs:35-44).
//
// The FFT is a fixed FP32 algorithm, reproduced operation for operation by
// the CPU oracle so that spectra (and everything downstream) are bit-exact:
//   N = 2*next_pow2(len) real points, M = N/2 complex points,
//   z[n] = x[2n] + i x[2n+1],  x[i] = series[i] - (f32)mean  (0 beyond len).
//   Twiddles W_N^x come from a quarter table ((f32)cos, (f32)sin of 2 pi r/N
//   for r <= N/8, mirrored above) and exact quadrant symmetry.
//   cmul(a, w) = (fma(a.re, w.re, -(a.im*w.im)), fma(a.re, w.im, a.im*w.re)).
//   M <= 4096: one Stockham sub-FFT.  Otherwise four-step M = M1*M2,
//   M1 = 2^ceil(m/2): pass 1 = column sub-FFTs over n1 (n = n1*M2 + n2) and
//   the twiddle W_M^(n2*k1); pass 2 = row sub-FFTs, fused with the real
//   post-processing X[k] = 0.5*(e.re + t.im, e.im - t.re), e = a + b,
//   t = cmul(a - b, W_N^k), a = Z[k], b = conj(Z[M-k]), and |X|^2.
//   Sub-FFT of size L: Stockham autosort stages with radices
//   [16]*(q/4) + [2|4|8]; DFT_8 = 2x4 and DFT_16 = 4x4 four-step with the
//   internal twiddles W_R^(n2*k1).
// A CTA transforms C columns (pass 1) or rows (pass 2) held in shared memory
// with one padding slot every 16 positions: position-major for columns,
// row-major for rows, each free of bank conflicts for its stages.  Every size
// is a template parameter, so all index arithmetic reduces to shifts and
// masks; each thread owns exactly one radix-16 butterfly per stage.  Stages
// are in place: every thread loads its inputs, the block synchronises, then
// stores.  The first stage's inputs come straight from where they lie (the
// staged series, the work buffer) and the last stage's outputs leave from
// registers (times the pass-1 twiddle to the work buffer; through the real
// post-processing to the spectrum), so a sub-FFT of three stages makes two
// round trips through shared memory.
// Bound: instruction issue (about 2.5 M warp instructions per 2^20-point
// trial) at half occupancy (64 registers, 2 CTAs of 512 threads per SM).
// Measured on a GB300, 2^20 points, 700 trials: pass 1 1.68 -> 1.55 ms, pass 2
// 1.67 -> 1.37 ms against stages that all went through shared memory.
#include <cuda_runtime.h>

#include <type_traits>

#include <algorithm>
#include <cmath>
#include <vector>

#include "psr_internal.h"

namespace psr {
namespace {

__host__ __device__ constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x >> 1); }
__host__ __device__ constexpr int cols_for(int L) {
  return L >= 8192 ? 1 : (8192 / L > 16 ? 16 : 8192 / L);
}
__host__ __device__ constexpr int threads_for(int L, int C) {
  return ((L / 16) * C < 32 ? 32 : (L / 16) * C);
}

// Shared-memory slot of (position, column) for C columns: the linear index
// e = pos*C + col padded by one slot every 16 (conflict-free for the fill,
// every Stockham load/store pattern and the drains of both passes).
template <int C>
__device__ __forceinline__ int lay(int pos, int col) {
  const int e = pos * C + col;
  return e + (e >> 4);
}
template <int L, int C>
__host__ __device__ constexpr int lay_slots() {
  return L * C + (L * C) / 16 + 1;
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y));
}
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
  return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)),
                     __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}
__device__ __forceinline__ float2 mul_mi(float2 d) { return make_float2(d.y, -d.x); }

// W_N^x for x in [0, N) from the quarter table (lq = log2(N/4)).
__device__ __forceinline__ float2 twN(const float2 *__restrict__ Q, uint32_t x, int lq) {
  const uint32_t q = x >> lq, r = x & ((1u << lq) - 1u);
  const float2 v = __ldg(&Q[r]);
  switch (q & 3u) {
    case 0: return make_float2(v.x, -v.y);
    case 1: return make_float2(-v.y, -v.x);
    case 2: return make_float2(-v.x, v.y);
    default: return make_float2(v.y, v.x);
  }
}

__device__ __forceinline__ void dft2(float2 &v0, float2 &v1) {
  const float2 a = v0, b = v1;
  v0 = cadd(a, b);
  v1 = csub(a, b);
}
__device__ __forceinline__ void dft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3) {
  float2 a = cadd(v0, v2), b = csub(v0, v2);
  float2 c = cadd(v1, v3), d = mul_mi(csub(v1, v3));
  v0 = cadd(a, c);
  v1 = cadd(b, d);
  v2 = csub(a, c);
  v3 = csub(b, d);
}
// The internal twiddles of the radix-8 and radix-16 butterflies, W_16^y for
// y in {1, 2, 3, 4, 6, 9}, held in registers.  W_L^(y L/16) is the table
// entry for x = y N/16 whatever L is, so one set serves every sub-FFT size;
// load_w16 reads them from a sub-FFT's table (values identical to the table
// lookups they replace).
struct W16 {
  float2 w1, w2, w3, w4, w6, w9;
  template <int Y>
  __device__ __forceinline__ float2 get() const {
    static_assert(Y == 1 || Y == 2 || Y == 3 || Y == 4 || Y == 6 || Y == 9, "W_16 power");
    if constexpr (Y == 1) return w1;
    else if constexpr (Y == 2) return w2;
    else if constexpr (Y == 3) return w3;
    else if constexpr (Y == 4) return w4;
    else if constexpr (Y == 6) return w6;
    else return w9;
  }
};
template <int L>
__device__ __forceinline__ W16 load_w16(const float2 *Wl) {
  W16 c{};
  if constexpr (L >= 16) {
    c.w1 = Wl[1 * (L / 16)];
    c.w2 = Wl[2 * (L / 16)];
    c.w3 = Wl[3 * (L / 16)];
    c.w4 = Wl[4 * (L / 16)];
    c.w6 = Wl[6 * (L / 16)];
    c.w9 = Wl[9 * (L / 16)];
  } else if constexpr (L == 8) {  // W_8^n2 = W_16^(2 n2)
    c.w2 = Wl[1];
    c.w4 = Wl[2];
    c.w6 = Wl[3];
  }
  return c;
}

// W_R^y = W_16^(y 16/R).
__device__ __forceinline__ void dft8(float2 *v, const W16 &c) {
  float2 u[4][2];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    float2 a = v[n2], b = v[n2 + 4];
    dft2(a, b);
    u[n2][0] = a;
    u[n2][1] = b;
  }
  u[1][1] = cmul(u[1][1], c.get<2>());
  u[2][1] = cmul(u[2][1], c.get<4>());
  u[3][1] = cmul(u[3][1], c.get<6>());
#pragma unroll
  for (int k1 = 0; k1 < 2; ++k1) {
    float2 a = u[0][k1], b = u[1][k1], c = u[2][k1], d = u[3][k1];
    dft4(a, b, c, d);
    v[k1] = a;
    v[k1 + 2] = b;
    v[k1 + 4] = c;
    v[k1 + 6] = d;
  }
}
// The internal twiddles and second level of dft16.
__device__ __forceinline__ void dft16_second(float2 (&u)[4][4], float2 *v, const W16 &c) {
  u[1][1] = cmul(u[1][1], c.get<1>());
  u[1][2] = cmul(u[1][2], c.get<2>());
  u[1][3] = cmul(u[1][3], c.get<3>());
  u[2][1] = cmul(u[2][1], c.get<2>());
  u[2][2] = cmul(u[2][2], c.get<4>());
  u[2][3] = cmul(u[2][3], c.get<6>());
  u[3][1] = cmul(u[3][1], c.get<3>());
  u[3][2] = cmul(u[3][2], c.get<6>());
  u[3][3] = cmul(u[3][3], c.get<9>());
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    float2 a = u[0][k1], b = u[1][k1], c = u[2][k1], d = u[3][k1];
    dft4(a, b, c, d);
    v[k1] = a;
    v[k1 + 4] = b;
    v[k1 + 8] = c;
    v[k1 + 12] = d;
  }
}
__device__ __forceinline__ void dft16(float2 *v, const W16 &c) {
  float2 u[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    float2 a = v[n2], b = v[n2 + 4], c = v[n2 + 8], d = v[n2 + 12];
    dft4(a, b, c, d);
    u[n2][0] = a;
    u[n2][1] = b;
    u[n2][2] = c;
    u[n2][3] = d;
  }
  dft16_second(u, v, c);
}

// dft16 of inputs whose second half (v[8..15]) is zero: the first level's sums
// with zero are skipped (the same values up to the sign of zero, which cannot
// change |X|^2).
__device__ __forceinline__ void dft16_half(float2 *v, const W16 &c) {
  float2 u[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    const float2 a = v[n2], b = v[n2 + 4], d = mul_mi(b);
    u[n2][0] = cadd(a, b);
    u[n2][1] = cadd(a, d);
    u[n2][2] = csub(a, b);
    u[n2][3] = csub(a, d);
  }
  dft16_second(u, v, c);
}

template <int R>
__device__ __forceinline__ void dftR(float2 *v, const W16 &c) {
  if constexpr (R == 2) dft2(v[0], v[1]);
  else if constexpr (R == 4) dft4(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 8) dft8(v, c);
  else dft16(v, c);
}

// One in-place Stockham stage (radix R, Ns = product of earlier radices) on
// C columns of length L; NT threads, each owning 16/R butterflies.
// Slot distance of D positions when D*C is a multiple of 16 (the padding is
// then D*C/16 slots): lay<C>(p + D, c) = lay<C>(p, c) + lay_step<C, D>().
template <int C, int D>
__host__ __device__ constexpr int lay_step() {
  return D * C + (D * C) / 16;
}

template <int R, int L, int C, int NT, int Ns>
__device__ __forceinline__ void stage(float2 *sm, const float2 *Wl, const W16 &c16) {
  constexpr int nb = L / R;
  constexpr int total = nb * C;
  constexpr int BPT = (total + NT - 1) / NT;
  float2 v[BPT][R];
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int w = (int)threadIdx.x + i * NT;
    if (total % NT == 0 || w < total) {
      const int col = w % C, j = w / C;
      if constexpr ((nb * C) % 16 == 0) {
        const float2 *src = sm + lay<C>(j, col);
#pragma unroll
        for (int r = 0; r < R; ++r) v[i][r] = src[r * lay_step<C, nb>()];
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[i][r] = sm[lay<C>(j + r * nb, col)];
      }
      if constexpr (Ns > 1) {
        const int k = j % Ns;
        if (k != 0) {
#pragma unroll
          for (int r = 1; r < R; ++r) v[i][r] = cmul(v[i][r], Wl[r * k * (L / (Ns * R))]);
        }
      }
      dftR<R>(v[i], c16);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int w = (int)threadIdx.x + i * NT;
    if (total % NT == 0 || w < total) {
      const int col = w % C, j = w / C;
      const int base = (j / Ns) * Ns * R + j % Ns;
      if constexpr ((Ns * C) % 16 == 0) {
        float2 *dst = sm + lay<C>(base, col);
#pragma unroll
        for (int r = 0; r < R; ++r) dst[r * lay_step<C, Ns>()] = v[i][r];
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) sm[lay<C>(base + r * Ns, col)] = v[i][r];
      }
    }
  }
  __syncthreads();
}

template <int L, int C, int NT, int s>
__device__ __forceinline__ void stages16(float2 *sm, const float2 *Wl, const W16 &c) {
  if constexpr (s < ilog2(L) / 4) {
    stage<16, L, C, NT, (1 << (4 * s))>(sm, Wl, c);
    stages16<L, C, NT, s + 1>(sm, Wl, c);
  }
}

// Radix and stride (product of the earlier radices) of a sub-FFT's last stage.
__host__ __device__ constexpr int last_radix(int L) {
  return ilog2(L) % 4 == 0 ? 16 : 1 << (ilog2(L) % 4);
}

// The radix-16 stages s, s + 1, .. before the last stage.
template <int L, int C, int NT, int s>
__device__ __forceinline__ void stages_mid(float2 *sm, const float2 *Wl, const W16 &c) {
  if constexpr ((1 << (4 * s)) * last_radix(L) < L) {
    stage<16, L, C, NT, (1 << (4 * s))>(sm, Wl, c);
    stages_mid<L, C, NT, s + 1>(sm, Wl, c);
  }
}

// The last stage, its outputs handed to emit(j, col, v) instead of stored:
// butterfly (col, j) leaves v[r] at position j + r L / R.
template <int L, int C, int NT, class Emit>
__device__ __forceinline__ void last_stage(const float2 *sm, const float2 *Wl, const W16 &c16,
                                           Emit emit) {
  constexpr int R = last_radix(L), nb = L / R, total = nb * C, BPT = (total + NT - 1) / NT;
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int w = (int)threadIdx.x + i * NT;
    if (total % NT == 0 || w < total) {
      const int col = w % C, j = w / C;
      float2 v[R];
      if constexpr ((nb * C) % 16 == 0) {
        const float2 *src = sm + lay<C>(j, col);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[r * lay_step<C, nb>()];
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = sm[lay<C>(j + r * nb, col)];
      }
      if (j != 0) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul(v[r], Wl[r * j]);
      }
      dftR<R>(v, c16);
      emit(j, col, v);
    }
  }
}

template <int L, int C, int NT>
__device__ __forceinline__ void subfft(float2 *sm, const float2 *Wl, const W16 &c) {
  constexpr int q = ilog2(L);
  constexpr int NsLast = 1 << (4 * (q / 4));
  stages16<L, C, NT, 0>(sm, Wl, c);
  if constexpr (q % 4 == 1) stage<2, L, C, NT, NsLast>(sm, Wl, c);
  else if constexpr (q % 4 == 2) stage<4, L, C, NT, NsLast>(sm, Wl, c);
  else if constexpr (q % 4 == 3) stage<8, L, C, NT, NsLast>(sm, Wl, c);
}

template <int L>
__device__ __forceinline__ void build_wl(float2 *Wl, uint32_t N, const float2 *Q, int lq) {
  const uint32_t stride = N / (uint32_t)L;
  for (int y = threadIdx.x; y < L; y += blockDim.x) Wl[y] = twN(Q, (uint32_t)y * stride, lq);
}

// Real post-processing of one bin: a = Z[k], b = conj(Z[M-k]).
__device__ __forceinline__ float post_power(float2 a, float2 zb, float2 w) {
  const float2 b = make_float2(zb.x, -zb.y);
  const float2 e = cadd(a, b), o = csub(a, b);
  const float2 t = cmul(o, w);
  const float xr = __fmul_rn(0.5f, __fadd_rn(e.x, t.y));
  const float xi = __fmul_rn(0.5f, __fsub_rn(e.y, t.x));
  return __fadd_rn(__fmul_rn(xr, xr), __fmul_rn(xi, xi));
}

// Both bins of a mirrored pair at once: pk from a = zk, b = conj(zm) with
// W_N^k = w, and pm from a = zm, b = conj(zk) with W_N^(M-k) = (-w.re, w.im).
// The mirror's e, o and t are exactly (e.re, -e.im), (-o.re, o.im) and
// (t.re, -t.im) (round to nearest is symmetric in sign and the fma products
// are the same), so pm equals post_power(zm, zk, (-w.re, w.im)) bit for bit.
__device__ __forceinline__ void post_power_pair(float2 zk, float2 zm, float2 w, float &pk,
                                                float &pm) {
  const float2 b = make_float2(zm.x, -zm.y);
  const float2 e = cadd(zk, b), o = csub(zk, b);
  const float2 t = cmul(o, w);
  const float xr = __fmul_rn(0.5f, __fadd_rn(e.x, t.y));
  const float xi = __fmul_rn(0.5f, __fsub_rn(e.y, t.x));
  pk = __fadd_rn(__fmul_rn(xr, xr), __fmul_rn(xi, xi));
  const float yr = __fmul_rn(0.5f, __fsub_rn(e.x, t.y));
  const float yi = __fmul_rn(0.5f, __fadd_rn(e.y, t.x));  // -(mirror's xi)
  pm = __fadd_rn(__fmul_rn(yr, yr), __fmul_rn(yi, yi));
}

__device__ __forceinline__ float2 load_z(const float *__restrict__ row, uint64_t len, uint64_t n,
                                         float mean) {
  const uint64_t i0 = 2 * n;
  float x0 = 0.0f, x1 = 0.0f;
  if (i0 + 1 < len) {
    const float2 p = *reinterpret_cast<const float2 *>(row + i0);
    x0 = __fsub_rn(p.x, mean);
    x1 = __fsub_rn(p.y, mean);
  } else if (i0 < len) {
    x0 = __fsub_rn(row[i0], mean);
  }
  return make_float2(x0, x1);
}

// Partial sums of the power spectrum for the normalisation floor: f32
// TwoSum (error-free transformation) per thread, f64 across threads.
struct Acc2 {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void add(float b) {
    const float s = __fadd_rn(hi, b);
    const float bb = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    hi = s;
    lo = __fadd_rn(lo, err);
  }
};

// Block total of the per-thread (hi, lo) pairs: TwoSum merges across the warp in
// f32, the warps' pairs in f64, a lane each (FP64 runs at 1/64 of the f32 rate:
// 16 pairs added by one thread held every CTA of pass 2 for about 1500 cycles).
template <int NT>
__device__ __forceinline__ void block_sum_store(Acc2 acc, double *dst) {
  constexpr int NW = NT / 32 > 0 ? NT / 32 : 1;
  __shared__ float2 red[NW];
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float oh = __shfl_down_sync(0xffffffffu, acc.hi, o);
    const float ol = __shfl_down_sync(0xffffffffu, acc.lo, o);
    acc.add(oh);
    acc.lo = __fadd_rn(acc.lo, ol);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(acc.hi, acc.lo);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int w = (int)threadIdx.x;
    double t = w < NW ? (double)red[w].x + (double)red[w].y : 0.0;
#pragma unroll
    for (int o = NW / 2; o; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (w == 0) *dst = t;
  }
}

// Whole transform in one CTA per trial (M <= 4096).
template <int M>
__global__ void __launch_bounds__(threads_for(M, 1))
    k_fft_small(const float *__restrict__ series, uint64_t lds, uint64_t len,
                const float *__restrict__ means, const float2 *__restrict__ Q, int lq,
                uint32_t N, float *__restrict__ power, uint64_t ldp,
                double *__restrict__ psum) {
  constexpr int NT = threads_for(M, 1);
  extern __shared__ float2 dyn[];
  float2 *Wl = dyn;      // M entries
  float2 *sm = dyn + M;  // lay_slots<M, 1>() entries
  const uint64_t trial = blockIdx.x;
  const float *row = series + trial * lds;
  const float mean = means[trial];
  build_wl<M>(Wl, N, Q, lq);
  for (int n = threadIdx.x; n < M; n += NT) sm[lay<1>(n, 0)] = load_z(row, len, (uint64_t)n, mean);
  __syncthreads();
  const W16 c16 = load_w16<M>(Wl);
  subfft<M, 1, NT>(sm, Wl, c16);
  Acc2 acc;
  float *out = power + trial * ldp;
  for (int k = threadIdx.x; k <= M; k += NT) {
    const float p =
        post_power(sm[lay<1>(k % M, 0)], sm[lay<1>((M - k) % M, 0)], twN(Q, (uint32_t)k, lq));
    out[k] = p;
    acc.add(p);
  }
  block_sum_store<NT>(acc, psum + trial);
}

// z[n] from a staged pair of series values (as load_z reads them).
__device__ __forceinline__ float2 staged_z(float2 p, uint64_t len, uint64_t n, float mean) {
  const uint64_t i0 = 2 * n;
  if (i0 + 1 < len) return make_float2(__fsub_rn(p.x, mean), __fsub_rn(p.y, mean));
  if (i0 < len) return make_float2(__fsub_rn(p.x, mean), 0.0f);
  return make_float2(0.0f, 0.0f);
}

// 16-byte asynchronous global -> shared copy, cached in L2 only.
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// Copies the non-zero rows n1 < ceil(nz / M2) of column group n2_0 of `row`
// into stg[n1 * C + c] (float pairs), 16 bytes per thread and step; chunks
// starting at or past len are left alone (stage 0 never reads them).
template <int M1, int M2>
__device__ __forceinline__ void p1_stage_rows(float2 *stg, const float *__restrict__ row,
                                              uint64_t len, uint32_t n2_0) {
  constexpr int C = cols_for(M1), NT = threads_for(M1, C);
  static_assert(C % 2 == 0, "16-byte chunks of complex pairs");
  const uint64_t nz = (len + 1) / 2;
  const int rows = (int)((nz + M2 - 1) / M2);
  const int nchunk = rows * (C / 2);
  for (int q = threadIdx.x; q < nchunk; q += NT) {
    const int n1 = q / (C / 2), part = q % (C / 2);
    const uint64_t f = 2 * ((uint64_t)n1 * M2 + n2_0) + 4 * (uint64_t)part;
    if (f < len) cp_async16(stg + n1 * C + 2 * part, row + f);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Pass 1 on one column group: C columns n2 in [n2_0, n2_0 + C) of trial
// `row` (length M1 over n1), then W_M^(n2*k1), written to out[k1*M2 + n2].
// stg (if not null) holds the group's non-zero rows (p1_stage_rows);
// after_stage0() runs once every thread is done with stg.
template <int M1, int M2, class Hook>
__device__ __forceinline__ void p1_group(float2 *sm, const float2 *Wl, const W16 &c16,
                                         const float *__restrict__ row, uint64_t len,
                                         float mean, uint32_t n2_0,
                                         const float2 *__restrict__ tw1,
                                         float2 *__restrict__ out, const float2 *stg,
                                         Hook after_stage0) {
  constexpr int C = cols_for(M1), NT = threads_for(M1, C);
  const uint64_t nz = (len + 1) / 2;  // complex inputs that can be non-zero
  {
    // Stage 0 (radix 16, Ns = 1) straight from global memory (or the staged
    // rows): butterfly (col, j) takes positions j + r*M1/16 of its column and
    // stores its outputs at 16j + r.  The zero padding (n >= nz) is never
    // loaded.
    constexpr int nb = M1 / 16;
    constexpr int nbt = nb * C;
    constexpr int BPT = (nbt + NT - 1) / NT;
#pragma unroll
    for (int i = 0; i < BPT; ++i) {
      const int w = (int)threadIdx.x + i * NT;
      if (nbt % NT == 0 || w < nbt) {
        const int col = w % C, j = w / C;
        // (at most half the inputs can be non-zero: r < 8)
        float2 v[16];
        if (stg) {
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const uint64_t n = (uint64_t)(j + r * nb) * M2 + n2_0 + col;
            v[r] = n < nz ? staged_z(stg[(j + r * nb) * C + col], len, n, mean)
                          : make_float2(0.0f, 0.0f);
          }
        } else {
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const uint64_t n = (uint64_t)(j + r * nb) * M2 + n2_0 + col;
            v[r] = n < nz ? load_z(row, len, n, mean) : make_float2(0.0f, 0.0f);
          }
        }
        dft16_half(v, c16);
        if constexpr (16 % C == 0) {
          // e = (16j + r) C + col with col < C | 16: the padding of r C +
          // col is (r C) / 16, so every r is a constant offset
          float2 *dst = sm + 17 * C * j + col;
#pragma unroll
          for (int r = 0; r < 16; ++r) dst[r * C + (r * C) / 16] = v[r];
        } else {
#pragma unroll
          for (int r = 0; r < 16; ++r) sm[lay<C>(16 * j + r, col)] = v[r];
        }
      }
    }
  }
  __syncthreads();
  after_stage0();
  stages_mid<M1, C, NT, 1>(sm, Wl, c16);
  // W_M^(n2*k1) comes from a table laid out like the output, Tw1[k1*M2 +
  // n2] (values identical to the quarter-table lookup): reads coalesce.
  last_stage<M1, C, NT>(sm, Wl, c16, [&](int j, int col, float2 *v) {
    constexpr int R = last_radix(M1), nb = M1 / R;
    const uint32_t n2 = n2_0 + (uint32_t)col;
    const uint64_t at = (uint64_t)j * M2 + n2;
    float2 w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = __ldg(tw1 + at + (uint64_t)r * nb * M2);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (n2 * (uint32_t)(j + r * nb) != 0) v[r] = cmul(v[r], w[r]);
      out[at + (uint64_t)r * nb * M2] = v[r];
    }
  });
}

// Pass 1: column groups of every trial, persistent: CTA b takes groups b,
// b + gridDim.x, ... (group g = trial g / (M2/C), columns (g % (M2/C)) C
// ...), builds the twiddle table once, and while it transforms one group
// prefetches the next group's samples into L2 (one 64-byte run of C complex
// inputs per row).
// STAGED: the next group's non-zero rows are copied into shared memory
// (cp.async) while the CTA transforms the current group, instead of
// prefetched into L2, so stage 0 reads shared memory.
template <int M1, int M2, bool STAGED>
__global__ void __launch_bounds__(threads_for(M1, cols_for(M1)), 2)
    k_fft_pass1(const float *__restrict__ series, uint64_t lds, uint64_t len,
                const float *__restrict__ means, const float2 *__restrict__ Q, int lq,
                uint32_t N, const float2 *__restrict__ tw1, float2 *__restrict__ work,
                uint32_t ngroups) {
  constexpr int C = cols_for(M1);
  constexpr uint32_t M = (uint32_t)M1 * M2;
  constexpr uint32_t GPT = M2 / C;  // column groups per trial
  extern __shared__ float2 dyn[];
  float2 *Wl = dyn;       // M1 entries
  float2 *sm = dyn + M1;  // lay_slots<M1, C>() entries
  // staged rows after sm, rounded up to 16 bytes (the launch adds one slot)
  float2 *stg = STAGED ? reinterpret_cast<float2 *>(
                             (reinterpret_cast<uintptr_t>(sm + lay_slots<M1, C>()) + 15) &
                             ~(uintptr_t)15)
                       : nullptr;
  if constexpr (STAGED) {
    if (blockIdx.x < ngroups)
      p1_stage_rows<M1, M2>(stg, series + (uint64_t)(blockIdx.x / GPT) * lds, len,
                            (blockIdx.x % GPT) * (uint32_t)C);
  }
  build_wl<M1>(Wl, N, Q, lq);
  const uint64_t nz = (len + 1) / 2;
  __syncthreads();  // Wl
  const W16 c16 = load_w16<M1>(Wl);
  for (uint32_t grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    const uint64_t trial = grp / GPT;
    const uint32_t n2_0 = (grp % GPT) * (uint32_t)C;
    const uint32_t nx = grp + gridDim.x;
    if constexpr (STAGED) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // this group's rows are in stg
      p1_group<M1, M2>(sm, Wl, c16, series + trial * lds, len, means[trial], n2_0, tw1,
                       work + trial * (uint64_t)M, stg, [&]() {
                         if (nx < ngroups)
                           p1_stage_rows<M1, M2>(stg, series + (uint64_t)(nx / GPT) * lds, len,
                                                 (nx % GPT) * (uint32_t)C);
                       });
    } else {
      // (only inputs the next group loads: complex index < nz)
      const uint64_t pn = (uint64_t)threadIdx.x * M2 + (nx % GPT) * (uint32_t)C;
      if (nx < ngroups && pn < nz) {
        const float *pr = series + (uint64_t)(nx / GPT) * lds + 2 * pn;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(pr));
      }
      p1_group<M1, M2>(sm, Wl, c16, series + trial * lds, len, means[trial], n2_0, tw1,
                       work + trial * (uint64_t)M, nullptr, []() {});
    }
    __syncthreads();  // the next group's stage 0 overwrites sm
  }
}

// Pass 2's shared-memory layout: row ci starts at ci * p2_pitch, position pos
// at pos + pos / 16 of it.  Warps run along a row in the radix-16 stages
// (conflict-free by the padding); in the last stage a half-warp reads H rows
// x 16 / H positions, which the pitch (16 / H modulo 16) keeps in 16 different
// bank pairs.
template <int L>
__host__ __device__ constexpr int p2_pitch() {
  constexpr int H = cols_for(L) / 2, base = L + L / 16;
  return base + (16 / H + 16 - base % 16) % 16;
}
__device__ __forceinline__ int p2_slot(int pos) { return pos + (pos >> 4); }

// One in-place stage on C rows; W1 is the second stage's twiddle table
// [r][k] = W_L^(r k L / 256) (its lanes' 16 values of k are contiguous).
template <int R, int L, int C, int NT, int Ns>
__device__ __forceinline__ void stage_rows(float2 *sm, const float2 *Wl, const float2 *W1,
                                           const W16 &c16) {
  constexpr int nb = L / R, total = nb * C, BPT = (total + NT - 1) / NT, P = p2_pitch<L>();
  float2 v[BPT][R];
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int w = (int)threadIdx.x + i * NT, row = w / nb, j = w % nb;
    if (total % NT == 0 || w < total) {
      const float2 *src = sm + row * P;
#pragma unroll
      for (int r = 0; r < R; ++r) v[i][r] = src[p2_slot(j + r * nb)];
      const int k = j % Ns;
      if (k != 0) {
#pragma unroll
        for (int r = 1; r < R; ++r)
          v[i][r] = cmul(v[i][r], R == 16 && Ns == 16 ? W1[r * 16 + k]
                                                      : Wl[r * k * (L / (Ns * R))]);
      }
      dftR<R>(v[i], c16);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int w = (int)threadIdx.x + i * NT, row = w / nb, j = w % nb;
    if (total % NT == 0 || w < total) {
      float2 *dst = sm + row * P;
      const int base = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
      for (int r = 0; r < R; ++r) dst[p2_slot(base + r * Ns)] = v[i][r];
    }
  }
  __syncthreads();
}
template <int L, int C, int NT, int s>
__device__ __forceinline__ void stages_rows_mid(float2 *sm, const float2 *Wl, const float2 *W1,
                                                const W16 &c) {
  if constexpr ((1 << (4 * s)) * last_radix(L) < L) {
    stage_rows<16, L, C, NT, (1 << (4 * s))>(sm, Wl, W1, c);
    stages_rows_mid<L, C, NT, s + 1>(sm, Wl, W1, c);
  }
}

// Pass 2 on one row group of one trial: the row sub-FFTs of length M2, then
// the real post-processing and |X|^2.  Group 0 holds rows 0 and M1/2; group
// g >= 1 holds rows kb..kb+h-1 (kb = 1 + (g-1)*H) and M1-kb..M1-kb-h+1.
// Unused rows of the last group are zero and never written out.
// The first stage takes its inputs from the work buffer (16 loads in flight
// per thread while the CTA builds its twiddle tables).  Bin k2 of row k pairs
// with bin M2 - 1 - k2 of row M1 - k, and the last stage's butterfly j leaves
// bins j + r M2 / R: butterfly j of a row and butterfly M2 / R - 1 - j of its
// mirror hold R whole pairs, so one thread takes both and post-processes them
// in registers.  (Where the last radix is 16 the two would not fit: the stage
// goes through shared memory, as group 0's, whose rows pair differently.)
template <int M1, int M2>
__device__ __forceinline__ void p2_group(float2 *sm, float2 *Wl, float2 *W1, uint32_t N,
                                         const float2 *__restrict__ in, uint32_t g,
                                         const float2 *__restrict__ Q, int lq,
                                         float *__restrict__ out, double *__restrict__ psum_out) {
  constexpr int C = cols_for(M2), NT = threads_for(M2, C), H = C / 2, P = p2_pitch<M2>();
  constexpr uint32_t M = (uint32_t)M1 * M2;
  constexpr int nb0 = M2 / 16, R = last_radix(M2), nbl = M2 / R;
  int h;
  uint32_t kb = 0;
  if (g == 0) {
    h = 1;
  } else {
    kb = 1 + (g - 1) * (uint32_t)H;
    h = (int)min((uint32_t)H, (uint32_t)(M1 / 2 - kb));
  }
  auto row_of = [&](int ci) -> uint32_t {
    if (g == 0) return ci == 0 ? 0u : (uint32_t)(M1 / 2);
    return ci < H ? kb + (uint32_t)ci : (uint32_t)M1 - (kb + (uint32_t)(ci - H));
  };
  {
    static_assert(nb0 * C == NT, "one first-stage butterfly per thread");
    const int ci = (int)threadIdx.x / nb0, j = (int)threadIdx.x % nb0;
    float2 v[16];
    if (g == 0 ? ci < 2 : ci % H < h) {
      const float2 *src = in + (uint64_t)row_of(ci) * M2 + j;
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = src[r * nb0];
    } else {
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = make_float2(0.0f, 0.0f);
    }
    build_wl<M2>(Wl, N, Q, lq);
    if constexpr (M2 >= 256)
      for (int t = threadIdx.x; t < 256; t += NT)
        W1[t] = twN(Q, (uint32_t)((t >> 4) * (t & 15)) * (N / 256), lq);
    __syncthreads();
    const W16 c16 = load_w16<M2>(Wl);
    dft16(v, c16);
    float2 *dst = sm + ci * P + 17 * j;  // p2_slot(16 j + r) = 17 j + r
#pragma unroll
    for (int r = 0; r < 16; ++r) dst[r] = v[r];
  }
  __syncthreads();
  const W16 c16 = load_w16<M2>(Wl);
  stages_rows_mid<M2, C, NT, 1>(sm, Wl, W1, c16);
  Acc2 acc;
  if (g != 0 && R < 16) {
    // Full twiddle of bin k = kb + p + M1 k2: k2 < M2 / 2 (r < R / 2) lies in
    // the first quarter of the quarter-table's cycle, the rest in the second
    // (the quadrant rule of twN, fixed per r).  W_N^(M-k) = (-W_N^k.re,
    // W_N^k.im) holds bit for bit for the lookup (its mirrored half is the
    // swapped first half), up to the sign of zero components, which cannot
    // change |X|^2.
    constexpr int PPT = (H * nbl + NT - 1) / NT;
    static_assert(R == 16 || (H * nbl) % NT == 0, "whole pairs per thread");
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
      const int idx = (int)threadIdx.x + i * NT, p = idx % H, j = idx / H, jm = nbl - 1 - j;
      const uint32_t k0 = kb + (uint32_t)p + (uint32_t)M1 * (uint32_t)j;
      float2 wk[R], a[R], b[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 q = __ldg(&Q[k0 + (uint32_t)M1 * (uint32_t)nbl * (r < R / 2 ? r : r - R / 2)]);
        wk[r] = r < R / 2 ? make_float2(q.x, -q.y) : make_float2(-q.y, -q.x);
      }
      const float2 *sa = sm + p * P + p2_slot(j), *sb = sm + (H + p) * P + p2_slot(jm);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        a[r] = sa[r * (nbl + nbl / 16)];
        b[r] = sb[r * (nbl + nbl / 16)];
      }
      if (j != 0) {
#pragma unroll
        for (int r = 1; r < R; ++r) a[r] = cmul(a[r], Wl[r * j]);
      }
      if (jm != 0) {
#pragma unroll
        for (int r = 1; r < R; ++r) b[r] = cmul(b[r], Wl[r * jm]);
      }
      dftR<R>(a, c16);
      dftR<R>(b, c16);
      if (p < h) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t k = k0 + (uint32_t)M1 * (uint32_t)(r * nbl);
          float pk, pm;
          post_power_pair(a[r], b[R - 1 - r], wk[r], pk, pm);
          out[k] = pk;
          out[M - k] = pm;
          acc.add(pk);
          acc.add(pm);
        }
      }
    }
  } else {
    stage_rows<R, M2, C, NT, nbl>(sm, Wl, W1, c16);
    if (g == 0) {
      for (uint32_t idx = threadIdx.x; idx < 2 * M2; idx += NT) {
        const uint32_t k2 = idx % M2, which = idx / M2;
        uint32_t k, mk2;
        if (which == 0) {
          k = M1 * k2;
          mk2 = (M2 - k2) % M2;
        } else {
          k = M1 / 2 + M1 * k2;
          mk2 = M2 - 1 - k2;
        }
        const float2 *row = sm + which * P;
        const float p = post_power(row[p2_slot((int)k2)], row[p2_slot((int)mk2)], twN(Q, k, lq));
        out[k] = p;
        acc.add(p);
      }
      if (threadIdx.x == 0) {  // k = M (Nyquist): a = Z[0], b = conj(Z[0])
        const float p = post_power(sm[0], sm[0], twN(Q, M, lq));
        out[M] = p;
        acc.add(p);
      }
    } else {
      for (int idx = (int)threadIdx.x; idx < H * M2; idx += NT) {
        const int p = idx % H, k2 = idx / H;
        if (p >= h) continue;
        const uint32_t k = kb + (uint32_t)p + (uint32_t)M1 * (uint32_t)k2;
        float pk, pm;
        post_power_pair(sm[p * P + p2_slot(k2)], sm[(H + p) * P + p2_slot(M2 - 1 - k2)],
                        twN(Q, k, lq), pk, pm);
        out[k] = pk;
        out[M - k] = pm;
        acc.add(pk);
        acc.add(pm);
      }
    }
  }
  block_sum_store<NT>(acc, psum_out);
}

// Pass 2: one CTA per row group of every trial.
template <int M1, int M2>
__global__ void __launch_bounds__(threads_for(M2, cols_for(M2)), 2)
    k_fft_pass2(const float2 *__restrict__ work, const float2 *__restrict__ Q, int lq,
                uint32_t N, float *__restrict__ power, uint64_t ldp, double *__restrict__ psum,
                uint32_t ngroups, uint32_t ahead) {
  constexpr int C = cols_for(M2), NT = threads_for(M2, C), H = C / 2;
  constexpr uint32_t M = (uint32_t)M1 * M2;
  extern __shared__ float2 dyn[];
  float2 *Wl = dyn;       // M2 entries
  float2 *W1 = Wl + M2;   // 256 entries
  float2 *sm = W1 + 256;  // C rows of p2_pitch
  const uint64_t trial = blockIdx.y;
  const uint32_t g = blockIdx.x;
  {
    // Prefetch into L2 the rows of the CTA one resident wave ahead (linear
    // index + ahead): CTAs start roughly in index order, so it runs soon.
    const uint64_t lin = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x + ahead;
    if (ahead && lin < (uint64_t)gridDim.x * gridDim.y) {
      const uint32_t gn = (uint32_t)(lin % gridDim.x);
      const uint64_t tn = lin / gridDim.x;
      const uint32_t kbn = gn == 0 ? 0u : 1 + (gn - 1) * (uint32_t)H;
      const int hn = gn == 0 ? 1 : (int)min((uint32_t)H, (uint32_t)(M1 / 2 - kbn));
      constexpr int LPR = M2 * 8 / 128;  // 128-byte lines per row
      for (int t = threadIdx.x; t < 2 * hn * LPR; t += NT) {
        const int ci = t / LPR;
        const uint32_t k1 = gn == 0 ? (ci == 0 ? 0u : (uint32_t)(M1 / 2))
                                    : (ci < hn ? kbn + (uint32_t)ci
                                               : (uint32_t)M1 - (kbn + (uint32_t)(ci - hn)));
        const float2 *pr = work + tn * M + (uint64_t)k1 * M2 + (t % LPR) * 16;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(pr));
      }
    }
  }
  p2_group<M1, M2>(sm, Wl, W1, N, work + trial * (uint64_t)M, g, Q, lq, power + trial * ldp,
                   psum + trial * ngroups + g);
}

struct FftArgs {
  const float *series;
  uint64_t lds, len;
  const float *means;
  const float2 *Q;
  int lq;
  uint32_t N;
  const float2 *tw1;
  uint64_t ntrials;
  float2 *work;
  float *power;
  uint64_t ldp;
  double *psum;
  cudaStream_t st;
};

// Largest pass-1 dynamic shared memory that keeps two CTAs per SM with the
// staged rows (GB300: 228 KB per SM, 1 KB reserved per CTA, static arrays).
size_t g_pass1_stage_max = 110 * 1024;

// SM count of the current device (cached per device).
int sm_count(int &n) {
  static thread_local int dev_cached = -1, n_cached = 0;
  int dev = 0;
  PSR_CUDA(cudaGetDevice(&dev));
  if (dev != dev_cached) {
    PSR_CUDA(cudaDeviceGetAttribute(&n_cached, cudaDevAttrMultiProcessorCount, dev));
    dev_cached = dev;
  }
  n = n_cached;
  return PSR_OK;
}

template <int M>
int run_small(const FftArgs &a) {
  const size_t smem = (size_t)(M + lay_slots<M, 1>()) * sizeof(float2);
  PSR_CUDA(cudaFuncSetAttribute(k_fft_small<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem));
  k_fft_small<M><<<(unsigned)a.ntrials, threads_for(M, 1), smem, a.st>>>(
      a.series, a.lds, a.len, a.means, a.Q, a.lq, a.N, a.power, a.ldp, a.psum);
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

template <int M1, int M2>
int run_four_step(const FftArgs &a) {
  {
    constexpr int C = cols_for(M1);
    const size_t smem = (size_t)(M1 + lay_slots<M1, C>()) * sizeof(float2);
    // staged rows: ceil(nz / M2) <= M1 / 2 rows of C complex values (plus the
    // slot that aligns them to 16 bytes)
    const uint64_t rows = ((a.len + 1) / 2 + M2 - 1) / M2;
    const size_t smem_st = smem + (rows * C + 1) * sizeof(float2);
    int nsm = 0;
    PSR_TRY(sm_count(nsm));
    const uint32_t ngroups = (uint32_t)(M2 / C) * (uint32_t)a.ntrials;
    const uint32_t grid = std::min<uint32_t>(ngroups, 2u * (uint32_t)nsm);
    if (C % 2 == 0 && smem_st <= g_pass1_stage_max) {
      PSR_CUDA(cudaFuncSetAttribute(k_fft_pass1<M1, M2, true>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_st));
      k_fft_pass1<M1, M2, true><<<grid, threads_for(M1, C), smem_st, a.st>>>(
          a.series, a.lds, a.len, a.means, a.Q, a.lq, a.N, a.tw1, a.work, ngroups);
    } else {
      PSR_CUDA(cudaFuncSetAttribute(k_fft_pass1<M1, M2, false>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k_fft_pass1<M1, M2, false><<<grid, threads_for(M1, C), smem, a.st>>>(
          a.series, a.lds, a.len, a.means, a.Q, a.lq, a.N, a.tw1, a.work, ngroups);
    }
    PSR_CUDA(cudaGetLastError());
  }
  {
    constexpr int C = cols_for(M2);
    const size_t smem = (size_t)(M2 + 256 + C * p2_pitch<M2>()) * sizeof(float2);
    PSR_CUDA(cudaFuncSetAttribute(k_fft_pass2<M1, M2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
    const uint32_t ng = 1 + ((uint32_t)M1 / 2 - 1 + C / 2 - 1) / (C / 2);
    dim3 grid(ng, (unsigned)a.ntrials);
    int nsm2 = 0;
    PSR_TRY(sm_count(nsm2));
    k_fft_pass2<M1, M2><<<grid, threads_for(M2, C), smem, a.st>>>(
        a.work, a.Q, a.lq, a.N, a.power, a.ldp, a.psum, ng, 2u * (uint32_t)nsm2);
    PSR_CUDA(cudaGetLastError());
  }
  return PSR_OK;
}

// The quarter table, entries r <= N/8 and their mirrors N/4 - r (components
// swapped).  The angles of every N are those of the largest (2 pi r / N with
// N a power of two), and for each of them the device's f64 sincos rounds to
// the same f32 values as the host's, which the oracle uses (compared
// exhaustively).  On the host the tables of a 2^23-point transform took about
// 28 ms.
__global__ void __launch_bounds__(256) k_fft_quarter(uint64_t N, float2 *__restrict__ Q) {
  const uint64_t r = (uint64_t)blockIdx.x * 256 + threadIdx.x, n4 = N / 4, n8 = N / 8;
  if (r > n8) return;
  double sn, cs;
  sincos(6.283185307179586 * (double)r / (double)N, &sn, &cs);
  const float2 v = make_float2((float)cs, (float)sn);
  Q[r] = v;
  if (n4 - r > n8) Q[n4 - r] = make_float2(v.y, v.x);
}

// From QS_MIN points on by angle sums: 2 pi j / 2^25, j = 2^11 h + l <= 2^22, from
// 2049 + 2048 angles' f64 sines and cosines, which are a tenth of the f64
// work (FP64, 1/64 of the f32 rate, bounds the kernel).  Every N's angles are
// among these, and for each of them the product rounds to the f32 values of the
// direct evaluation (compared exhaustively).  Measured on a GB300, N = 2^23: 73 us
// direct, 3 + 14 now.
constexpr int QS_LO = 11, QS_TOP = 25;
constexpr uint64_t QS_MIN = 1ull << 17;
constexpr int QS_H = (1 << (QS_TOP - 3 - QS_LO)) + 1, QS_L = 1 << QS_LO;
__global__ void __launch_bounds__(256) k_fft_angles(double2 *__restrict__ T) {
  const int i = (int)(blockIdx.x * 256 + threadIdx.x);
  if (i >= QS_H + QS_L) return;
  const double j = i < QS_H ? (double)((uint64_t)i << QS_LO) : (double)(i - QS_H);
  double sn, cs;
  sincos(6.283185307179586 * j / (double)(1ull << QS_TOP), &sn, &cs);
  T[i] = make_double2(cs, sn);
}
__global__ void __launch_bounds__(256)
    k_fft_quarter_split(uint64_t N, int up, const double2 *__restrict__ T,
                        float2 *__restrict__ Q) {
  const uint64_t r = (uint64_t)blockIdx.x * 256 + threadIdx.x, n4 = N / 4, n8 = N / 8;
  if (r > n8) return;
  const uint32_t j = (uint32_t)(r << up);
  const double2 a = T[j >> QS_LO], b = T[QS_H + (j & (QS_L - 1))];
  const double cs = __fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y));
  const double sn = __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y));
  const float2 v = make_float2((float)cs, (float)sn);
  Q[r] = v;
  if (n4 - r > n8) Q[n4 - r] = make_float2(v.y, v.x);
}

// Tw1[k1*M2 + n2] = W_N^(2*n2*k1) = W_M^(n2*k1), by the device lookup.
__global__ void __launch_bounds__(256)
    k_fft_tw1(const float2 *__restrict__ Q, int lq, int lm2, uint64_t M,
              float2 *__restrict__ tw1) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  const uint64_t k1 = i >> lm2, n2 = i & ((1ull << lm2) - 1);
  if (i < M) tw1[i] = twN(Q, (uint32_t)(2 * n2 * k1), lq);
}

}  // namespace

uint64_t FftPlan::pass2_ctas() const {
  if (m <= 12) return 1;
  const uint32_t C = (uint32_t)(M2 >= 8192 ? 1 : std::min<uint64_t>(16, 8192 / M2));
  const uint32_t H = C / 2;
  return 1 + ((uint32_t)M1 / 2 - 1 + H - 1) / H;
}

int FftPlan::init(uint64_t series_len, cudaStream_t st) {
  if (series_len < 2) {
    set_error("periodicity: series of at least two samples required");
    return PSR_EINVAL;
  }
  uint64_t p = 1;
  while (p < series_len) p <<= 1;
  N = 2 * p;
  M = p;
  if (M > (1ull << 24)) {
    set_error("periodicity: FFT size above 2^25 is not supported");
    return PSR_EINVAL;
  }
  len = series_len;
  m = 0;
  while ((1ull << m) < M) ++m;
  M1 = 1ull << ((m + 1) / 2);
  M2 = 1ull << (m / 2);
  int lq = 0;
  while ((1ull << lq) < N / 4) ++lq;
  PSR_TRY(Q.ensure((N / 4 + 1) * sizeof(float2)));
  if (m > 12) PSR_TRY(tw1.ensure(M * sizeof(float2)));
  const unsigned qctas = (unsigned)((N / 8 + 1 + 255) / 256);
  if (N >= QS_MIN) {
    // (the angles lie in tw1's memory, 512 KB or more, until its own kernel)
    double2 *T = tw1.as<double2>();
    static_assert(QS_MIN / 2 * sizeof(float2) >= (QS_H + QS_L) * sizeof(double2), "room");
    k_fft_angles<<<(QS_H + QS_L + 255) / 256, 256, 0, st>>>(T);
    k_fft_quarter_split<<<qctas, 256, 0, st>>>(N, QS_TOP - (lq + 2), T, Q.as<float2>());
  } else {
    k_fft_quarter<<<qctas, 256, 0, st>>>(N, Q.as<float2>());
  }
  if (m > 12) {
    k_fft_tw1<<<(unsigned)(M / 256), 256, 0, st>>>(Q.as<float2>(), lq, ilog2((int)M2), M,
                                                   tw1.as<float2>());
  }
  PSR_CUDA(cudaGetLastError());
  return PSR_OK;
}

int launch_raw_power_ex(const FftPlan &p, const float *d_series, uint64_t lds,
                        const float *d_means, uint64_t ntrials, float2 *d_work, float *d_power,
                        uint64_t ldp, double *d_psum, cudaStream_t st) {
  int lq = 0;
  while ((1ull << lq) < p.N / 4) ++lq;
  FftArgs a{d_series, lds,          p.len,   d_means, p.Q.as<float2>(), lq, (uint32_t)p.N,
            p.tw1.as<float2>(), ntrials, d_work, d_power, ldp, d_psum, st};
  switch (p.m) {
    case 1: return run_small<2>(a);
    case 2: return run_small<4>(a);
    case 3: return run_small<8>(a);
    case 4: return run_small<16>(a);
    case 5: return run_small<32>(a);
    case 6: return run_small<64>(a);
    case 7: return run_small<128>(a);
    case 8: return run_small<256>(a);
    case 9: return run_small<512>(a);
    case 10: return run_small<1024>(a);
    case 11: return run_small<2048>(a);
    case 12: return run_small<4096>(a);
    case 13: return run_four_step<128, 64>(a);
    case 14: return run_four_step<128, 128>(a);
    case 15: return run_four_step<256, 128>(a);
    case 16: return run_four_step<256, 256>(a);
    case 17: return run_four_step<512, 256>(a);
    case 18: return run_four_step<512, 512>(a);
    case 19: return run_four_step<1024, 512>(a);
    case 20: return run_four_step<1024, 1024>(a);
    case 21: return run_four_step<2048, 1024>(a);
    case 22: return run_four_step<2048, 2048>(a);
    case 23: return run_four_step<4096, 2048>(a);
    case 24: return run_four_step<4096, 4096>(a);
    default:
      set_error("periodicity: unsupported FFT size");
      return PSR_EINVAL;
  }
}

int launch_raw_power_tables(uint64_t len, uint64_t N, const float2 *d_Q, const float2 *d_tw1,
                            const float *d_series, uint64_t lds, const float *d_means,
                            uint64_t ntrials, float2 *d_work, float *d_power, uint64_t ldp,
                            double *d_psum, cudaStream_t st) {
  int lq = 0;
  while ((1ull << lq) < N / 4) ++lq;
  int m = 0;
  while ((1ull << m) < N / 2) ++m;
  FftArgs a{d_series, lds, len, d_means, d_Q, lq, (uint32_t)N, d_tw1, ntrials, d_work, d_power,
            ldp, d_psum, st};
  switch (m) {
    case 1: return run_small<2>(a);
    case 2: return run_small<4>(a);
    case 3: return run_small<8>(a);
    case 4: return run_small<16>(a);
    case 5: return run_small<32>(a);
    case 6: return run_small<64>(a);
    case 7: return run_small<128>(a);
    case 8: return run_small<256>(a);
    case 9: return run_small<512>(a);
    case 10: return run_small<1024>(a);
    case 11: return run_small<2048>(a);
    case 12: return run_small<4096>(a);
    case 13: return run_four_step<128, 64>(a);
    case 14: return run_four_step<128, 128>(a);
    case 15: return run_four_step<256, 128>(a);
    case 16: return run_four_step<256, 256>(a);
    case 17: return run_four_step<512, 256>(a);
    case 18: return run_four_step<512, 512>(a);
    case 19: return run_four_step<1024, 512>(a);
    case 20: return run_four_step<1024, 1024>(a);
    default:
      set_error("periodicity: unsupported FFT size");
      return PSR_EINVAL;
  }
}

}  // namespace psr
