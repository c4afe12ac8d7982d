// K-d: per-partition normalisation of G2/IP/IF into g2 and its standard error.
//
// Replaces Corr::normalizeG2s (src/xpcs/corr.cpp:927-1091).  BuildQMap's
// q -> sbin -> pixel mapping is flattened into entries (one per (q, sbin): q
// ascending, sbin ascending, pixels in raster order) and every entry's pixel
// range is cut into chunks of at most NCH pixels.
//
// float64 result (the reported one):
//   k_norm_part    one warp per (chunk, NT delays) reads G2/IP/IF of the
//                  chunk's pixels once and produces, per delay: sum G2, sum
//                  IP, sum IF, sum (x - s) and sum (x - s)^2 with x = G2 / (IP
//                  IF), NaN -> 0 and still counted (quirk Q8), and s the mean
//                  of the chunk's first 32 ratios, so that the variance loses
//                  nothing to cancellation and one pass suffices.
//                  Per-element arithmetic is double-word ("float-float") on
//                  the FP32 pipes -- TwoSum, FMA-based TwoProd, the quotient
//                  of a float by a double-word, and Sum2 compensated sums of
//                  Ogita, Rump & Oishi (2005) for the per-lane totals --
//                  because GB300's FP64 rate is a small fraction of its FP32
//                  rate; the sums over a warp use the double-word addition of
//                  Joldes, Muller & Popescu (ACM TOMS 2017), and everything
//                  after is FP64.
//   k_norm_finish  one warp per (q, tau): entry ratio (G2/n)/((IP/n)(IF/n))
//                  (:966-1013), g2 = mean of the non-NaN ratios (:1018-1040);
//                  the ring's mean from the chunks' sums and its M2 as the sum
//                  of every chunk's own and of n (chunk mean - mean)^2;
//                  stderr = sqrt(1/n) sqrt(M2/n) (:1043-1087).
// float32 result (optional, bit-identical to the reference's float output):
//   k_f32_transpose / k_q_f32 / k_entry_f32 / k_q_mean_f32 replay the reference's sequential
//   float operations in its order, including the running-mean/M2 update of
//   every pixel.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "overlap.cuh"
#include "xpcs_internal.h"

namespace xg {
namespace {

constexpr int NT = 4;            // delays a warp takes together
constexpr int NW = 4;            // warps per block
constexpr int NPART = 6;         // doubles per (chunk, delay)
constexpr int NCH_MIN = 128, NCH_MAX = 1024;  // pixels per chunk

// ------------------------------------------------ double-word arithmetic

struct dw {
  float h, l;
};

__device__ __forceinline__ dw two_sum(float a, float b) {
  float s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}
__device__ __forceinline__ dw fast_two_sum(float a, float b) {  // |a| >= |b|
  float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ dw two_prod(float a, float b) {
  float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}
// double-word + double-word (AccurateDWPlusDW)
__device__ __forceinline__ dw dw_add(dw x, dw y) {
  dw s = two_sum(x.h, y.h), t = two_sum(x.l, y.l);
  dw v = fast_two_sum(s.h, __fadd_rn(s.l, t.h));
  return fast_two_sum(v.h, __fadd_rn(t.l, v.l));
}
// float / double-word: a quotient from the reciprocal of the high word, then
// the quotient of the FMA remainder a - q (bh + bl) as the low word
// (relative error a few 2^-48)
__device__ __forceinline__ dw f_div_dw(float a, dw b) {
  if (a == 0.f) return {0.f, 0.f};  // 0 / b is 0 or NaN, and NaN counts as 0
  const float rb = __frcp_rn(b.h);
  float q = __fmul_rn(a, rb);
  if (!isfinite(q) || q == 0.f) return {__fdiv_rn(a, b.h), 0.f};
  float r = __fmaf_rn(-q, b.h, a);
  r = __fmaf_rn(-q, b.l, r);
  return fast_two_sum(q, __fmul_rn(r, rb));
}
// Sum2 (Ogita, Rump & Oishi, SIAM J. Sci. Comput. 26(6), 2005): a running
// float sum and, beside it, the float sum of every addition's exact rounding
// error; as accurate as summing in twice the precision, at one TwoSum and one
// addition per term.
struct sum2 {
  float s, c;
};
__device__ __forceinline__ void s2_add(sum2 &a, float x) {
  const dw t = two_sum(a.s, x);
  a.s = t.h;
  a.c = __fadd_rn(a.c, t.l);
}
// a double-word term: its low word joins the error sum
__device__ __forceinline__ void s2_add(sum2 &a, dw x) {
  s2_add(a, x.h);
  a.c = __fadd_rn(a.c, x.l);
}
__device__ __forceinline__ dw s2_value(const sum2 &a) { return two_sum(a.s, a.c); }
__device__ __forceinline__ double to_double(dw x) { return (double)x.h + (double)x.l; }

__device__ __forceinline__ float rcp_approx(float b) {  // within 1 ulp
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}

// x = g / (a b) as a double-word, NaN -> 0.  The quotient of the approximate
// reciprocal is corrected by two FMA residuals (relative error a few 2^-48);
// quotients whose residuals could underflow, and non-finite ones, take the
// general form.
__device__ __forceinline__ dw ratio_dw(float g, float a, float b) {
  const dw p = two_prod(a, b);
  const float rb = rcp_approx(p.h);
  const float q = __fmul_rn(g, rb);
  const float r = __fmaf_rn(-q, p.l, __fmaf_rn(-q, p.h, g));
  float ql = __fmul_rn(r, rb);
  ql = __fmaf_rn(__fmaf_rn(-ql, p.h, r), rb, ql);
  dw x = {q, ql};
  const float aq = fabsf(q), ag = fabsf(g), ap = fabsf(p.h);
  if (!(aq > 0x1p-60f && aq < 0x1p60f && ag > 0x1p-60f && ap > 0x1p-60f && ap < 0x1p60f)) {
    x = g == 0.f ? dw{0.f, 0.f} : f_div_dw(g, p);
    if (isnan(x.h) || isnan(x.l)) x = {0.f, 0.f};
  }
  return x;
}

// part layout: [chunk][tau][NPART] = sum G2, sum IP, sum IF, sum (x - s),
// sum (x - s)^2, s.
// Bound by instruction issue, about 120 instructions per element: issue active
// 59 % of the time at 512 x 512 x 10,000 frames, 74 % at 1,024 x 1,024.  Against a block per (chunk of 4,096 pixels, delay) with the ratios
// kept in shared memory for a second pass (168 instructions per element, a
// quarter of them in the block's reductions): 1,024 x 1,024 pixels, 88 delays
// 359 us instead of 602; 512 x 512, 34 delays 50 instead of 73.  Four delays
// together share the pixel list and let one transposing reduction over the
// warp sum all 20 values (21 double-word additions instead of 100).  The
// largest relative error of stderr against FP64 over seven series was 1.9e-14
// (3.5e-14 before), its rms 0.6 to 0.8 of what it was.
__global__ void __launch_bounds__(NW * 32)
k_norm_part(int D, int P, int NC, const int32_t *__restrict__ ch_k0,
            const int32_t *__restrict__ ch_k1, const int32_t *__restrict__ pix,
            const float *__restrict__ G2, const float *__restrict__ IP,
            const float *__restrict__ IF, double *__restrict__ part) {
  overlap_after();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * NW + (threadIdx.x >> 5), t0 = blockIdx.y * NT;
  if (c >= NC) return;
  const int k0 = ch_k0[c], k1 = ch_k1[c];
  // the block's rows of the arrays: delays past the last one repeat it, unused
  const float *rg[NT], *ra[NT], *rb[NT];
#pragma unroll
  for (int j = 0; j < NT; j++) {
    const size_t o = (size_t)min(t0 + j, D - 1) * P;
    rg[j] = G2 + o;
    ra[j] = IP + o;
    rb[j] = IF + o;
  }
  sum2 sg[NT], si[NT], sf[NT], sd[NT], sq[NT];
  float s[NT];
#pragma unroll
  for (int j = 0; j < NT; j++) sg[j] = si[j] = sf[j] = sd[j] = sq[j] = {0.f, 0.f};
  // the next 32 pixels' values are in flight while these are summed, their
  // pixel indices one step earlier
  float gn[NT], an[NT], bn[NT];
  const auto load = [&](int p) {
#pragma unroll
    for (int j = 0; j < NT; j++) {
      gn[j] = p >= 0 ? rg[j][(uint32_t)p] : 0.f;
      an[j] = p >= 0 ? ra[j][(uint32_t)p] : 0.f;
      bn[j] = p >= 0 ? rb[j][(uint32_t)p] : 0.f;
    }
  };
  load(k0 + lane < k1 ? pix[k0 + lane] : -1);
  int pn = k0 + 32 + lane < k1 ? pix[k0 + 32 + lane] : -1;
  for (int k = k0; k < k1; k += 32) {
    const bool in = k + lane < k1;
    float g[NT], a[NT], b[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
      g[j] = gn[j];
      a[j] = an[j];
      b[j] = bn[j];
    }
    load(pn);
    pn = k + 64 + lane < k1 ? pix[k + 64 + lane] : -1;
    dw x[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) x[j] = ratio_dw(g[j], a[j], b[j]);
    if (k == k0) {  // the shift: the mean of the first ratios
      const float n = (float)min(32, k1 - k0);
#pragma unroll
      for (int j = 0; j < NT; j++) {
        float m = x[j].h;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) m = __fadd_rn(m, __shfl_xor_sync(FULL, m, w));
        s[j] = __fdiv_rn(m, n);
      }
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
      s2_add(sg[j], g[j]);
      s2_add(si[j], a[j]);
      s2_add(sf[j], b[j]);
      if (in) {
        const dw d0 = two_sum(x[j].h, -s[j]);
        const float dl = __fadd_rn(d0.l, x[j].l);
        s2_add(sd[j], dw{d0.h, dl});
        const dw q = two_prod(d0.h, d0.h);
        s2_add(sq[j], dw{q.h, __fmaf_rn(__fmul_rn(2.f, d0.h), dl, __fmaf_rn(dl, dl, q.l))});
      }
    }
  }
  // sums over the warp: at each step a lane keeps one half of its values and
  // hands the other to its partner, so that a lane ends with one value
  constexpr int NV = 5 * NT;
  static_assert(NV == 20, "the steps below halve 20 values");
  dw v[NV + 1];
#pragma unroll
  for (int j = 0; j < NT; j++) {
    v[5 * j] = s2_value(sg[j]);
    v[5 * j + 1] = s2_value(si[j]);
    v[5 * j + 2] = s2_value(sf[j]);
    v[5 * j + 3] = s2_value(sd[j]);
    v[5 * j + 4] = s2_value(sq[j]);
  }
  const auto halve = [&](auto cnt, int w) {
    constexpr int n = decltype(cnt)::value, h = (n + 1) / 2;
    const bool up = lane & w;
    if (n & 1) v[n] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < h; i++) {
      const dw keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = dw_add(keep, dw{__shfl_xor_sync(FULL, send.h, w), __shfl_xor_sync(FULL, send.l, w)});
    }
  };
  halve(std::integral_constant<int, 20>{}, 16);
  halve(std::integral_constant<int, 10>{}, 8);
  halve(std::integral_constant<int, 5>{}, 4);
  halve(std::integral_constant<int, 3>{}, 2);
  halve(std::integral_constant<int, 2>{}, 1);
  // the value this lane ended with: 20 -> 10 + 10 -> 5 + 5 -> 3 + 2 -> 2 + 1
  // (2 + 0) -> 1 + 1
  const int c4 = lane & 4 ? 2 : 3, c2 = lane & 2 ? c4 - 2 : 2;
  const int id = (lane & 16 ? 10 : 0) + (lane & 8 ? 5 : 0) + (lane & 4 ? 3 : 0) +
                 (lane & 2 ? 2 : 0) + (lane & 1);
  const int t = t0 + id / 5;
  if ((lane & 1) < c2 && t < D)
    part[((size_t)c * D + t) * NPART + id % 5] = to_double(v[0]);
#pragma unroll
  for (int j = 0; j < NT; j++)
    if (lane == j && t0 + j < D) part[((size_t)c * D + t0 + j) * NPART + 5] = (double)s[j];
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) x += __shfl_xor_sync(0xffffffffu, x, w);
  return x;
}

// Five sums over the warp, the same in every lane: 8 FP64 additions by
// halving the values as above (5 -> 3 + 2 -> 2 + 1 -> 1 + 1) instead of 25.
__device__ __forceinline__ void warp_sum5(double (&v)[5]) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double a[3], b[2];
  const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double hi = i < 2 ? v[i + 3] : 0.0;
    a[i] = (u16 ? hi : v[i]) + __shfl_xor_sync(FULL, u16 ? v[i] : hi, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const double hi = i < 1 ? a[2] : 0.0;
    b[i] = (u8 ? hi : a[i]) + __shfl_xor_sync(FULL, u8 ? a[i] : hi, 8);
  }
  double c = (u4 ? b[1] : b[0]) + __shfl_xor_sync(FULL, u4 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(FULL, c, 2);
  c += __shfl_xor_sync(FULL, c, 1);
  v[0] = __shfl_sync(FULL, c, 0);
  v[1] = __shfl_sync(FULL, c, 4);
  v[2] = __shfl_sync(FULL, c, 8);
  v[3] = __shfl_sync(FULL, c, 16);
  v[4] = __shfl_sync(FULL, c, 20);
}

// sum (x - mean)^2 over the pixels [k0, k1) in a pass of its own, in FP64, for
// rings whose chunk sums cancel: nothing is lost however close the ratios lie.
__device__ double deviations(int k0, int k1, double mean, const int32_t *__restrict__ pix,
                             const float *__restrict__ g, const float *__restrict__ a,
                             const float *__restrict__ b) {
  double M2 = 0.0;
  for (int k = k0 + (threadIdx.x & 31); k < k1; k += 32) {
    const int32_t p = pix[k];
    const double d = to_double(ratio_dw(g[p], a[p], b[p])) - mean;
    M2 = fma(d, d, M2);
  }
  return warp_sum(M2);
}

// One warp per (q, tau), lanes over the ring's chunks.  Bound by FP64 issue
// (a division is some 25 instructions at 1/64 of the FP32 rate), so the
// formulas keep the divisions to one per entry and three per ring.  One
// thread merging the chunks in turn took 62 us at 18 rings x 88 delays and 40
// at 9 x 34; 19 and 14 now.
// A ring whose spread is small beside its shifts' distance from the mean (one
// pixel, equal ratios, dead pixels first) goes over its pixels again: where M2 is
// less than a 16th of sum (x - s)^2, their rounding would show in it, and could
// leave it negative.
__global__ void k_norm_finish(int NQ, int D, const int32_t *__restrict__ qep,
                              const int32_t *__restrict__ qrow,
                              const int32_t *__restrict__ e_chunk_ptr,
                              const int32_t *__restrict__ ch_k0, const int32_t *__restrict__ ch_k1,
                              const double *__restrict__ part, int P,
                              const int32_t *__restrict__ pix, const float *__restrict__ G2,
                              const float *__restrict__ IP, const float *__restrict__ IF,
                              double *__restrict__ g2, double *__restrict__ se) {
  overlap_after();
  const int lane = threadIdx.x & 31;
  const int idx = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (idx >= NQ * D) return;
  const int qi = idx / D, t = idx - qi * D;
  double gacc = 0.0, n = 0.0, sx = 0.0;
  int gcnt = 0;
  for (int e = qep[qi]; e < qep[qi + 1]; e++) {
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // sum G2, IP, IF, x; pixels
    for (int c = e_chunk_ptr[e] + lane; c < e_chunk_ptr[e + 1]; c += 32) {
      const double *q = part + ((size_t)c * D + t) * NPART;
      const double nc = (double)(ch_k1[c] - ch_k0[c]);
      v[0] += q[0];
      v[1] += q[1];
      v[2] += q[2];
      v[3] += fma(nc, q[5], q[3]);
      v[4] += nc;
    }
    warp_sum5(v);
    n += v[4];
    sx += v[3];
    const double r = v[0] * v[4] / (v[1] * v[2]);  // (G2/n) / ((IP/n) (IF/n))
    if (!isnan(r)) {
      gacc += r;
      gcnt++;
    }
  }
  // sum (x - mean)^2 = sum (x - s)^2 + 2 (s - mean) sum (x - s) + n (s - mean)^2
  const double mean = sx / n;
  const int c0 = e_chunk_ptr[qep[qi]], c1 = e_chunk_ptr[qep[qi + 1]];
  double about = 0.0, shift = 0.0;  // sum (x - s)^2, and the rest
  for (int c = c0 + lane; c < c1; c += 32) {
    const double *q = part + ((size_t)c * D + t) * NPART;
    const double nc = (double)(ch_k1[c] - ch_k0[c]), d = q[5] - mean;
    about += q[4];
    shift = fma(d, fma(nc, d, 2.0 * q[3]), shift);
  }
  {  // both over the warp, a half-warp each, in as many FP64 additions as one takes
    const bool up = lane & 16;
    double v = (up ? shift : about) + __shfl_xor_sync(0xffffffffu, up ? about : shift, 16);
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) v += __shfl_xor_sync(0xffffffffu, v, w);
    about = __shfl_sync(0xffffffffu, v, 0);
    shift = __shfl_sync(0xffffffffu, v, 16);
  }
  double M2 = about + shift;
  if (M2 < 0.0625 * about) {  // (not NaN, and not a ring of zeros)
    const size_t o = (size_t)t * P;
    M2 = deviations(ch_k0[c0], ch_k1[c1 - 1], mean, pix, G2 + o, IP + o, IF + o);
  }
  if (lane == 0) {
    const int row = qrow[qi];
    g2[(size_t)t * NQ + row] = gacc / (double)gcnt;
    se[(size_t)t * NQ + row] = sqrt(M2) / n;  // sqrt(1/n) sqrt(M2/n)
  }
}

// ------------------------------------------------ float32, reference order
//
// Every float sum below runs in the reference's order; what changes is where
// its operands come from.  k_f32_transpose writes G2, IP, IF and the per-pixel
// ratio x = G2 / (IP IF) (NaN -> 0) in q-ordered, pixel-major layout
// [mapped pixel][tau], so the sequential sums of neighbouring taus (adjacent
// threads) read adjacent words.  The running mean's division by the sample
// count uses the correctly rounded reciprocal of the count (__frcp_rn) and
// one FMA residual correction (Markstein; Muller et al., Handbook of
// Floating-Point Arithmetic, ch. 4), which gives the IEEE quotient for every
// float numerator and every integer count up to 2^20 (checked exhaustively
// against __fdiv_rn on the GPU: every significand, every count); larger
// counts, zeros and non-finite numerators use __fdiv_rn.

constexpr int TR_K = 32, TR_T = 32;  // transpose tile: mapped pixels x taus

__global__ void __launch_bounds__(256)
k_f32_transpose(int NK, int D, int Dp, int P, const int32_t *__restrict__ pix,
                const float *__restrict__ G2, const float *__restrict__ IP,
                const float *__restrict__ IF, float *__restrict__ Tg, float *__restrict__ Ti,
                float *__restrict__ Tf, float *__restrict__ X, int32_t *__restrict__ unsafe) {
  __shared__ float sg[TR_T][TR_K + 1], si[TR_T][TR_K + 1], sf[TR_T][TR_K + 1];
  const int k0 = blockIdx.x * TR_K, t0 = blockIdx.y * TR_T;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  // read: lanes over mapped pixels (pixels of a ring run in raster order)
  const int k = k0 + tx;
  const int p = k < NK ? pix[k] : 0;
  for (int r = ty; r < TR_T; r += 8) {
    const int t = t0 + r;
    if (k < NK && t < D) {
      const size_t o = (size_t)t * P + p;
      sg[r][tx] = G2[o];
      si[r][tx] = IP[o];
      sf[r][tx] = IF[o];
    }
  }
  __syncthreads();
  // write: lanes over taus
  const int t = t0 + tx;
  for (int r = ty; r < TR_K; r += 8) {
    const int kk = k0 + r;
    bool bad = false;
    if (kk < NK && t < D) {
      const float g = sg[tx][r], a = si[tx][r], b = sf[tx][r];
      const size_t o = (size_t)kk * Dp + t;
      Tg[o] = g;
      Ti[o] = a;
      Tf[o] = b;
      float x = __fdiv_rn(g, __fmul_rn(a, b));
      x = isnan(x) ? 0.f : x;
      X[o] = x;
      bad = !(x == 0.f || (x >= 0x1p-20f && x <= 0x1p20f));
    }
    // any ratio outside the range where the q-ring replay's running mean
    // needs no special case (k_q_f32)
    if (__any_sync(0xffffffffu, bad) && tx == 0) atomicOr(unsafe, 1);
  }
}

// a / n for the running mean: n is the (integer-valued) sample count and y
// = __frcp_rn(n) its correctly rounded reciprocal, which depends on the count
// only and so stays off the chain of dependent operations
__device__ __forceinline__ float div_count(float a, float n, int ni, float y) {
  if (ni > (1 << 20) || a == 0.f || !isfinite(a) || fabsf(a) < 1e-30f) return __fdiv_rn(a, n);
  const float q0 = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-q0, n, a), y, q0);
}

// The replay kernels below run one block per q ring (or per entry) and one
// thread per tau.  The rows [k][0..Dp) of the block's pixel range (Dp: the
// delays padded to a multiple of 4, so that every row range is a 16-byte
// aligned, contiguous span) are brought into shared memory in chunks of up to
// 256 rows by 1-D bulk copies (cp.async.bulk, one per array, issued by one
// thread and completing on an mbarrier), double-buffered: chunk c+1 is in
// flight while the threads step through chunk c, so each thread's sequential
// chain reads shared memory instead of waiting on global loads.
constexpr int FR_SMEM = 200 * 1024;  // shared memory budget of a replay block
constexpr int FR_ROWS = 256;         // most rows of a chunk
constexpr uint32_t FR_WAIT_LIMIT = 1u << 22;  // polls before a wait is given up

__device__ __forceinline__ uint32_t fr_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void fr_bar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(fr_u32(bar)));
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(fr_u32(bar + 1)));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Waits for the phase of the given parity; false after FR_WAIT_LIMIT polls.
__device__ __forceinline__ bool fr_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t a = fr_u32(bar);
  for (uint32_t it = 0; it < FR_WAIT_LIMIT; it++) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// One thread: rows [r0, r0 + nrow) of each row-major [k][Dp] array into
// dst[a], completing on bar.
__device__ __forceinline__ void fr_bulk(const float *const *src, float *const *dst, int narr,
                                        int64_t r0, int nrow, int Dp, uint64_t *bar) {
  const uint32_t bytes = (uint32_t)nrow * (uint32_t)Dp * 4u;
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fr_u32(bar)),
               "r"(bytes * (uint32_t)narr)
               : "memory");
  for (int a = 0; a < narr; a++)
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(fr_u32(dst[a])), "l"(src[a] + (size_t)r0 * Dp), "r"(bytes), "r"(fr_u32(bar))
        : "memory");
}

// The chunk loop shared by the replay kernels: `narr` arrays of the rows
// [k0, k0 + n) streamed through the two buffers of `buf` ([2][narr][ch][Dp]),
// `step(b, rows, row0)` called by every thread for each chunk in order (b:
// the chunk's buffer, row0: its first row in the range).  Returns false, after setting DEVERR_WAIT, if a copy's
// wait expired; the copies still in flight are then waited for (again with a
// limit) before the block leaves.
template <class Step>
__device__ __forceinline__ bool fr_stream(const float *const *src, int narr, int64_t k0, int n,
                                          int ch, int Dp, float *buf, uint64_t *bar,
                                          int32_t *err, Step step) {
  const int t = threadIdx.x, nch = (n + ch - 1) / ch;
  const size_t bw = (size_t)narr * ch * Dp;
  auto issue = [&](int c) {
    float *dst[3];
    for (int a = 0; a < narr; a++) dst[a] = buf + (size_t)(c & 1) * bw + (size_t)a * ch * Dp;
    fr_bulk(src, dst, narr, k0 + (int64_t)c * ch, min(ch, n - c * ch), Dp, &bar[c & 1]);
  };
  if (t == 0) fr_bar_init(bar);
  __syncthreads();
  if (t == 0) {
    if (nch > 0) issue(0);
    if (nch > 1) issue(1);
  }
  bool ok = true;
  int c = 0;
  for (; c < nch; c++) {
    ok = __syncthreads_and(fr_wait(&bar[c & 1], (uint32_t)(c >> 1) & 1u)) != 0;
    if (!ok) break;
    step(c & 1, min(ch, n - c * ch), c * ch);
    __syncthreads();  // every thread is done with the buffer before it is refilled
    if (t == 0 && c + 2 < nch) issue(c + 2);
  }
  if (!ok && t == 0) {
    atomicOr(err, DEVERR_WAIT);
    // the copies issued for chunks c and c + 1, if any, before the block goes
    for (int d = c; d < min(c + 2, nch); d++) fr_wait(&bar[d & 1], (uint32_t)(d >> 1) & 1u);
  }
  return ok;
}

// One block per entry, thread tau: the entry's sums of G2, IP, IF in pixel
// order, / pixels, ratio (corr.cpp:966-1013).
__global__ void k_entry_f32(int NE, int D, int Dp, int FR_CH, const int32_t *__restrict__ epp,
                            const float *__restrict__ Tg, const float *__restrict__ Ti,
                            const float *__restrict__ Tf, float *__restrict__ ratio,
                            int32_t *__restrict__ err) {
  overlap_begin();
  extern __shared__ __align__(16) float fr_buf[];  // [2][3][FR_CH][Dp], then 2 mbarriers
  uint64_t *bar = (uint64_t *)(fr_buf + (size_t)2 * 3 * FR_CH * Dp);
  const int e = blockIdx.x, t = threadIdx.x;
  const int k0 = epp[e], n = epp[e + 1] - k0;
  const float *src[3] = {Tg, Ti, Tf};
  float sg = 0.f, si = 0.f, sf = 0.f;
  const size_t aw = (size_t)FR_CH * Dp;
  const bool ok = fr_stream(src, 3, k0, n, FR_CH, Dp, fr_buf, bar, err, [&](int b, int rows, int) {
    if (t >= D) return;
    const float *bg = fr_buf + (size_t)b * 3 * aw, *bi = bg + aw, *bf = bg + 2 * aw;
#pragma unroll 4
    for (int r = 0; r < rows; r++) {
      sg = __fadd_rn(sg, bg[r * Dp + t]);
      si = __fadd_rn(si, bi[r * Dp + t]);
      sf = __fadd_rn(sf, bf[r * Dp + t]);
    }
  });
  if (ok && t < D) {
    const float cnt = (float)n;
    sg = __fdiv_rn(sg, cnt);
    si = __fdiv_rn(si, cnt);
    sf = __fdiv_rn(sf, cnt);
    ratio[(size_t)e * D + t] = __fdiv_rn(sg, __fmul_rn(si, sf));
  }
  overlap_end();
}

// g2 of a q bin and tau = mean of the non-NaN entry ratios (corr.cpp:1018-1040).
__global__ void k_q_mean_f32(int NQ, int D, const int32_t *__restrict__ qep,
                             const int32_t *__restrict__ qrow, const float *__restrict__ ratio,
                             float *__restrict__ g2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NQ * D) return;
  const int qi = i / D, t = i - qi * D;
  float acc = 0.f, cnt = 0.f;
  for (int e = qep[qi]; e < qep[qi + 1]; e++) {
    const float r = ratio[(size_t)e * D + t];
    acc = __fadd_rn(acc, isnan(r) ? 0.f : r);
    cnt = __fadd_rn(cnt, isnan(r) ? 0.f : 1.f);
  }
  g2[(size_t)t * NQ + qrow[qi]] = __fdiv_rn(acc, cnt);
}

// One block per q ring, thread tau: stderr from the running mean / M2 over the
// ring's pixels in order, NaN counted as 0 (corr.cpp:1043-1087).  Few blocks,
// each a long chain: the entries' kernel runs on the other SMs meanwhile (640 x
// 480 x 2,000 frames with the side statistics: 3.16 ms one after the other, 2.83).
__global__ void k_q_f32(int NQ, int D, int Dp, int FR_CH, const int32_t *__restrict__ qep,
                        const int32_t *__restrict__ qrow, const int32_t *__restrict__ epp,
                        const float *__restrict__ X, float *__restrict__ se,
                        const int32_t *__restrict__ unsafe, int32_t *__restrict__ err) {
  overlap_begin();
  extern __shared__ __align__(16) float fr_buf[];  // [2][FR_CH][Dp], then 2 mbarriers
  const bool all_safe = *unsafe == 0;
  uint64_t *bar = (uint64_t *)(fr_buf + (size_t)2 * FR_CH * Dp);
  const int qi = blockIdx.x, t = threadIdx.x;
  const int row = qrow[qi];
  // The reference's sample count (samples += 1.0f per pixel) is the exact
  // count below 2^24 and stays at 2^24 from there on.  Its correctly rounded
  // reciprocal depends on the count only: the block computes each chunk's
  // into a table, off the chain of dependent operations that each tau's
  // running mean is.
  __shared__ __align__(16) float rtab[FR_ROWS];
  float avg = 0.f, sd = 0.f;
  const int k0 = epp[qep[qi]], n = epp[qep[qi + 1]] - k0;
  const float *src[1] = {X};
  const bool ok = fr_stream(src, 1, k0, n, FR_CH, Dp, fr_buf, bar, err, [&](int b, int rows,
                                                                          int row0) {
    for (int r = t; r < rows; r += blockDim.x) rtab[r] = __frcp_rn((float)(row0 + r + 1));
    __syncthreads();
    if (t >= D) return;
    const float *bx = fr_buf + (size_t)b * FR_CH * Dp;
    // When every ratio of the series is 0 or in [2^-20, 2^20] (flagged by
    // k_f32_transpose), the running mean of non-negative values over at most
    // 2^20 counts stays 0 or about [2^-40, 2^20] (checked at each chunk):
    // every difference a is then 0 (which leaves the mean as it is however it
    // is divided) or finite and at least about 2^-64 in size (the spacing of
    // floats near 2^-41), far inside the range where the reciprocal-and-
    // residual quotient is the IEEE one; the quotient is never NaN, and the
    // chain runs without a branch.
    if (all_safe && row0 + rows <= (1 << 20) &&
        (avg == 0.f || (avg >= 0x1p-40f && avg <= 0x1p20f))) {
      const auto step = [&](float x, float y, float cnt) {
        const float a = __fsub_rn(x, avg);
        const float q0 = __fmul_rn(a, y);
        avg = __fadd_rn(avg, __fmaf_rn(__fmaf_rn(-q0, cnt, a), y, q0));
        sd = __fadd_rn(sd, __fmul_rn(a, __fsub_rn(x, avg)));
      };
      // 8 rows at a time, the next 8 rows' ratios and reciprocals loaded while
      // these are stepped through, so that the chain of 5 dependent operations
      // waits on nothing else: 2.1 instead of 2.6 ms on a ring of 114,811
      // pixels, 0.83 instead of 1.00 ms at 640 x 480
      const float c0 = (float)row0;
      float x[8], y[8], xn[8], yn[8];
      const auto load = [&](int r) {
#pragma unroll
        for (int u = 0; u < 8; u++) xn[u] = bx[(r + u) * Dp + t];
        const float4 a = *(const float4 *)(rtab + r), b = *(const float4 *)(rtab + r + 4);
        yn[0] = a.x, yn[1] = a.y, yn[2] = a.z, yn[3] = a.w;
        yn[4] = b.x, yn[5] = b.y, yn[6] = b.z, yn[7] = b.w;
      };
      const int full = rows & ~7;
      if (full) load(0);
#pragma unroll 2
      for (int r = 0; r < full; r += 8) {
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = xn[u], y[u] = yn[u];
        if (r + 8 < full) load(r + 8);
        const float c = __fadd_rn(c0, (float)r);  // counts below 2^24: exact
#pragma unroll
        for (int u = 0; u < 8; u++) step(x[u], y[u], __fadd_rn(c, (float)(u + 1)));
      }
      for (int r = full; r < rows; r++)
        step(bx[r * Dp + t], rtab[r], __fadd_rn(c0, (float)(r + 1)));
    } else if (row0 + rows <= (1 << 20)) {
#pragma unroll 4
      for (int r = 0; r < rows; r++) {
        const float x = bx[r * Dp + t];
        const float cnt = (float)(row0 + r + 1);
        const float a = __fsub_rn(x, avg);
        // a / cnt by the reciprocal and one FMA residual correction: the IEEE
        // quotient for counts up to 2^20 and 1e-30 <= |a| <= FLT_MAX; zero,
        // tiny, infinite and NaN operands take the division itself
        const float q0 = __fmul_rn(a, rtab[r]);
        float tmp00 = __fmaf_rn(__fmaf_rn(-q0, cnt, a), rtab[r], q0);
        if (!(fabsf(a) >= 1e-30f && fabsf(a) <= 3.40282347e38f)) tmp00 = __fdiv_rn(a, cnt);
        tmp00 = isnan(tmp00) ? 0.f : tmp00;
        avg = __fadd_rn(avg, tmp00);
        sd = __fadd_rn(sd, __fmul_rn(a, __fsub_rn(x, avg)));
      }
    } else {
      for (int r = 0; r < rows; r++) {
        const float x = bx[r * Dp + t];
        const int k = row0 + r + 1;
        const float cnt = (float)min(k, 1 << 24);
        const float a = __fsub_rn(x, avg);
        float tmp00 = k <= (1 << 20) ? div_count(a, cnt, k, rtab[r]) : __fdiv_rn(a, cnt);
        tmp00 = isnan(tmp00) ? 0.f : tmp00;
        avg = __fadd_rn(avg, tmp00);
        sd = __fadd_rn(sd, __fmul_rn(a, __fsub_rn(x, avg)));
      }
    }
  });
  if (ok && t < D) {
    const float samples = (float)min(n, 1 << 24);
    const float stdNorm = __fdiv_rn(sd, samples);
    const float inv = __fdiv_rn(1.f, samples);
    se[(size_t)t * NQ + row] = __fmul_rn(__fsqrt_rn(inv), __fsqrt_rn(stdNorm));
  }
}

}  // namespace

// Chunks of up to 1,024 pixels, smaller ones where those would leave fewer
// than 16 warps per SM (152 SMs) for the series' pixels and delays.
void build_norm_chunks(Series &s) {
  const QMap &q = s.qmap;
  const double units = (double)q.pix.size() * ((s.D + NT - 1) / NT);
  int nch = NCH_MAX;
  while (nch > NCH_MIN && units / nch < 152.0 * 16) nch /= 2;
  std::vector<int32_t> k0, k1, eptr(1, 0);
  for (int e = 0; e < q.nentries(); e++) {
    for (int a = q.entry_pix_ptr[e]; a < q.entry_pix_ptr[e + 1]; a += nch) {
      k0.push_back(a);
      k1.push_back(std::min(a + nch, q.entry_pix_ptr[e + 1]));
    }
    eptr.push_back((int32_t)k0.size());
  }
  s.n_chunks = (int32_t)k0.size();
  cudaStream_t st = s.stream;
  auto up = [&](DBuf<int32_t> &b, const std::vector<int32_t> &v) {
    b.reserve(v.size() ? v.size() : 1, st);
    if (!v.empty())
      XG_CUDA(cudaMemcpyAsync(b.p, v.data(), 4 * v.size(), cudaMemcpyHostToDevice, st));
  };
  up(s.n_ch_k0, k0);
  up(s.n_ch_k1, k1);
  up(s.n_e_chunk_ptr, eptr);
}

void run_normalize(Series &s, bool want64, bool want32) {
  cudaStream_t st = s.stream;
  const int D = s.D, P = s.P, NQ = s.qmap.nq(), NE = s.qmap.nentries();
  if (D == 0 || NQ == 0) return;
  if (want64) {
    s.n_g2.reserve((size_t)NQ * D, st);
    s.n_se.reserve((size_t)NQ * D, st);
    const int NC = s.n_chunks;
    s.n_part.reserve((size_t)(NC > 0 ? NC : 1) * D * NPART, st);
    if (NC > 0) {
      launch_overlapped(k_norm_part, dim3((NC + NW - 1) / NW, (D + NT - 1) / NT), NW * 32, 0, st,
                        D, P, NC, s.n_ch_k0.p, s.n_ch_k1.p, s.n_pix.p, s.G2.p, s.IP.p, s.IF.p,
                        s.n_part.p);
    }
    const int bs = 128;
    launch_overlapped(k_norm_finish, (unsigned)(((int64_t)NQ * D * 32 + bs - 1) / bs), bs, 0, st,
                      NQ, D, s.n_q_entry_ptr.p, s.n_q_row.p, s.n_e_chunk_ptr.p, s.n_ch_k0.p,
                      s.n_ch_k1.p, s.n_part.p, P, s.n_pix.p, s.G2.p, s.IP.p, s.IF.p, s.n_g2.p,
                      s.n_se.p);
  }
  if (want32) {
    const QMap &qm = s.qmap;
    const int NK = qm.entry_pix_ptr.empty() ? 0 : qm.entry_pix_ptr.back();
    s.n_ratio32.reserve((size_t)(NE > 0 ? NE : 1) * D, st);
    s.n_g2f.reserve((size_t)NQ * D, st);
    s.n_sef.reserve((size_t)NQ * D, st);
    // rows of the transposed arrays padded to a multiple of 4 delays: 16-byte
    // aligned row ranges for the replay kernels' bulk copies
    const int Dp = (D + 3) & ~3;
    const size_t nt = (size_t)(NK > 0 ? NK : 1) * Dp;
    s.n_tg.reserve(nt, st);
    s.n_ti.reserve(nt, st);
    s.n_tf.reserve(nt, st);
    s.n_tx.reserve(nt, st);
    s.n_unsafe.reserve(1, st);
    XG_CUDA(cudaMemsetAsync(s.n_unsafe.p, 0, sizeof(int32_t), st));
    if (NK > 0) {
      k_f32_transpose<<<dim3((NK + TR_K - 1) / TR_K, (D + TR_T - 1) / TR_T), 256, 0, st>>>(
          NK, D, Dp, P, s.n_pix.p, s.G2.p, s.IP.p, s.IF.p, s.n_tg.p, s.n_ti.p, s.n_tf.p,
          s.n_tx.p, s.n_unsafe.p);
      XG_CHECK_LAUNCH();
    }
    if (D > 1024) throw Error(XPCS_ERR_INVALID_ARGUMENT, "more than 1024 delays");
    const int bs = (D + 31) / 32 * 32;
    const int ch_e = std::max(1, std::min(FR_ROWS, (FR_SMEM - 64) / (24 * Dp)));
    const int ch_q = std::max(1, std::min(FR_ROWS, (FR_SMEM - 64) / (8 * Dp)));
    const size_t sm_e = sizeof(float) * 2 * 3 * (size_t)ch_e * Dp + 2 * sizeof(uint64_t);
    const size_t sm_q = sizeof(float) * 2 * (size_t)ch_q * Dp + 2 * sizeof(uint64_t);
    allow_smem(k_entry_f32);
    allow_smem(k_q_f32, sizeof(float) * FR_ROWS);
    k_q_f32<<<NQ, bs, sm_q, st>>>(NQ, D, Dp, ch_q, s.n_q_entry_ptr.p, s.n_q_row.p,
                                  s.n_entry_pix_ptr.p, s.n_tx.p, s.n_sef.p, s.n_unsafe.p,
                                  &s.stats.p->error);
    XG_CHECK_LAUNCH();
    if (NE > 0)
      launch_overlapped(k_entry_f32, NE, bs, sm_e, st, NE, D, Dp, ch_e, s.n_entry_pix_ptr.p,
                        s.n_tg.p, s.n_ti.p, s.n_tf.p, s.n_ratio32.p, &s.stats.p->error);
    k_q_mean_f32<<<(NQ * D + 127) / 128, 128, 0, st>>>(NQ, D, s.n_q_entry_ptr.p, s.n_q_row.p,
                                                       s.n_ratio32.p, s.n_g2f.p);
    XG_CHECK_LAUNCH();
  }
}

}  // namespace xg
