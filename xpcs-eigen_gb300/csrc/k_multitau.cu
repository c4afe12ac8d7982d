// K-c: per-pixel multi-tau G2 / IP / IF.
//
// Replaces Corr::multiTau2 (src/xpcs/corr.cpp:315-431).  For every pixel with
// events and every delay (level L, tau):
//   on a level change lastframe halves (odd -> -1 first) and the row is
//   compacted in place: index/2, equal neighbours merged by addition, indices
//   >= lastframe dropped, every live value halved (:349-390);
//   IP  = sum of v over events with t < lastframe - tau,
//   G2  = sum of v(t) * v(t + tau), the partner found by std::lower_bound over
//         the row buffer (:406),
//   IF  = sum of v over events with tau <= t < lastframe,
//   each divided by (lastframe - tau) (:420-424).
//
// Integer paths (values are integers, sum |v| < 4096): a level-L value is an
// integer numerator N over 2^L, every float partial sum of the reference is
// exact, so integer sums scaled by 2^-L (2^-2L for G2) followed by one IEEE
// division reproduce the reference bit for bit.
//   * IP and IF do not depend on the compaction: level L keeps exactly the
//     events with frame < lastframe << L, so IP(tau) = S(t_ip) and
//     IF(tau) = S(lastframe << L) - S(tau_frames), S(T) = sum of v over
//     original events with frame < T.  Two merge sweeps over the sorted row
//     and the (monotone) per-delay thresholds give all of them.
//   * G2 needs the compacted rows: per level the row is compacted in place
//     (the same buffer the reference keeps, stale tail included) and the
//     pairs whose bin distance lies in the level's delay window are summed.
//     In REFERENCE mode a pair counts only when lower_bound over the whole
//     buffer lands on the partner; that always holds while the buffer is
//     globally sorted, which is tracked per level from the junction between
//     the new prefix and the stale tail.
// k_mt_thread: one thread per pixel, rows packed (frame << 16 | int16 value)
//   in shared memory with a lane-interleaved layout (conflict-free), outputs
//   written straight to [D][P] (32 consecutive pixels per warp = coalesced).
//   Dense levels take their pairs by byte products over windows of the level's
//   bins in the thread's scratch words; levels of few bins whose values do not
//   fit bytes, or with more than 8 delays, find pairs from an occupancy bitmask
//   there; sparse levels check each source's next three entries without
//   branching.  Pixels of other classes are left to the kernels below.
// k_mt_warp:   one warp per pixel, rows packed in shared memory: rows of up
//   to 256 events (8 warps per block), up to 1024 (4 warps per block) and up
//   to 4096 (2 warps per block).
// k_mt_float:  one thread per pixel replaying the reference's float
//   operations in its order (no fused multiply-add) on a scratch copy.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "mt_replay.cuh"
#include "overlap.cuh"
#include "xpcs_internal.h"

namespace xg {
namespace {

constexpr int MT_WARPS = 2;  // warps per block of the thread-per-pixel kernel
constexpr int WP_WARPS = 8;  // warps per block of the warp-per-pixel kernel
constexpr int MT_MID_CAP = 1024;  // long rows up to this length: 4 warps per block
constexpr int MID_WARPS = 4;
// Bins per entry up to which a level's pairs are taken by byte products
// (mt_warp_pixel).  The integer rows of 263 x 251 pixels x 16,000 frames, 744
// events each, take 2.95 / 2.25 / 2.00 / 1.97 / 1.98 ms with 0 (pairs by
// search and bitmask only) / 4 / 8 / 16 / 40.
constexpr int MB_RATIO = 16;
// The same for the thread kernel (mt_thread_rows), of the warp's longest row; its
// windows have at least MT_MIN_SCR scratch words.  At 1 Mpx x 10,000 frames,
// rows of 50 events, the integer rows take 2.53 / 2.29 / 2.27 / 2.26 / 2.25 /
// 2.41 ms with 0 / 4 / 8 / 12 / 16 / 20 bins per entry; at 512 x 512 x 1,000
// frames, rows of 10 and 4 delays a level, 161 / 143 / 139 / 141 us with 8 / 10
// / 12 / 16 words (8 are too few for any level's window).
constexpr int TB_RATIO = 12;
constexpr int LONG_WARPS = 2;  // warps per block for rows of up to MT_LONG_CAP events

// std::lower_bound as libstdc++ implements it (halving the remaining length),
// over lane-interleaved packed words (frame in the high half).
__device__ __forceinline__ int lower_bound_packed(const uint32_t *row, int n, int32_t x) {
  int first = 0, len = n;
  while (len > 0) {
    int half = len >> 1;
    if ((int32_t)(row[(first + half) * 32] >> 16) < x) {
      first += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return first;
}

__device__ __forceinline__ float pow2_neg(int e) { return __int_as_float((127 - e) << 23); }

// (float)num * 2^-shift / den as the reference's float arithmetic produces it
// (num is an integer below 2^24, den an integer below 2^16 as a float).  The
// IEEE quotient comes from the correctly rounded reciprocal by one residual
// correction (Markstein 1990; Muller et al., Handbook of Floating-Point
// Arithmetic, ch. 4): q0 = x*y, r = x - q0*den (exact by FMA), q = q0 + r*y.
// It equals the IEEE division for every 24-bit significand x and every integer
// den in [1, 65536] (checked exhaustively on the GPU against __fdiv_rn).
__device__ __forceinline__ float scaled_quotient(int num, int shift, float den, float rcp) {
  if (num == 0) return 0.f;
  const float x = __fmul_rn((float)num, pow2_neg(shift));
  if (!(den > 0.f)) return x;
  const float q0 = __fmul_rn(x, rcp);
  return __fmaf_rn(__fmaf_rn(-q0, den, x), rcp, q0);
}

// The same without branches, for divisors prepared by div_prep: num = 0 gives
// +0 through the correction steps, and a delay without division carries
// (den, rcp) = (1, 1), for which the steps return x unchanged.
__device__ __forceinline__ float scaled_quotient_nb(int num, int shift, float den, float rcp) {
  const float x = __fmul_rn((float)num, pow2_neg(shift));
  const float q0 = __fmul_rn(x, rcp);
  return __fmaf_rn(__fmaf_rn(-q0, den, x), rcp, q0);
}
__device__ __forceinline__ void div_prep(float &den, float &rcp) {
  if (!(den > 0.f)) {
    den = 1.f;
    rcp = 1.f;
  }
}

__device__ __forceinline__ int32_t pk_t(uint32_t w) { return (int32_t)(w >> 16); }
__device__ __forceinline__ int32_t pk_v(uint32_t w) { return (int32_t)(int16_t)(w & 0xffffu); }
__device__ __forceinline__ uint32_t pk(int32_t t, int32_t v) {
  return ((uint32_t)t << 16) | ((uint32_t)v & 0xffffu);
}

__device__ __forceinline__ void copy_plan(uint8_t *dst, const uint8_t *src, size_t bytes) {
  for (int k = threadIdx.x; k < (int)(bytes / 4); k += blockDim.x)
    ((int32_t *)dst)[k] = ((const int32_t *)src)[k];
}

// ------------------------------------------------------ thread per pixel

// Levels of at most 32 x (scratch words) bins: the thread keeps its row's
// occupied bins as a bitmask in its scratch words (lane-interleaved, one
// 32-bit word per 32 bins).  Bins in a row's live prefix are distinct and
// increasing, so the entry at bin b sits at position popcount(bits below b):
// one 64-bit window of the mask after a source's bin gives both the position
// of its first partner and which of the level's delays have one.  The KM >=
// count accumulators stay in registers and overwrite the mask once the
// sources are done; sources stop at the first bin whose first partner would
// be past lastframe.
template <int KM>
__device__ __forceinline__ void bins_pairs(const uint32_t *row, int m, int lf, int tlo,
                                                int count, int32_t *acc) {
  const uint32_t *mk = (const uint32_t *)acc;
  const int nw = (lf + 31) >> 5;
  int a[KM];
#pragma unroll
  for (int k = 0; k < KM; k++) a[k] = 0;
  const uint64_t gap = (1ull << (tlo - 1)) - 1ull;
  const uint32_t cmask = (1u << count) - 1u;
  for (int i = 0; i < m; i++) {
    const uint32_t wi = row[i * 32];
    const int ti = pk_t(wi);
    if (ti + tlo >= lf) break;
    const int s = ti + 1, q = s >> 5, sh = s & 31;  // s < lf: word q exists
    const uint32_t m0 = mk[q * 32];
    const uint32_t m1 = q + 1 < nw ? mk[(q + 1) * 32] : 0u;
    const uint32_t m2 = q + 2 < nw ? mk[(q + 2) * 32] : 0u;
    const uint64_t W = ((uint64_t)__funnelshift_r(m1, m2, sh) << 32) | __funnelshift_r(m0, m1, sh);
    int j = i + 1 + __popcll(W & gap);
    const uint32_t w = (uint32_t)(W >> (tlo - 1)) & cmask;
    const int vi = pk_v(wi);
#pragma unroll
    for (int k = 0; k < KM; k++) {
      if (w & (1u << k)) {
        a[k] += vi * pk_v(row[j * 32]);
        j++;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KM; k++)
    if (k < count) acc[k * 32] = a[k];
}

// Denser levels (at most TB_RATIO bins per entry of the warp's longest row):
// windows of the level's bins lie in the thread's W scratch words as bytes, one
// a bin, zero where no entry is.  The partners of 4 bins for delay tlo + k are
// the 4 bytes tlo + k further on: a funnel shift of two words gives them and a
// 4-way byte product the sum, so that a word costs 1 + 3 shifts and KM products
// whatever its bins hold, and no lane waits for another's search.  (Measured
// beside TB_RATIO; KM = 16 took 107 registers instead of 61 and was slower at
// every size.)  After a window the words that held only partners move to the
// front.  False (the same
// for all lanes): a value of some lane is not within a byte; acc is undefined.
template <int KM>
__device__ __forceinline__ bool byte_pairs_thread(const uint32_t *row, int m, int lf, int tlo,
                                                  int count, int W, int32_t *acc) {
  constexpr int Q = KM / 4;
  const int off = tlo >> 2, sh = (tlo & 3) * 8, H = off + Q + 1;  // H: words of partners only
  int a[KM];
#pragma unroll
  for (int k = 0; k < KM; k++) a[k] = 0;
#pragma unroll 4
  for (int q = 0; q < W; q++) acc[q * 32] = 0;
  unsigned most = 0;  // a negative value is past 255 as well
  int i = 0;
  uint32_t e = m > 0 ? row[0] : 0u;
  for (int b0 = 0;;) {
    const int bend = b0 + 4 * W;
    while (i < m && pk_t(e) < bend) {
      const int r = pk_t(e) - b0;
      most = max(most, e & 0xffffu);
      ((uint8_t *)acc)[(r >> 2) * 128 + (r & 3)] = (uint8_t)e;
      i++;
      e = row[i * 32];  // one past the row at most: a scratch word, not used
    }
    const int nown = min(W - H, (lf - b0 + 3) >> 2);
    const int32_t *X = acc + off * 32;
    // s[q][r]: the 4 bytes from 4 (w + q) + tlo + r on
    uint32_t s[Q][4], x1 = X[32], z = __funnelshift_r(X[0], x1, sh);
    const auto next = [&](int w, uint32_t (&d)[4]) {  // word w of the shifted stream
      const uint32_t x2 = X[(w + 2) * 32], z1 = __funnelshift_r(x1, x2, sh);
      d[0] = z;
#pragma unroll
      for (int r = 1; r < 4; r++) d[r] = __funnelshift_r(z, z1, 8 * r);
      x1 = x2;
      z = z1;
    };
#pragma unroll
    for (int q = 0; q < Q - 1; q++) next(q, s[q + 1]);
#pragma unroll 4
    for (int w = 0; w < nown; w++) {
#pragma unroll
      for (int q = 0; q < Q - 1; q++)
#pragma unroll
        for (int r = 0; r < 4; r++) s[q][r] = s[q + 1][r];
      next(w + Q - 1, s[Q - 1]);
      const uint32_t own = acc[w * 32];
      acc[w * 32] = 0;  // for the next window
#pragma unroll
      for (int k = 0; k < KM; k++) a[k] = (int)__dp4a(own, s[k / 4][k % 4], (unsigned)a[k]);
    }
    b0 += 4 * nown;
    if (b0 >= lf) break;
#pragma unroll 4
    for (int h = 0; h < H; h++) {
      acc[h * 32] = acc[(nown + h) * 32];  // nown >= H here
      acc[(nown + h) * 32] = 0;
    }
  }
  if (__any_sync(0xffffffffu, most > 255u)) return false;
#pragma unroll
  for (int k = 0; k < KM; k++)
    if (k < count) acc[k * 32] = a[k];
  return true;
}

// The 32 consecutive pixels of a warp (this lane's is p; mine: its outputs are
// written here, zeros for a row of 0 events), each lane's row of n0 events packed in its column of wbase, the warp's (CAP
// + scratch words) x 32 words of shared memory: the body of the
// thread-per-pixel kernels after the rows are loaded.
template <int CAP>
__device__ __forceinline__ void mt_thread_rows(const uint8_t *__restrict__ plan_g, int p, int n0,
                                               bool mine,
                                               float *__restrict__ G2, float *__restrict__ IP,
                                               float *__restrict__ IF, uint32_t *wbase) {
  // the plan is read from global memory: every lane of a warp reads the same
  // words (one L1-cached broadcast), and shared memory is left to the rows
  const McPlan *pl = (const McPlan *)plan_g;
  const int D = pl->D;
  const McArrays ar = mc_arrays(plan_g, D);
  const int P = pl->P, nlev = pl->nlev, mode = pl->mode;
  const int scr = pl->scr;
  const int lane = threadIdx.x & 31;
  uint32_t *row = wbase + lane;
  int32_t *acc = (int32_t *)(row + CAP * 32);  // scratch, also S(t_end) per level
  // total and S(t_end) per level (sweep from the end; t_end non-increasing)
  int total = 0;
  for (int i = 0; i < n0; i++) total += pk_v(row[i * 32]);
  {
    int j = n0 - 1, rsum = 0;
    for (int g = 0; g < nlev; g++) {
      const int te = pl->lv[g].t_end;
      while (j >= 0 && pk_t(row[j * 32]) >= te) {
        rsum += pk_v(row[j * 32]);
        j--;
      }
      acc[g * 32] = total - rsum;
    }
  }
  // IP and IF in one sweep over the delays, level group by level group: the
  // IP thresholds t_ip decrease with the delay index (a pointer from the end
  // of the row), the IF thresholds tau (in frames) increase (one from the
  // start).  Lane k loads the thresholds and divisor of the chunk's k-th
  // delay, and they are broadcast by shuffle.
  {
    const unsigned FULL = 0xffffffffu;
    int jp = n0 - 1, rsum = 0, jf = 0, ssum = 0;
    uint32_t wp = n0 > 0 ? row[(n0 - 1) * 32] : 0u;  // word at jp
    uint32_t wf = n0 > 0 ? row[0] : 0u;              // word at jf
    for (int g = 0; g < nlev; g++) {
      const McLevel L = pl->lv[g];
      const int lvl = L.level, s_end = acc[g * 32];
      for (int d0 = L.first; d0 < L.first + L.count; d0 += 32) {
        const int nd = min(32, L.first + L.count - d0);
        int tp_l = 0, tf_l = 0;
        float den_l = 0.f, rc_l = 0.f;
        if (lane < nd) {
          tp_l = ar.t_ip[d0 + lane];
          tf_l = ar.tau_abs[d0 + lane];
          den_l = ar.denom[d0 + lane];
          rc_l = ar.rcp[d0 + lane];
          div_prep(den_l, rc_l);
        }
        for (int k = 0; k < nd; k++) {
          const int Tp = __shfl_sync(FULL, tp_l, k), Tf = __shfl_sync(FULL, tf_l, k);
          const float den = __shfl_sync(FULL, den_l, k), rc = __shfl_sync(FULL, rc_l, k);
          // one step of each pointer without a branch (lanes step at different
          // delays), then a loop for the lanes that need more
          bool ap = jp >= 0 && pk_t(wp) >= Tp, af = jf < n0 && pk_t(wf) < Tf;
          {
            const uint32_t np = row[max(jp - 1, 0) * 32], nf = row[min(jf + 1, CAP - 1) * 32];
            rsum += ap ? pk_v(wp) : 0;
            ssum += af ? pk_v(wf) : 0;
            jp -= ap ? 1 : 0;
            jf += af ? 1 : 0;
            wp = ap ? (jp >= 0 ? np : 0u) : wp;
            wf = af ? (jf < n0 ? nf : 0u) : wf;
          }
          ap = jp >= 0 && pk_t(wp) >= Tp;
          af = jf < n0 && pk_t(wf) < Tf;
          if (__any_sync(FULL, ap || af)) {
            while (jp >= 0 && pk_t(wp) >= Tp) {
              rsum += pk_v(wp);
              jp--;
              wp = jp >= 0 ? row[jp * 32] : 0u;
            }
            while (jf < n0 && pk_t(wf) < Tf) {
              ssum += pk_v(wf);
              jf++;
              wf = jf < n0 ? row[jf * 32] : 0u;
            }
          }
          // lanes without a row of this kernel have n0 = 0: both numerators are 0
          if (mine) {
            const size_t o = (size_t)(d0 + k) * P + p;
            IP[o] = scaled_quotient_nb(total - rsum, lvl, den, rc);
            IF[o] = scaled_quotient_nb(s_end - ssum, lvl, den, rc);
          }
        }
      }
    }
  }

  // G2: level by level on the compacted buffer
  int m = n0;
  bool J = true, U = true;  // junction at m sorted; stale suffix [m, n0) sorted
  for (int g = 0; g < nlev; g++) {
    const McLevel L = pl->lv[g];
    if (L.compact && m > 0) {
      const int lf = L.lastframe;
      int index = -1, prev = INT_MIN;
      uint32_t wnext = row[0];
      for (int i = 0; i < m; i++) {
        const uint32_t w = wnext;
        wnext = row[min(i + 1, CAP - 1) * 32];  // ahead of the writes (index <= i)
        const int t = pk_t(w) >> 1;
        if (t >= lf) break;
        if (t == prev) {
          const uint32_t h = row[index * 32];
          row[index * 32] = pk(t, pk_v(h) + pk_v(w));
        } else {
          row[++index * 32] = pk(t, pk_v(w));
          prev = t;
        }
      }
      const int m2 = index + 1;
      U = (m2 < m) ? (J && U) : U;
      J = (m2 == 0 || m2 >= n0) ? true : (pk_t(row[(m2 - 1) * 32]) <= pk_t(row[m2 * 32]));
      m = m2;
    }
    const bool sorted = mode != XPCS_MODE_REFERENCE || (J && U);
    const int tlo = L.tau_lo, thi = L.tau_lo + L.count - 1;
    // warp-uniform: every lane of the warp sees the same level
    const int lf = L.lastframe;
    bool bytes = false;
    // a window's words: at least as many with sources as without
    if (tlo >= 1 && L.count <= 8 && 2 * ((tlo >> 2) + (L.count <= 4 ? 2 : 3)) <= scr &&
        lf <= TB_RATIO * __reduce_max_sync(0xffffffffu, m)) {
      if (L.count <= 4)
        bytes = byte_pairs_thread<4>(row, m, lf, tlo, L.count, scr, acc);
      else
        bytes = byte_pairs_thread<8>(row, m, lf, tlo, L.count, scr, acc);
    }
    const bool bins = tlo >= 1 && thi <= 64 && L.count <= 16 && L.lastframe <= 32 * scr;
    if (bytes) {
      if (!sorted) {
        // taken out again: entries that lower_bound over the whole buffer does
        // not find (none up to the tail's first bin when the tail ascends)
        const int tail0 = U && m < n0 ? pk_t(row[m * 32]) : (U ? INT_MAX : -1);
        for (int j = 1; j < m; j++) {
          const uint32_t wj = row[j * 32];
          const int tj = pk_t(wj);
          if (tj <= tail0 || lower_bound_packed(row, n0, tj) == j) continue;
          for (int i = j - 1; i >= 0; i--) {
            const uint32_t wi = row[i * 32];
            const int d = tj - pk_t(wi);
            if (d > thi) break;
            if (d >= tlo) acc[(d - tlo) * 32] -= pk_v(wi) * pk_v(wj);
          }
        }
      }
    } else if (bins && sorted) {
      // mask words in the scratch: zeroed, then one store per word that holds
      // an entry (the bins increase along the prefix)
      const int nw = (L.lastframe + 31) >> 5;
      for (int q = 0; q < nw; q++) acc[q * 32] = 0;
      int cq = -1;
      uint32_t cb = 0u;
      for (int i = 0; i < m; i++) {
        const int t = pk_t(row[i * 32]);
        if ((t >> 5) != cq) {
          if (cq >= 0) acc[cq * 32] = (int32_t)cb;
          cq = t >> 5;
          cb = 0u;
        }
        cb |= 1u << (t & 31);
      }
      if (cq >= 0) acc[cq * 32] = (int32_t)cb;
      if (L.count <= 8)
        bins_pairs<8>(row, m, L.lastframe, tlo, L.count, acc);
      else
        bins_pairs<16>(row, m, L.lastframe, tlo, L.count, acc);
    } else if (sorted) {
      for (int k = 0; k < L.count; k++) acc[k * 32] = 0;
      // per source the next three entries are checked without a branch (lanes
      // stay together); a loop runs only while the third one is still short of
      // the window's end.  Rows of 50 events at 1 Mpx: the integer rows 2.17 ms
      // with two entries, 2.13 with three, 2.07 also unrolled by three.
      const unsigned cnt = (unsigned)L.count;
      const uint32_t r0 = row[0], r1 = row[32];  // not used where m is less
      const uint32_t r2 = m > 2 ? row[64] : 0xffff0000u;
      int tb = pk_t(r0) + tlo, vi = pk_v(r0);
      int t1 = pk_t(r1), v1 = pk_v(r1), t2 = pk_t(r2), v2 = pk_v(r2);
#pragma unroll 3
      for (int i = 0; i < m - 1; i++) {
        const uint32_t w3 = i + 3 < m ? row[(i + 3) * 32] : 0xffff0000u;  // frame 65535, value 0
        const int t3 = pk_t(w3), v3 = pk_v(w3);
        const int u1 = t1 - tb, u2 = t2 - tb, u3 = t3 - tb;  // delays past the level's first
        const bool p1 = (unsigned)u1 < cnt, p2 = (unsigned)u2 < cnt, p3 = (unsigned)u3 < cnt;
        int32_t x1 = 0, x2 = 0, x3 = 0;  // u1 < u2 < u3: three sums, read before any is written
        if (p1) x1 = acc[u1 * 32];
        if (p2) x2 = acc[u2 * 32];
        if (p3) x3 = acc[u3 * 32];
        // the nearest last: a last entry in frame 65535 shares its sum with the
        // 0 that stands past the row's end
        if (p3) acc[u3 * 32] = x3 + vi * v3;
        if (p2) acc[u2 * 32] = x2 + vi * v2;
        if (p1) acc[u1 * 32] = x1 + vi * v1;
        if (u3 < (int)cnt - 1 && i + 4 < m) {
          for (int j = i + 4; j < m; j++) {
            const uint32_t wj = row[j * 32];
            const int u = pk_t(wj) - tb;
            if (u >= (int)cnt) break;
            if (u >= 0) acc[u * 32] += vi * pk_v(wj);
          }
        }
        tb = t1 + tlo;
        vi = v1;
        t1 = t2;
        v1 = v2;
        t2 = t3;
        v2 = v3;
      }
    } else {
      // the buffer is not globally sorted: a pair counts only when the
      // reference's lower_bound over the whole buffer lands on the partner
      for (int k = 0; k < L.count; k++) acc[k * 32] = 0;
      for (int i = 0; i < m; i++) {
        const uint32_t wi = row[i * 32];
        const int ti = pk_t(wi);
        for (int j = i + 1; j < m; j++) {
          const uint32_t wj = row[j * 32];
          const int d = pk_t(wj) - ti;
          if (d > thi) break;
          if (d >= tlo && lower_bound_packed(row, n0, pk_t(wj)) == j)
            acc[(d - tlo) * 32] += pk_v(wi) * pk_v(wj);
        }
      }
    }
    // divisors broadcast by shuffle as in the IP/IF sweep; lanes without a
    // row of this kernel have zero sums
    for (int d0 = L.first; d0 < L.first + L.count; d0 += 32) {
      const int nd = min(32, L.first + L.count - d0);
      float den_l = 0.f, rc_l = 0.f;
      if (lane < nd) {
        den_l = ar.denom[d0 + lane];
        rc_l = ar.rcp[d0 + lane];
        div_prep(den_l, rc_l);
      }
      for (int k = 0; k < nd; k++) {
        const float den = __shfl_sync(0xffffffffu, den_l, k), rc = __shfl_sync(0xffffffffu, rc_l, k);
        if (mine)
          G2[(size_t)(d0 + k) * P + p] =
              scaled_quotient_nb(acc[(d0 - L.first + k) * 32], 2 * L.level, den, rc);
      }
    }
  }
}

// One warp's 32 consecutive pixels p0 .. p0+31 of a series: the rows loaded
// and run, shared by the per-series launch and by the batch's work-queue
// launch.
template <int CAP>
__device__ __forceinline__ void mt_thread_warp(const uint8_t *__restrict__ plan_g,
                                               const int64_t *__restrict__ row_ptr,
                                               const int32_t *__restrict__ row_len,
                                               const uint8_t *__restrict__ pclass,
                                               const int32_t *__restrict__ ev_frame,
                                               const float *__restrict__ ev_val,
                                               float *__restrict__ G2, float *__restrict__ IP,
                                               float *__restrict__ IF, int p0,
                                               uint32_t *wbase) {
  const int P = ((const McPlan *)plan_g)->P, lane = threadIdx.x & 31;
  if (p0 >= P) return;
  const int p = p0 + lane;
  const int c = p < P ? pclass[p] : PCLASS_FLOAT;
  const bool mine = c == PCLASS_THREAD || c == PCLASS_EMPTY;  // the others' kernels write theirs
  if (!__any_sync(0xffffffffu, mine)) return;
  const int n0 = c == PCLASS_THREAD ? row_len[p] : 0;
  if (!__any_sync(0xffffffffu, n0 > 0)) {  // zeros only
    if (!mine) return;
    const int D = ((const McPlan *)plan_g)->D;
    for (int d = 0; d < D; d++) {
      const size_t o = (size_t)d * P + p;
      G2[o] = IP[o] = IF[o] = 0.f;
    }
    return;
  }

  // cooperative, coalesced load of the warp's rows (consecutive pixels have
  // consecutive rows), scattered to the owning lane's slots; four chunks of
  // 32 events in flight per lane.  Positions are relative to the warp's first
  // event: when a lane owns a packed row every frame is below 65536, so the
  // 32 rows span fewer than 2^21 events.
  const unsigned FULL = 0xffffffffu;
  const int plast = min(p0 + 32, P);
  const int64_t e0 = row_ptr[p0];
  const int nw = (int)(row_ptr[plast] - e0);
  const int my_b = p < P ? (int)(row_ptr[p] - e0) : nw;
  const int lo = __reduce_min_sync(FULL, n0 > 0 ? my_b : INT_MAX);
  const int hi = __reduce_max_sync(FULL, n0 > 0 ? my_b + n0 : 0);
  for (int base = lo; base < hi; base += 128) {
    int dst[4], fr[4];
    float vl[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int e = base + u * 32 + lane;
      int owner = 0;  // last lane whose row starts at or before e
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const int cand = owner + o;
        const int cb = __shfl_sync(FULL, my_b, cand & 31);
        if (cand < 32 && cb <= e) owner = cand;
      }
      const int slot = e - __shfl_sync(FULL, my_b, owner);
      const int olen = __shfl_sync(FULL, n0, owner);
      dst[u] = (e < hi && slot < olen) ? slot * 32 + owner : -1;
      if (dst[u] >= 0) {
        fr[u] = ev_frame[e0 + e];
        vl[u] = ev_val[e0 + e];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (dst[u] >= 0) wbase[dst[u]] = pk(fr[u], __float2int_rn(vl[u]));
  }
  __syncwarp();
  mt_thread_rows<CAP>(plan_g, p, n0, mine, G2, IP, IF, wbase);
}

// ---------------------------------------------------- overlapping launches
//
// The multi-tau kernels of a series write the results of different pixels, so
// one may begin while the last blocks of the one before still run: each calls
// overlap_begin first (the next launch_overlapped kernel may start once every
// block of this one has) and overlap_end last (this kernel is complete only
// when the one before is, so that what follows in the stream waits for all of
// them).  What they read was written before the first, which is launched
// plainly.  The longest rows' launch, a few warps busy for as long as their
// rows take, comes first and the other launches fill the chip beside it; a
// counter hands out the rows, since blocks begin at different times (a fixed
// share for each block: 2.6 ms).  263 x 251 pixels x 16,000 frames, rows of 744
// events: the integer rows 1.97 ms one launch after the other, 1.62 overlapped.

template <int CAP>
__global__ void __launch_bounds__(MT_WARPS * 32, 16)
k_mt_thread(const uint8_t *__restrict__ plan_g, const int64_t *__restrict__ row_ptr,
            const int32_t *__restrict__ row_len, const uint8_t *__restrict__ pclass,
            const int32_t *__restrict__ ev_frame, const float *__restrict__ ev_val,
            float *__restrict__ G2, float *__restrict__ IP, float *__restrict__ IF) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int scr = ((const McPlan *)plan_g)->scr;
  const int warp = threadIdx.x >> 5;
  uint32_t *wbase = (uint32_t *)smem + (size_t)warp * (CAP + scr) * 32;
  overlap_begin();
  mt_thread_warp<CAP>(plan_g, row_ptr, row_len, pclass, ev_frame, ev_val, G2, IP, IF,
                      (blockIdx.x * MT_WARPS + warp) * 32, wbase);
  overlap_end();
}

// ------------------------------------------------------- warp per pixel

// lower_bound over a contiguous packed row (frame in the high half)
__device__ __forceinline__ int lower_bound_row(const uint32_t *row, int n, int32_t x) {
  int first = 0, len = n;
  while (len > 0) {
    int half = len >> 1;
    if ((int32_t)(row[first + half] >> 16) < x) {
      first += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return first;
}

// In-place compaction of the live prefix row[0, m) for the next level
// (warp-cooperative): frame/2, equal neighbours merged, frames >= lastframe
// dropped.  Entries at and beyond the returned length are left untouched
// (the reference's stale tail).
__device__ int compact_row(uint32_t *row, int m, int lastframe, int lane) {
  const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
  int gbase = 0;
  int prev = INT_MIN;  // halved frame of the entry before the current chunk
  for (int c0 = 0; c0 < m; c0 += 32) {
    const int i = c0 + lane;
    const bool in = i < m;
    const uint32_t w = in ? row[i] : 0u;
    const int ti = in ? (pk_t(w) >> 1) : INT_MAX;
    int vi = in ? pk_v(w) : 0;
    if (i + 1 < m) {
      const uint32_t w2 = row[i + 1];
      if ((pk_t(w2) >> 1) == ti) vi += pk_v(w2);  // rows hold distinct frames: pairs at most
    }
    int tp = __shfl_up_sync(FULL, ti, 1);
    if (lane == 0) tp = prev;
    const bool head = in && ti != tp && ti < lastframe;
    const unsigned hm = __ballot_sync(FULL, head);
    prev = __shfl_sync(FULL, ti, 31);
    __syncwarp();
    if (head) row[gbase + __popc(hm & lt)] = pk(ti, vi);
    gbase += __popc(hm);
    __syncwarp();
    if (prev >= lastframe) break;
  }
  return gbase;
}

// G2 sums of one level from its bins as bytes: S holds the level's values, one
// byte per bin, zero where no entry is and in the MB_PAD words past the last
// bin.  Lanes take words of 4 bins: for each delay the bins that far on (byte
// funnel shifts of the words after) meet the lane's own in a 4-way byte
// product, so an empty bin costs no test and an occupied one no search.
// a[k]: this lane's share of delay tlo + k, KM delays from tlo <= 31 on.
constexpr int MB_PAD = 16;
template <int KM>
__device__ __forceinline__ void byte_pairs(const uint32_t *S, int lf, int tlo, int lane,
                                           unsigned (&a)[KM]) {
  const uint32_t *T = S + (tlo >> 2);
  const int sh = (tlo & 3) * 8, nw = (lf + 3) >> 2;
  for (int w = lane; w < nw; w += 32) {
    const uint32_t own = S[w];
    uint32_t x[KM / 4 + 2], z[KM / 4 + 1];
#pragma unroll
    for (int j = 0; j < KM / 4 + 2; j++) x[j] = T[w + j];
#pragma unroll
    for (int j = 0; j < KM / 4 + 1; j++) z[j] = __funnelshift_r(x[j], x[j + 1], sh);
#pragma unroll
    for (int k = 0; k < KM; k++) {
      const uint32_t p =
          k % 4 ? __funnelshift_r(z[k / 4], z[k / 4 + 1], 8 * (k % 4)) : z[k / 4];
      a[k] = __dp4a(own, p, a[k]);
    }
  }
}

// One warp per pixel of `list` (count at *count_p) whose row holds more than
// min_n and at most `cap` events, packed (frame << 16 | int16 value) in the warp's shared memory, with
// the row's inclusive prefix sums and per-lane accumulators beside it.
//   IP / IF: from the original row, as in the thread kernel: lanes take the
//     delays and look the thresholds up in the prefix sums.
//   G2: per level, warp-cooperative compaction, then every lane takes the
//     sources lane, lane+32, ... in one flat loop over (source, partner)
//     visits into its own accumulators, summed over the warp at the end of
//     the level.  Where at least one bin in MB_RATIO holds an entry and the
//     level's bins fit the prefix-sum array (done with after IP/IF) as bytes,
//     byte products take the place of the visits (byte_pairs); entries that
//     the reference's search misses (an unsorted buffer) are then taken out
//     again as partners.  Where only words fit and a fifth of the bins hold an
//     entry, the array holds the values by bin (counts above 255) and a source
//     finds each partner by one lookup.  On other sorted levels of at most 32
//     delays, none above 64, where the row could reach every delay (m x
//     (thi + 1) >= lastframe), the same words hold the row's occupancy bitmask:
//     a source reads the 64 bins after it, finds its first partner's index by a
//     population count over the bins below tau_lo and visits only the occupied
//     bins of the delay window.
// One pixel p of a series with a row of n0 events from event b on (min_n < n0
// <= cap): the body of the warp-per-pixel kernel, shared by its per-series launches and by
// the batch's work-queue launches.  pl / ar: the plan (shared or global
// memory); row, S: the warp's 2 x cap words; acc: this lane's accumulators
// (acc[k * 32]).
__device__ __forceinline__ void mt_warp_pixel(const McPlan *pl, const McArrays &ar, int p,
                                              int64_t b, int n0,
                                              const int32_t *__restrict__ ev_frame,
                                              const float *__restrict__ ev_val,
                                              float *__restrict__ G2, float *__restrict__ IP,
                                              float *__restrict__ IF, int cap, uint32_t *row,
                                              int32_t *S, int32_t *acc) {
  const int P = pl->P, mode = pl->mode, D = pl->D;
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  int carry = 0;
  for (int c0 = 0; c0 < n0; c0 += 32) {
    const int i = c0 + lane;
    int x = 0;
    if (i < n0) {
      x = __float2int_rn(ev_val[b + i]);
      row[i] = pk(ev_frame[b + i], x);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    if (i < n0) S[i] = x + carry;
    carry += __shfl_sync(FULL, x, 31);
  }
  __syncwarp();
  // IP(d) = S(t_ip[d]); IF(d) = S(t_end of its level) - S(tau_abs[d]); S(T) = sum of
  // v over frames < T
  for (int d = lane; d < D; d += 32) {
    const int g = ar.gi[d];
    const int lvl = pl->lv[g].level;
    const int c_ip = lower_bound_row(row, n0, ar.t_ip[d]);
    const int c_end = lower_bound_row(row, n0, pl->lv[g].t_end);
    const int c_tau = lower_bound_row(row, n0, ar.tau_abs[d]);
    const int ip = c_ip ? S[c_ip - 1] : 0;
    const int iff = (c_end ? S[c_end - 1] : 0) - (c_tau ? S[c_tau - 1] : 0);
    IP[(size_t)d * P + p] = scaled_quotient(ip, lvl, ar.denom[d], ar.rcp[d]);
    IF[(size_t)d * P + p] = scaled_quotient(iff, lvl, ar.denom[d], ar.rcp[d]);
  }
  int m = n0;
  bool J = true, U = true;  // junction at m sorted; stale suffix [m, n0) sorted
  for (int gi = 0; gi < pl->nlev; gi++) {
    const McLevel L = pl->lv[gi];
    if (L.compact && m > 0) {
      const int m2 = compact_row(row, m, L.lastframe, lane);
      U = (m2 < m) ? (J && U) : U;
      J = (m2 == 0 || m2 >= n0) ? true : (pk_t(row[m2 - 1]) <= pk_t(row[m2]));
      m = m2;
    }
    const bool sorted = mode != XPCS_MODE_REFERENCE || (J && U);
    const int tlo = L.tau_lo, thi = L.tau_lo + L.count - 1;
    const int lf = L.lastframe;
    bool bytes = tlo >= 1 && tlo <= 31 && L.count <= 16 && ((lf + 3) >> 2) + MB_PAD <= cap &&
                 lf <= MB_RATIO * m;
    if (bytes) {
      const int nw = (lf + 3) >> 2;
      for (int q = lane; q < nw + MB_PAD; q += 32) S[q] = 0;
      __syncwarp();
      unsigned most = 0;  // a negative value is past 255 as well
      for (int k = lane; k < m; k += 32) {
        const uint32_t e = row[k];
        most = max(most, (unsigned)pk_v(e));
        ((uint8_t *)S)[pk_t(e)] = (uint8_t)pk_v(e);
      }
      bytes = __reduce_max_sync(FULL, most) <= 255u;
      __syncwarp();
    }
    if (bytes) {
      const auto level = [&](auto km) {
        constexpr int KM = decltype(km)::value;
        unsigned a[KM];
#pragma unroll
        for (int k = 0; k < KM; k++) a[k] = 0;
        byte_pairs<KM>((const uint32_t *)S, lf, tlo, lane, a);
        if (!sorted) {
          // partners that lower_bound over the whole buffer does not find: none
          // up to the tail's first bin when the tail ascends
          const int tail0 = U && m < n0 ? pk_t(row[m]) : (U ? INT_MAX : -1);
          for (int i = lane; i < m; i += 32) {
            const int t = pk_t(row[i]);
            if (t <= tail0 || lower_bound_row(row, n0, t) == i) continue;
            const unsigned v = (unsigned)pk_v(row[i]);
#pragma unroll
            for (int k = 0; k < KM; k++)
              if (t - tlo - k >= 0) a[k] -= v * ((const uint8_t *)S)[t - tlo - k];
          }
        }
        int mine = 0;
#pragma unroll
        for (int k = 0; k < KM; k++) {
          if (k >= L.count) break;
          const int tot = __reduce_add_sync(FULL, (int)a[k]);
          if (lane == k) mine = tot;
        }
        if (lane < L.count) {
          const int d = L.first + lane;
          G2[(size_t)d * P + p] = scaled_quotient(mine, 2 * L.level, ar.denom[d], ar.rcp[d]);
        }
        __syncwarp();
      };
      if (L.count <= 8)
        level(std::integral_constant<int, 8>{});
      else
        level(std::integral_constant<int, 16>{});
      continue;
    }
    for (int k = 0; k < L.count; k++) acc[k * 32] = 0;
    if (sorted && tlo >= 1 && lf <= cap && 5 * m >= lf) {
      // at least a fifth of the level's bins hold an entry: the prefix sums
      // S are done with, and S becomes the row's values by bin, so that each
      // source finds its partner for every delay with one lookup (a missing
      // bin reads 0, which adds nothing)
      for (int bq = lane; bq < lf; bq += 32) S[bq] = 0;
      __syncwarp();
      for (int k = lane; k < m; k += 32) S[pk_t(row[k])] = pk_v(row[k]);
      __syncwarp();
      for (int i = lane; i < m; i += 32) {
        const uint32_t wi = row[i];
        const int ti = pk_t(wi), vi = pk_v(wi);
        for (int k = 0; k < L.count; k++) {
          const int tb = ti + tlo + k;
          if (tb < lf) acc[k * 32] += vi * S[tb];
        }
      }
    } else if (sorted && tlo >= 1 && thi <= 64 && L.count <= 32 && lf <= 32 * cap &&
               m * (thi + 1) >= lf) {
      // about one entry or more per delay window: S (done with after IP/IF)
      // becomes the level's occupancy bitmask.  Bins of the prefix are distinct
      // and increasing, so the entry at bin b is at position popcount(bits
      // below b): one 64-bit window of the mask after a source's bin gives the
      // position of its first partner (entries closer than the smallest delay
      // are counted, not visited) and which delays have a partner
      uint32_t *mk = (uint32_t *)S;
      const int nw = (lf + 31) >> 5;
      for (int q = lane; q < nw; q += 32) mk[q] = 0u;
      __syncwarp();
      for (int k = lane; k < m; k += 32) {
        const int t = pk_t(row[k]);
        atomicOr(&mk[t >> 5], 1u << (t & 31));
      }
      __syncwarp();
      const uint64_t gap = (1ull << (tlo - 1)) - 1ull;
      const uint32_t cmask = L.count >= 32 ? 0xffffffffu : ((1u << L.count) - 1u);
      for (int i = lane; i < m; i += 32) {
        const uint32_t wi = row[i];
        const int ti = pk_t(wi);
        if (ti + tlo >= lf) break;  // this and later sources have no partner below lastframe
        const int s0 = ti + 1, q = s0 >> 5, sh = s0 & 31;  // s0 < lf: word q exists
        const uint32_t m0 = mk[q];
        const uint32_t m1 = q + 1 < nw ? mk[q + 1] : 0u;
        const uint32_t m2 = q + 2 < nw ? mk[q + 2] : 0u;
        const uint64_t W =
            ((uint64_t)__funnelshift_r(m1, m2, sh) << 32) | __funnelshift_r(m0, m1, sh);
        int j = i + 1 + __popcll(W & gap);
        uint32_t w = (uint32_t)(W >> (tlo - 1)) & cmask;
        const int vi = pk_v(wi);
        while (w) {
          const int k = __ffs(w) - 1;
          acc[k * 32] += vi * pk_v(row[j]);
          j++;
          w &= w - 1u;
        }
      }
      __syncwarp();
    } else {
      int i = lane, j = lane + 1;
      uint32_t wi = i < m ? row[i] : 0u;
      uint32_t wj = j < m ? row[j] : 0u;
      while (i < m) {
        const int d = pk_t(wj) - pk_t(wi);
        if (j < m && d <= thi) {
          if (d >= tlo && (sorted || lower_bound_row(row, n0, pk_t(wj)) == j))
            acc[(d - tlo) * 32] += pk_v(wi) * pk_v(wj);
          j++;
        } else {
          i += 32;
          if (i >= m) break;
          wi = row[i];
          j = i + 1;
        }
        wj = j < m ? row[j] : 0u;
      }
    }
    for (int k0 = 0; k0 < L.count; k0 += 32) {  // a lane each for 32 delays
      int mine = 0;
      const int nk = min(32, L.count - k0);
      for (int k = 0; k < nk; k++) {
        const int tot = __reduce_add_sync(FULL, acc[(k0 + k) * 32]);
        if (lane == k) mine = tot;
      }
      if (lane < nk) {
        const int d = L.first + k0 + lane;
        G2[(size_t)d * P + p] = scaled_quotient(mine, 2 * L.level, ar.denom[d], ar.rcp[d]);
      }
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256)
k_mt_warp(const uint8_t *__restrict__ plan_g, const int32_t *__restrict__ list,
          const int32_t *__restrict__ count_p, int32_t min_n, int32_t cap,
          const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ row_len,
          const int32_t *__restrict__ ev_frame, const float *__restrict__ ev_val,
          float *__restrict__ G2, float *__restrict__ IP, float *__restrict__ IF,
          int32_t *__restrict__ next) {
  extern __shared__ __align__(16) uint8_t smem[];
  overlap_begin();
  const int nw = *count_p;
  if (nw == 0) return overlap_end();
  const int D = ((const McPlan *)plan_g)->D;
  const size_t pb = mc_plan_bytes(D);
  copy_plan(smem, plan_g, pb);
  __syncthreads();
  const McPlan *pl = (const McPlan *)smem;
  const McArrays ar = mc_arrays(smem, D);
  const int ACC = max(pl->acc, pl->nlev);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *row = (uint32_t *)(smem + pb) + (size_t)warp * (2 * cap + 32 * ACC);
  int32_t *S = (int32_t *)(row + cap);
  int32_t *acc = S + cap + lane;  // acc[k * 32]: this lane's accumulator k
  // rows one by one from a counter: blocks begin as the launch before ends
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(next, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= nw) break;
    const int p = list[q];
    const int n0 = row_len[p];
    if (n0 <= min_n || n0 > cap) continue;  // another launch's share of the list
    mt_warp_pixel(pl, ar, p, row_ptr[p], n0, ev_frame, ev_val, G2, IP, IF, cap, row, S, acc);
  }
  overlap_end();
}

// ------------------------------------------------ batch work-queue launches
//
// The multi-tau of every member of a batch as persistent grids that pull work
// items from a device counter: 32-pixel groups of every member with the same
// thread-kernel row capacity in one launch, the warp-per-pixel rows of every
// member in one launch per row tier.  Small members' items run beside large
// members' items, and no member's kernel leaves a tail of idle SMs.

// Thread-per-pixel items: group g of the queue is group g - first of the
// member whose range holds it.  wbase strides by the batch's largest scratch.
template <int CAP>
__global__ void __launch_bounds__(MT_WARPS * 32, 16)
k_mt_thread_queue(const MtQueueMember *__restrict__ tab, int32_t n, int32_t total,
                  int32_t scr_max, int32_t *__restrict__ next) {
  extern __shared__ __align__(16) uint8_t smem[];
  overlap_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *wbase = (uint32_t *)smem + (size_t)warp * (CAP + scr_max) * 32;
  for (;;) {
    int g = 0;
    if (lane == 0) g = atomicAdd(next, 1);
    g = __shfl_sync(0xffffffffu, g, 0);
    if (g >= total) break;
    int lo = 0, hi = n - 1;  // the last member whose first group is <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tab[mid].first <= g) lo = mid;
      else hi = mid - 1;
    }
    const MtQueueMember &m = tab[lo];
    mt_thread_warp<CAP>(m.plan, m.row_ptr, m.row_len, m.pclass, m.ev_frame, m.ev_val, m.G2, m.IP,
                        m.IF, (g - m.first) * 32, wbase);
    __syncwarp();
  }
  overlap_end();
}

// Warp-per-pixel items: entry q of the members' warp lists (use_long = 0) or
// long-row lists, concatenated in table order; rows outside (min_n, cap]
// belong to another tier's launch.  The plan is read from global memory.
__global__ void __launch_bounds__(256)
k_mt_warp_queue(const MtQueueMember *__restrict__ tab, int32_t n, int32_t use_long,
                int32_t min_n, int32_t cap, int32_t acc_max, int32_t *__restrict__ next) {
  extern __shared__ __align__(16) uint8_t smem[];
  overlap_begin();
  int32_t *pref = (int32_t *)smem;  // [n + 1]: first entry of each member's list
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    int32_t t = 0;
    for (int i = 0; i < n; i++) {
      pref[i] = t;
      t += use_long ? tab[i].stats->nlong : tab[i].stats->nwarp;
    }
    pref[n] = t;
  }
  __syncthreads();
  const int total = pref[n];
  const size_t pref_bytes = mc_align16(sizeof(int32_t) * (size_t)(n + 1));
  uint32_t *row = (uint32_t *)(smem + pref_bytes) + (size_t)warp * (2 * cap + 32 * acc_max);
  int32_t *S = (int32_t *)(row + cap);
  int32_t *acc = S + cap + lane;
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(next, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= total) break;
    int lo = 0, hi = n - 1;  // the last member whose list starts at or before q
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pref[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    const MtQueueMember &m = tab[lo];
    const int p = (use_long ? m.llist : m.wlist)[q - pref[lo]];
    const int n0 = m.row_len[p];
    if (n0 <= min_n || n0 > cap) continue;
    const McPlan *pl = (const McPlan *)m.plan;
    const McArrays ar = mc_arrays(m.plan, pl->D);
    mt_warp_pixel(pl, ar, p, m.row_ptr[p], n0, m.ev_frame, m.ev_val, m.G2, m.IP, m.IF, cap, row,
                  S, acc);
  }
  overlap_end();
}

// --------------------------------------------------------- float replay

__global__ void __launch_bounds__(128)
k_mt_float(const uint8_t *__restrict__ plan_g, const int32_t *__restrict__ flist,
           const DevStats *__restrict__ stats, const int64_t *__restrict__ row_ptr,
           const int32_t *__restrict__ row_len, const int32_t *__restrict__ ev_frame,
           const float *__restrict__ ev_val, const float *__restrict__ fscale,
           int32_t *__restrict__ sc_frame, float *__restrict__ sc_val, float *__restrict__ G2,
           float *__restrict__ IP, float *__restrict__ IF) {
  const McPlan *pl = (const McPlan *)plan_g;
  const int D = pl->D, P = pl->P;
  const McArrays ar = mc_arrays(plan_g, D);
  const int nf = stats->nfloat;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nf; q += gridDim.x * blockDim.x) {
    const int p = flist[q];
    const int64_t b = row_ptr[p];
    const int n0 = row_len[p];
    int32_t *idx = sc_frame + b;
    float *val = sc_val + b;
    for (int i = 0; i < n0; i++) {
      idx[i] = ev_frame[b + i];
      // normalize_by_framesum: v / (frameSum[f] / mean) (main.cpp:330-333)
      val[i] = fscale ? __fdiv_rn(ev_val[b + i], fscale[idx[i]]) : ev_val[b + i];
    }
    replay_pixel(pl, ar, P, p, idx, val, n0, G2, IP, IF);
  }
}

// ------------------------------------------------ float rows, warp per pixel
//
// The same operations as k_mt_float, in the same order per sum, with the work
// of one pixel spread over a warp:
//   * the row is compacted in place in the scratch buffer exactly as the
//     reference does it (so the stale tail is the reference's), 32 entries per
//     step: each entry's half index, a ballot of the group starts and the pair
//     sum (v[i] + v[i+1]) / 2 of merged neighbours;
//   * lower_bound over the whole buffer lands on a prefix entry j exactly when
//     lower_bound(idx[j]) == j ("findable"); the search result is monotone in
//     its argument, so a pair (r, j) counts iff idx[j] == idx[r] + tau and j is
//     findable.  While the buffer is sorted (tracked per level from the
//     junctions between the prefix and the older segments) every entry is
//     findable; otherwise each lane runs the reference's search for its entry;
//   * each float sum (G2, IP, IF of every delay of the level) is a chain that
//     one lane accumulates in the reference's order: per 32 entries the lanes
//     first write their terms (v*v' of the pair with distance tau, or v inside
//     the IP / IF ranges, else +0, which leaves a sum unchanged) to shared
//     memory, then each chain's lane adds its 32 terms in entry order.
// Partners lie at most tau entries ahead (distinct ascending indices), so a
// ring of two 32-entry tiles holds every partner of the current tile.
constexpr int FW_WARPS = 4;
constexpr int FW_MAXC = 32;  // delays per level and largest delay in level units
// Term rows of 36 floats: 16-byte aligned, so a chain's lane reads its 32
// terms as 8 float4 loads; lanes 0-7 of such a load (chains 0-7) touch banks
// 4*chain .. 4*chain+3, distinct, so the loads stay free of bank conflicts.
constexpr int FW_TSTRIDE = 36;
constexpr int FW_WIN = 128;  // bins of the per-warp partner window

// Shared memory of one warp: ring idx[64], val[64]; the bin window's values
// [FW_WIN]; terms [3 * acc][FW_TSTRIDE] and the shared IP/IF row
// [FW_TSTRIDE]; rounded up to 16 bytes.  (The ring's findable flags are a
// register mask: at 16 delays in a level this makes 8,080 bytes, and 4 warps
// per block fit 7 blocks on an SM.)
__host__ __device__ constexpr size_t fw_warp_bytes(int acc_max) {
  return (64 * 8 + FW_WIN * 4 + (3 * (size_t)acc_max + 1) * FW_TSTRIDE * 4 + 15) & ~(size_t)15;
}

__device__ __forceinline__ int lower_bound_g(const int32_t *a, int n, int32_t x) {
  int first = 0, len = n;
  while (len > 0) {
    const int half = len >> 1;
    if (a[first + half] < x) {
      first += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return first;
}

// Entry tb + lane of the level's row with its findable flag, fetched into
// registers (fw_fetch) some time before it goes into its ring slot (fw_put),
// so that the load's latency passes while a tile is processed.
struct FwEntry {
  int32_t x;
  float v;
  uint8_t f;
};

__device__ __forceinline__ FwEntry fw_fetch(int tb, int lane, int L, int n0, bool all_find,
                                            const int32_t *idx, const float *val) {
  FwEntry e{0, 0.f, 0};
  const int j = tb + lane;
  if (j < L) {
    e.x = idx[j];
    e.v = val[j];
    e.f = all_find ? 1 : (lower_bound_g(idx, n0, e.x) == j);
  }
  return e;
}

// The ring's findable flags are one 64-bit mask, the same in every lane: tb is
// a multiple of 32, so a tile fills one half of the ring, bits (tb & 32) on.
__device__ __forceinline__ void fw_put(int tb, int lane, int L, const FwEntry &e, int32_t *ridx,
                                       float *rval, uint64_t &fmask) {
  const int j = tb + lane, slot = j & 63;
  if (j < L) {
    ridx[slot] = e.x;
    rval[slot] = e.v;
  }
  const uint64_t b = __ballot_sync(0xffffffffu, j < L && e.f);
  const int sh = tb & 32;
  fmask = (fmask & ~(0xffffffffull << sh)) | (b << sh);
}

__device__ __forceinline__ bool fw_findable(uint64_t fmask, int j) {
  return (fmask >> (j & 63)) & 1u;
}

// One pixel p with a row of n0 events from event b on: the scratch row idx /
// val, the warp's shared memory wb (fw_warp_bytes).
__device__ __forceinline__ void fw_pixel(const McPlan *pl, const McArrays &ar, int p, int64_t b,
                                         int n0, const int32_t *__restrict__ ev_frame,
                                         const float *__restrict__ ev_val,
                                         const float *__restrict__ fscale, int32_t *idx,
                                         float *val, float *__restrict__ G2,
                                         float *__restrict__ IP, float *__restrict__ IF,
                                         uint8_t *wb) {
  const int P = pl->P, nlev = pl->nlev, acc_max = pl->acc;
  const bool ref = pl->mode == XPCS_MODE_REFERENCE;
  const int lane = threadIdx.x & 31;
  int32_t *ridx = (int32_t *)wb;
  float *rval = (float *)(wb + 256);
  // bin b of the window: the value of the entry at b0 + b when it is
  // findable, else 0; the G2 term v * 0 = +-0 then leaves its chain
  // unchanged (the chains start at +0 and x + -x is +0, so no chain is ever
  // -0, and a + +-0 == a for every other a)
  float *bval = (float *)(wb + 512);
  float *terms = (float *)(wb + 512 + FW_WIN * 4);
  float *vrow = terms + (size_t)3 * acc_max * FW_TSTRIDE;
  for (int i0 = 0; i0 < n0; i0 += 4 * 32) {
    int32_t f[4];
    float x[4];
#pragma unroll
    for (int h = 0; h < 4; h++) {  // the loads first, in flight together
      const int i = i0 + h * 32 + lane;
      if (i < n0) {
        f[h] = ev_frame[b + i];
        x[h] = ev_val[b + i];
      }
    }
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int i = i0 + h * 32 + lane;
      if (i < n0) {
        idx[i] = f[h];
        // normalize_by_framesum: v / (frameSum[f] / mean) (main.cpp:330-333)
        val[i] = fscale ? __fdiv_rn(x[h], fscale[f[h]]) : x[h];
      }
    }
  }
  __syncwarp();
  int L = n0;
  bool tail_sorted = true, dead = false;
  for (int gi = 0; gi < nlev; gi++) {
    const McLevel lv = pl->lv[gi];
    const int lastframe = lv.lastframe, cnt = lv.count, t0 = lv.tau_lo;
    if (lv.compact && !dead) {
      const int prevL = L;
      // the junction between the previous prefix and the older tail
      bool junction_ok = true;
      if (prevL < n0) junction_ok = idx[prevL - 1] <= idx[prevL];
      if ((idx[0] >> 1) >= lastframe) {
        dead = true;  // nothing is kept: lastIndex becomes 1 on a stale entry
      } else {
        int out = 0, carry_h = -1;
        // chunks of 32 entries, each loaded two chunks ahead: a chunk's
        // pass writes only below its own end, so the entries in flight
        // are never overwritten before they are used
        int32_t ia = lane < prevL ? idx[lane] : INT_MAX;
        float va = lane < prevL ? val[lane] : 0.f;
        int32_t ia1 = 32 + lane < prevL ? idx[32 + lane] : INT_MAX;
        float va1 = 32 + lane < prevL ? val[32 + lane] : 0.f;
        for (int base = 0; base < prevL; base += 32) {
          const int a2 = base + 64 + lane;
          const int32_t ia2 = a2 < prevL ? idx[a2] : INT_MAX;
          const float va2 = a2 < prevL ? val[a2] : 0.f;
          const int a = base + lane;
          const bool in = a < prevL;
          const bool has_b = a + 1 < prevL;
          // the next entry: the lane above's, or the next chunk's first
          int32_t ib = __shfl_down_sync(0xffffffffu, ia, 1);
          float vb = __shfl_down_sync(0xffffffffu, va, 1);
          const int32_t ib1 = __shfl_sync(0xffffffffu, ia1, 0);
          const float vb1 = __shfl_sync(0xffffffffu, va1, 0);
          if (lane == 31) {
            ib = ib1;
            vb = vb1;
          }
          const int h = ia >> 1, hb = ib >> 1;
          int hp = __shfl_up_sync(0xffffffffu, h, 1);
          if (lane == 0) hp = carry_h;
          const bool keep = in && (a == 0 || h != hp) && h < lastframe;
          const bool merge = keep && has_b && hb == h;
          float sv = va;
          if (merge) sv = __fadd_rn(va, vb);
          sv = __fmul_rn(sv, 0.5f);  // == sv / 2 (exact scaling)
          const unsigned bal = __ballot_sync(0xffffffffu, keep);
          const bool stop = __any_sync(0xffffffffu, in && h >= lastframe);
          carry_h = __shfl_sync(0xffffffffu, h, 31);
          __syncwarp();
          if (keep) {
            const int o = out + __popc(bal & ((1u << lane) - 1u));
            idx[o] = h;
            val[o] = sv;
          }
          out += __popc(bal);
          __syncwarp();
          if (stop) break;
          ia = ia1;
          va = va1;
          ia1 = ia2;
          va1 = va2;
        }
        L = out;
        tail_sorted = tail_sorted && (L >= prevL || junction_ok);
      }
    }
    if (dead) {
      for (int c = lane; c < cnt; c += 32) {
        const size_t o = (size_t)(lv.first + c) * P + p;
        G2[o] = 0.f;
        IP[o] = 0.f;
        IF[o] = 0.f;
      }
      continue;
    }
    // every prefix entry is findable unless the reference searches a buffer
    // that is out of order
    const bool all_find = !ref || (tail_sorted && (L >= n0 || idx[L - 1] <= idx[L]));
    const int kmax = t0 + cnt - 1;
    const int nchain = 3 * cnt;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    // ring slots past the row end are never read (partners stop at L)
    uint64_t fmask = 0;
    fw_put(0, lane, L, fw_fetch(0, lane, L, n0, all_find, idx, val), ridx, rval, fmask);
    fw_put(32, lane, L, fw_fetch(32, lane, L, n0, all_find, idx, val), ridx, rval, fmask);
    for (int base = 0; base < L; base += 32) {
      // the tile after next, in flight while this one is processed
      const FwEntry nx = fw_fetch(base + 64, lane, L, n0, all_find, idx, val);
      __syncwarp();
      const int r = base + lane;
      const bool valid = r < L;
      const int nt = min(32, L - base);  // entries in this tile
      const int32_t src = valid ? ridx[r & 63] : 0;
      const float v = valid ? rval[r & 63] : 0.f;
      // partners: when the tile and its partners span fewer than FW_WIN
      // bins, through a per-warp bin array (one lookup per delay), else by
      // scanning the following entries
      const int32_t b0 = ridx[base & 63];
      const bool use_bins = ridx[(base + nt - 1) & 63] + kmax - b0 < FW_WIN;
      if (use_bins) {
        ((float4 *)bval)[lane] = make_float4(0.f, 0.f, 0.f, 0.f);  // FW_WIN = 128 bins
        __syncwarp();
        if (valid) bval[src - b0] = fw_findable(fmask, r) ? v : 0.f;
        const int q2 = base + 32 + lane;
        if (lane < kmax && q2 < L) {
          const int tb = ridx[q2 & 63] - b0;
          if (tb < FW_WIN) bval[tb] = fw_findable(fmask, q2) ? rval[q2 & 63] : 0.f;
        }
        __syncwarp();
      }
      // inside [kmax, lastframe - kmax) every IP and IF term of the tile is v:
      // the IP/IF chains then read one shared row
      const bool bulk = b0 >= kmax && ridx[(base + nt - 1) & 63] < lastframe - kmax;
      if (valid) {
        if (bulk) {
          vrow[lane] = v;
        } else {
          float *tp = terms + (size_t)cnt * FW_TSTRIDE + lane;
          float *tf = tp + (size_t)cnt * FW_TSTRIDE;
#pragma unroll
          for (int c = 0; c < FW_MAXC; c++) {
            if (c >= cnt) break;
            const int tau = t0 + c;
            tp[c * FW_TSTRIDE] = src < lastframe - tau ? v : 0.f;
            tf[c * FW_TSTRIDE] = (src >= tau && src < lastframe) ? v : 0.f;
          }
        }
        // a partner is a prefix entry, so it lies below lastframe and the
        // reference's src < lastframe - tau test holds for every pair found
        if (use_bins) {
          const float *bw = bval + (src + t0 - b0);  // + c <= src - b0 + kmax < FW_WIN
          float *tg = terms + lane;
          if ((cnt & 3) == 0) {  // e.g. every level of 8 delays: one test per 4 delays
#pragma unroll
            for (int c = 0; c < FW_MAXC; c += 4) {
              if (c >= cnt) break;
#pragma unroll
              for (int u = 0; u < 4; u++) tg[(c + u) * FW_TSTRIDE] = __fmul_rn(v, bw[c + u]);
            }
          } else {
#pragma unroll
            for (int c = 0; c < FW_MAXC; c++) {
              if (c >= cnt) break;
              tg[c * FW_TSTRIDE] = __fmul_rn(v, bw[c]);
            }
          }
        } else {
          for (int c = 0; c < cnt; c++) terms[(size_t)c * FW_TSTRIDE + lane] = 0.f;
          for (int k = t0 > 0 ? 1 : 0; k <= kmax; k++) {
            const int qk = r + k;
            if (qk >= L) break;
            const int d = ridx[qk & 63] - src;
            if (d > kmax) break;
            if (d >= t0 && fw_findable(fmask, qk))
              terms[(size_t)(d - t0) * FW_TSTRIDE + lane] = __fmul_rn(v, rval[qk & 63]);
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int ch = lane + 32 * j;
        if (ch < nchain) {
          const float *tr = (bulk && ch >= cnt) ? vrow : terms + (size_t)ch * FW_TSTRIDE;
          float a = acc[j];
          if (nt == 32) {
            const float4 *t4 = (const float4 *)tr;
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const float4 y = t4[i];
              a = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(a, y.x), y.y), y.z), y.w);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; i++) {
              if (i >= nt) break;
              a = __fadd_rn(a, tr[i]);
            }
          }
          acc[j] = a;
        }
      }
      __syncwarp();
      // the tile after next replaces this one in the ring
      fw_put(base + 64, lane, L, nx, ridx, rval, fmask);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int ch = lane + 32 * j;
      if (ch < nchain) {
        const int type = ch / cnt, c = ch - type * cnt;
        const int d = lv.first + c;
        const float den = ar.denom[d];
        const float x = den > 0.f ? __fdiv_rn(acc[j], den) : acc[j];
        float *dst = type == 0 ? G2 : (type == 1 ? IP : IF);
        dst[(size_t)d * P + p] = x;
      }
    }
  }
}

__global__ void __launch_bounds__(FW_WARPS * 32, 7)
k_mt_fwarp(const uint8_t *__restrict__ plan_g, const int32_t *__restrict__ flist,
           DevStats *__restrict__ stats, const int64_t *__restrict__ row_ptr,
           const int32_t *__restrict__ row_len, const int32_t *__restrict__ ev_frame,
           const float *__restrict__ ev_val, const float *__restrict__ fscale,
           int32_t *__restrict__ sc_frame, float *__restrict__ sc_val, float *__restrict__ G2,
           float *__restrict__ IP, float *__restrict__ IF) {
  extern __shared__ __align__(16) uint8_t fw_smem[];
  const McPlan *pl = (const McPlan *)plan_g;
  const McArrays ar = mc_arrays(plan_g, pl->D);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint8_t *wb = fw_smem + (size_t)w * fw_warp_bytes(pl->acc);
  const int nf = stats->nfloat;
  // pixels are handed out one per warp from a counter: rows differ in length
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(&stats->fnext, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= nf) break;
    const int p = flist[q];
    const int64_t b = row_ptr[p];
    fw_pixel(pl, ar, p, b, row_len[p], ev_frame, ev_val, fscale, sc_frame + b, sc_val + b, G2, IP,
             IF, wb);
    __syncwarp();
  }
  overlap_end();
}

// ------------------------------------------- caller rows, nothing allocated
//
// The row kernels for rows that come without classes, lengths or work lists
// (noalloc.cu): every kernel finds its own rows among the caller's row
// pointers and reads a row's class from its events, so no per-pixel array is
// needed.  A row is regular when its frames ascend strictly within [0, F) and
// its values are below 2^126 (the float-row kernel multiplies by 0 where the
// reference forms no product, and halving sums must not overflow); regular
// rows take the kernels of a series, the others the replay (noalloc.cu).
// status[1] collects the kinds of rows seen, so that a kernel without rows
// returns at once; status[2 ..] are the kernels' pixel counters.
// Measured (256 x 250 pixels, 3,000 frames, 2.8 M events): the call 4,530 us
// with one thread replaying each row from global memory, 300 us now, 202 of them
// in k_na_thread: 2,000 warps, less than one wave, 33 % issue.
constexpr int NA_GRAB = 4;  // pixels a warp takes at a time

// Row p: its first event and length; false (and the status bit) when it lies
// outside the events.
__device__ __forceinline__ bool na_row(const NaRows &v, int p, int64_t &b, int &n) {
  b = v.row_ptr[p];
  const int64_t e = v.row_ptr[p + 1];
  const bool ok = b >= 0 && e >= b && e <= v.events;
  n = ok ? (int)(e - b) : 0;
  return ok;
}

// Class of row [b, b + n), the same in every lane: NA_INT (n <= MT_LONG_CAP),
// NA_FLOAT or NA_IRREGULAR.
__device__ __forceinline__ int na_class(const NaRows &v, int64_t b, int n) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  bool reg = true, integ = v.F <= 65536 && n <= MT_LONG_CAP;
  int total = 0;  // a lane's share: at most 128 values of at most 4,096 while integ
  int last = -1;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const int f = i < n ? v.frame[b + i] : INT_MAX;
    const float x = i < n ? v.value[b + i] : 0.f;
    int prev = __shfl_up_sync(FULL, f, 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(FULL, f, 31);
    if (i < n) {
      reg = reg && f > prev && f < v.F && fabsf(x) < 0x1p126f;
      integ = integ && x == truncf(x) && fabsf(x) < 16777216.f;
      total += integ ? (int)fminf(fabsf(x), 4096.f) : 0;
    }
  }
  reg = __all_sync(FULL, reg);
  integ = __all_sync(FULL, integ);
  if (!reg) return NA_IRREGULAR;
  return integ && __reduce_add_sync(FULL, total) < 4096 ? NA_INT : NA_FLOAT;
}

// One thread per pixel: rows of up to CAP events, each lane loading and
// classifying its own; every other pixel gets zeros here, overwritten by the
// kernels below.
template <int CAP>
__global__ void __launch_bounds__(MT_WARPS * 32, 16) k_na_thread(NaRows v) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int scr = ((const McPlan *)v.plan)->scr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *wbase = (uint32_t *)smem + (size_t)warp * (CAP + scr) * 32;
  uint32_t *row = wbase + lane;
  const int64_t p0 = ((int64_t)blockIdx.x * MT_WARPS + warp) * 32;
  if (p0 >= v.P) return;
  const int p = (int)p0 + lane;
  int64_t b = 0;
  int n = 0, n0 = 0, kinds = 0;
  if (lane < v.P - p0 && !na_row(v, p, b, n)) atomicOr(v.status, 1);
  if (n > CAP) {
    kinds = n <= MT_WARP_CAP ? 1 : (n <= MT_MID_CAP ? 2 : (n <= MT_LONG_CAP ? 4 : NA_FLOAT));
  } else if (n > 0) {
    bool reg = true, integ = v.F <= 65536;
    int total = 0, prev = -1;
    for (int i0 = 0; i0 < n; i0 += 4) {
      int f[4];
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {  // the loads first, in flight together
        f[u] = i0 + u < n ? v.frame[b + i0 + u] : 0;
        x[u] = i0 + u < n ? v.value[b + i0 + u] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (i0 + u >= n) break;
        reg = reg && f[u] > prev && f[u] < v.F && fabsf(x[u]) < 0x1p126f;
        integ = integ && x[u] == truncf(x[u]) && fabsf(x[u]) < 16777216.f;
        total += integ ? (int)fminf(fabsf(x[u]), 4096.f) : 0;
        row[(i0 + u) * 32] = pk(f[u], __float2int_rn(x[u]));
        prev = f[u];
      }
    }
    if (reg && integ && total < 4096)
      n0 = n;
    else
      kinds = reg ? NA_FLOAT : NA_IRREGULAR;
  }
  kinds = __reduce_or_sync(0xffffffffu, (unsigned)kinds);
  if (lane == 0 && kinds) atomicOr(v.status + 1, kinds);
  __syncwarp();
  mt_thread_rows<CAP>(v.plan, p, n0, lane < v.P - p0, v.G2, v.IP, v.IF, wbase);
}

// The pixels of a warp, NA_GRAB at a time from the counter `next`: calls
// row(p, b, n) for those whose row has min_n < n <= max_n events.
template <class Row>
__device__ __forceinline__ void na_pixels(const NaRows &v, int32_t *next, int min_n, int max_n,
                                          Row row) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int groups = v.P / NA_GRAB + (v.P % NA_GRAB != 0);
  for (;;) {
    int g = 0;
    if (lane == 0) g = atomicAdd(next, 1);
    g = __shfl_sync(FULL, g, 0);
    if (g >= groups) break;
    const int p0 = g * NA_GRAB;
    int64_t b = 0;
    int n = 0;
    if (lane < min(NA_GRAB, v.P - p0)) na_row(v, p0 + lane, b, n);
    unsigned m = __ballot_sync(FULL, n > min_n && n <= max_n);
    while (m) {
      const int l = __ffs(m) - 1;
      m &= m - 1u;
      row(p0 + l, __shfl_sync(FULL, b, l), __shfl_sync(FULL, n, l));
      __syncwarp();
    }
  }
}

// One warp per pixel: integer rows of min_n < n <= cap events (kind bit
// `kind`); rows that are not get their kind recorded for the kernels after.
__global__ void __launch_bounds__(256)
k_na_warp(NaRows v, int32_t kind, int32_t min_n, int32_t cap, int32_t *next) {
  extern __shared__ __align__(16) uint8_t smem[];
  if (!(v.status[1] & kind)) return;
  const McPlan *pl = (const McPlan *)v.plan;
  const McArrays ar = mc_arrays(v.plan, pl->D);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ACC = max(pl->acc, pl->nlev);
  uint32_t *row = (uint32_t *)smem + (size_t)warp * (2 * cap + 32 * ACC);
  int32_t *S = (int32_t *)(row + cap);
  int32_t *acc = S + cap + lane;
  na_pixels(v, next, min_n, cap, [&](int p, int64_t b, int n) {
    const int c = na_class(v, b, n);
    if (c != NA_INT) {
      if (lane == 0) atomicOr(v.status + 1, c);
      return;
    }
    mt_warp_pixel(pl, ar, p, b, n, v.frame, v.value, v.G2, v.IP, v.IF, cap, row, S, acc);
  });
}

// One warp per pixel: float rows of any length.  It works on scratch copies
// of its rows; a descending row pointer (reported by the thread kernel) can
// make rows share scratch words, so the replay takes the float rows then.
__global__ void __launch_bounds__(FW_WARPS * 32, 7) k_na_fwarp(NaRows v, int32_t *next) {
  extern __shared__ __align__(16) uint8_t fw_smem[];
  if (v.status[0] || !(v.status[1] & NA_FLOAT)) return;
  const McPlan *pl = (const McPlan *)v.plan;
  const McArrays ar = mc_arrays(v.plan, pl->D);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint8_t *wb = fw_smem + (size_t)w * fw_warp_bytes(pl->acc);
  na_pixels(v, next, 0, INT_MAX, [&](int p, int64_t b, int n) {
    const int c = na_class(v, b, n);
    if (c == NA_IRREGULAR && lane == 0) atomicOr(v.status + 1, c);
    if (c != NA_FLOAT) return;
    fw_pixel(pl, ar, p, b, n, v.frame, v.value, nullptr, v.sc_frame + b, v.sc_val + b, v.G2, v.IP,
             v.IF, wb);
  });
}

// ---------------------------------------------- float rows, thread per pixel
//
// The same float sums with one pixel per thread, for rows of up to
// Series::float_cap events.  A warp takes 32 rows of about the same length
// (k_ft_sort) and keeps them in a scratch slot of its own in device memory
// (L2 for the usual rows), entry-interleaved: entry j of every lane is one
// coalesced 256-byte line of (bin, value) pairs, and the warp walks j in
// lockstep, the loads two entries ahead.  One pass per
// level forms the level's sums and, in the same step, writes the next level's
// compacted row in place, exactly as the reference leaves it (stale tail
// included).  A 32-bit mask of the bins before the current one (bit d - 1: an
// entry d bins back) tells which delays have a partner that ends in it, and a
// ring of the last 16 values in shared memory holds those partners, so that
// every delay's sum takes its products in the order of the reference (by the
// earlier entry, which is also the order of the later one).  The IF sums
// start at their first entry; the IP sums are one running sum, read off where
// it passes each delay's threshold.
// Bound by instruction issue (95 k warp instructions for 32 rows of 154 events,
// 56 % issue) and, where the slots outgrow the L2, by their traffic (27 % of DRAM
// throughput there).
// Measured against the warp-per-row kernel, which spends about 430 warp
// instructions on 32 entries of one row (float rows as a whole, ms):
//   dense  960^2 x 2,000 frames, 154 events a row   11.15 -> 4.53
//   dense  640^2 x 4,000, 294                        8.28 -> 4.58
//   flat   509 x 387 x 1,500, 58                     1.72 -> 0.72
//   flat   1024^2 x 1,000, 9                         5.45 -> 1.64
constexpr int FT_WARPS = 4;
constexpr int FT_AHEAD = 2;  // entries loaded ahead
constexpr int FT_PREF = 4;   // entries fetched into L1 ahead
constexpr double FT_MEAN_MAX = 2000.0;                   // longest mean row it is used for
constexpr double FT_PIX_FACTOR = 1.4e-5;                 // rows of up to this x pixels means
constexpr size_t FT_SLOT_BYTES = (size_t)3 << 30;        // most device memory of the slots
constexpr int FT_WIN_PIX = 4096;  // pixels sorted by row length together
constexpr int FT_TILE = 33;  // row of the 32 x 32 staging tile, padded
constexpr int FT_MAXC = 16;  // delays per level, and the ring's entries
constexpr int FT_MAXD = 16;  // largest delay in bins: the partners are among the last 16 entries

// Shared memory of a warp: the staging tiles while the rows are loaded, then
// the ring (each value at slots j & 15 and 16 + (j & 15), so that a partner's
// predecessors lie below it) and the IP sums of a level.
constexpr int FT_WORDS = 2 * 32 * FT_TILE;
static_assert(FT_WORDS >= 3 * FT_MAXC * 32, "the ring and the IP sums reuse the staging tiles");

struct FtState {
  uint2 *S;          // this lane's column of the slot: entry j at S[j * 32]
  float *ring, *ip;  // this lane's columns in shared memory
  int n0, m;         // events of the row, entries of the level's prefix
  bool tail_sorted;  // the buffer from m on ascends
  bool sorted;       // the whole buffer ascends
  int tail0;         // first bin of the tail

  __device__ __forceinline__ int lower_bound(int x) const {  // libstdc++'s halving
    int first = 0, len = n0;
    while (len > 0) {
      const int half = len >> 1;
      if ((int)S[(first + half) * 32].x < x) {
        first += half + 1;
        len -= half + 1;
      } else {
        len = half;
      }
    }
    return first;
  }
  // After the prefix of prev entries (last bin t_last) became `out` entries
  // (last bin o_last) in place.
  __device__ __forceinline__ void compacted(int prev, int t_last, int out, int o_last) {
    const bool junction_ok = prev >= n0 || t_last <= (int)S[prev * 32].x;
    m = out;
    tail_sorted = tail_sorted && (m >= prev || junction_ok);
    tail0 = m < n0 ? (int)S[m * 32].x : INT_MAX;
    sorted = m == 0 || (tail_sorted && o_last <= tail0);
  }
};

// One pass over the level's entries.  SUMS: the sums of cnt <= KM delays from
// tlo on (lf: the level's lastframe); CHECK: an entry counts as a partner only
// where the search over the whole buffer finds it; NEXT: the entries compacted
// for the next level (lfn: its lastframe).
template <int KM, bool SUMS, bool CHECK, bool NEXT>
__device__ __forceinline__ void ft_pass(FtState &f, int lf, int tlo, int cnt, int lfn,
                                        float (&g2)[KM], float (&iff)[KM]) {
  const unsigned FULL = 0xffffffffu;
  const int m = f.m, mmax = __reduce_max_sync(FULL, m);
  const int thi = tlo + cnt - 1;
  const uint32_t cmask = (1u << cnt) - 1u, gap = (1u << (tlo - 1)) - 1u;
  float run = 0.f;
  int kip = cnt - 1;       // IP sums of the delays above kip are read off
  uint32_t before = 0u;    // bins before the previous entry's
  int tp = 0;
  int out = 0, ph = -1;    // next level: entries written, pending bin and value
  float pv = 0.f;
  uint2 pf[FT_AHEAD];
#pragma unroll
  for (int u = 0; u < FT_AHEAD; u++) pf[u] = u < m ? f.S[u * 32] : make_uint2(0u, 0u);
  for (int j0 = 0; j0 < mmax; j0 += FT_AHEAD) {
#pragma unroll
    for (int u = 0; u < FT_AHEAD; u++) {
      const int j = j0 + u;
      const bool act = j < m;
      const int t = act ? (int)pf[u].x : tp + 1;  // idle lanes: no partner, +0 to the sums
      const float v = act ? __uint_as_float(pf[u].y) : 0.f;
      if (FT_PREF && j + FT_PREF < m)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(f.S + (j + FT_PREF) * 32));
      if (j + FT_AHEAD < m) pf[u] = f.S[(j + FT_AHEAD) * 32];
      if (SUMS) {
        const int step = t - tp;
        before = j == 0 || step > 32 ? 0u : ((before << 1 | 1u) << (step - 1));
        uint32_t w = act ? (before >> (tlo - 1)) & cmask : 0u;
        if (CHECK && w && !f.sorted && !(f.tail_sorted && t <= f.tail0) && f.lower_bound(t) != j)
          w = 0u;
        const float *pr = f.ring + (16 + ((j - 1 - __popc(before & gap)) & 15)) * 32;
#pragma unroll
        for (int k = 0; k < KM; k++) {
          if (w & (1u << k)) {
            g2[k] = __fadd_rn(g2[k], __fmul_rn(*pr, v));
            pr -= 32;
          }
        }
        f.ring[(j & 15) * 32] = v;
        f.ring[(16 + (j & 15)) * 32] = v;
        if (__all_sync(FULL, t >= thi)) {
#pragma unroll
          for (int k = 0; k < KM; k++) iff[k] = __fadd_rn(iff[k], v);
        } else {
#pragma unroll
          for (int k = 0; k < KM; k++)
            if (t >= tlo + k) iff[k] = __fadd_rn(iff[k], v);
        }
        while (act && kip >= 0 && t >= lf - tlo - kip) {
          f.ip[kip * 32] = run;
          kip--;
        }
        run = __fadd_rn(run, v);
      }
      if (NEXT && act) {
        const int h = t >> 1;
        if (h == ph) {
          pv = __fadd_rn(pv, v);  // distinct frames: pairs at most
        } else {
          if (ph >= 0 && ph < lfn) {
            f.S[out * 32] = make_uint2((uint32_t)ph, __float_as_uint(__fmul_rn(pv, 0.5f)));
            out++;
          }
          ph = h;
          pv = v;
        }
      }
      tp = act ? t : tp;
    }
  }
  if (SUMS)
    for (; kip >= 0; kip--) f.ip[kip * 32] = run;
  if (NEXT && m > 0) {
    int o_last = -1;
    if (ph < lfn) {
      f.S[out * 32] = make_uint2((uint32_t)ph, __float_as_uint(__fmul_rn(pv, 0.5f)));
      out++;
      o_last = ph;
    } else if (out > 0) {
      o_last = (int)f.S[(out - 1) * 32].x;
    }
    f.compacted(m, tp, out, o_last);
  }
}

template <int KM>
__device__ __forceinline__ void ft_run_level(FtState &f, const McPlan *pl, const McArrays &ar,
                                             int gi, bool ref, bool mine, float *out,
                                             int32_t Dp) {
  const McLevel L = pl->lv[gi];
  const int lfn = gi + 1 < pl->nlev ? pl->lv[gi + 1].lastframe : 0;  // 0: nothing is kept
  float g2[KM], iff[KM];
#pragma unroll
  for (int k = 0; k < KM; k++) g2[k] = iff[k] = 0.f;
  if (gi > 0 && ref && __any_sync(0xffffffffu, !f.sorted)) {
    // the search needs the buffer as it is: the sums first, then the compaction
    ft_pass<KM, true, true, false>(f, L.lastframe, L.tau_lo, L.count, 0, g2, iff);
    float none[1];
    ft_pass<1, false, false, true>(f, 0, 1, 1, lfn, none, none);
  } else {
    ft_pass<KM, true, false, true>(f, L.lastframe, L.tau_lo, L.count, lfn, g2, iff);
  }
  if (!mine) return;
  float ip[KM];
#pragma unroll
  for (int k = 0; k < KM; k++) {
    const float den = k < L.count ? ar.denom[L.first + k] : 0.f;
    ip[k] = k < L.count ? f.ip[k * 32] : 0.f;
    if (den > 0.f) {
      g2[k] = __fdiv_rn(g2[k], den);
      ip[k] = __fdiv_rn(ip[k], den);
      iff[k] = __fdiv_rn(iff[k], den);
    }
  }
  float *o = out + L.first;
  if (L.count == KM && KM % 4 == 0 && (L.first & 3) == 0) {  // the usual level: whole sectors
#pragma unroll
    for (int k = 0; k < KM; k += 4) {
      *(float4 *)(o + k) = make_float4(g2[k], g2[k + 1], g2[k + 2], g2[k + 3]);
      *(float4 *)(o + Dp + k) = make_float4(ip[k], ip[k + 1], ip[k + 2], ip[k + 3]);
      *(float4 *)(o + 2 * Dp + k) = make_float4(iff[k], iff[k + 1], iff[k + 2], iff[k + 3]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < KM; k++) {
      if (k >= L.count) break;
      o[k] = g2[k];
      o[Dp + k] = ip[k];
      o[2 * Dp + k] = iff[k];
    }
  }
}

// The float rows of every window of FT_WIN_PIX pixels, longest first, into the
// window's part of `list` (-1 past the last): a counting sort by length / 4.
// A warp lasts as long as its longest row, and neighbouring pixels' rows can
// differ tenfold (dense frames: each pixel's gain decides how much of the
// noise passes its threshold).  The window is small enough for the partly
// written output lines of the windows at work to stay in L2.
__global__ void __launch_bounds__(256)
k_ft_sort(int32_t P, const int32_t *__restrict__ row_len, const uint8_t *__restrict__ pclass,
          int32_t *__restrict__ list) {
  constexpr int NB = 1024, PER = FT_WIN_PIX / 256;
  __shared__ int32_t cnt[NB];
  __shared__ int32_t wsum[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * FT_WIN_PIX;
  for (int k = threadIdx.x; k < NB; k += 256) cnt[k] = 0;
  __syncthreads();
  int bin[PER];
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const int64_t p = base + i * 256 + threadIdx.x;
    bin[i] = -1;
    if (p < P && pclass[p] == PCLASS_FTHREAD) {
      bin[i] = max(0, NB - 1 - (row_len[p] >> 2));  // longest first
      atomicAdd(&cnt[bin[i]], 1);
    }
  }
  __syncthreads();
  // exclusive scan of the NB counters, 4 per thread
  int c[4], s = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    c[k] = s;
    s += cnt[threadIdx.x * 4 + k];
  }
  int x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  int off = x - s, total = 0;
  for (int k = 0; k < 8; k++) {
    if (k < w) off += wsum[k];
    total += wsum[k];
  }
#pragma unroll
  for (int k = 0; k < 4; k++) cnt[threadIdx.x * 4 + k] = off + c[k];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PER; i++)
    if (bin[i] >= 0) list[base + atomicAdd(&cnt[bin[i]], 1)] = (int32_t)(base + i * 256 + threadIdx.x);
  for (int k = total + threadIdx.x; k < FT_WIN_PIX; k += 256) list[base + k] = -1;
}

// 32 entries of the sorted lists at a time, handed out per warp from a
// counter; slots: `cap` lines of 32 entries for every warp of the grid.  KA /
// KB: the most delays of level 0 and of the others.
template <int KA, int KB>
__global__ void __launch_bounds__(FT_WARPS * 32, 5)
k_mt_fthread(const uint8_t *__restrict__ plan_g, int32_t cap, uint2 *__restrict__ slots,
             const int32_t *__restrict__ list, const int64_t *__restrict__ row_ptr,
             const int32_t *__restrict__ row_len, const int32_t *__restrict__ ev_frame,
             const float *__restrict__ ev_val, const float *__restrict__ fscale,
             DevStats *__restrict__ stats, int32_t Dp, float *__restrict__ stage) {
  overlap_begin();
  __shared__ float ft_sm[FT_WARPS][FT_WORDS];
  const unsigned FULL = 0xffffffffu;
  const McPlan *pl = (const McPlan *)plan_g;
  const McArrays ar = mc_arrays(plan_g, pl->D);
  const int P = pl->P, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool ref = pl->mode == XPCS_MODE_REFERENCE;
  const int groups = (P + FT_WIN_PIX - 1) / FT_WIN_PIX * (FT_WIN_PIX / 32);
  float *tf = ft_sm[w], *tv = tf + 32 * FT_TILE;
  FtState f;
  f.S = slots + ((size_t)blockIdx.x * FT_WARPS + w) * cap * 32 + lane;
  f.ring = ft_sm[w] + lane;
  f.ip = ft_sm[w] + 2 * FT_MAXC * 32 + lane;
  for (;;) {
    int g = 0;
    if (lane == 0) g = atomicAdd(&stats->ftnext, 1);
    g = __shfl_sync(FULL, g, 0);
    if (g >= groups) break;
    const int p = list[(size_t)g * 32 + lane];
    const bool mine = p >= 0;
    if (!__any_sync(FULL, mine)) continue;
    f.n0 = f.m = mine ? row_len[p] : 0;
    const int64_t b0 = mine ? row_ptr[p] : 0;
    // 32 entries of every row at a time: read coalesced row by row into the
    // padded tiles, then taken by the owning lanes
    const int nmax = __reduce_max_sync(FULL, f.n0);
    for (int e0 = 0; e0 < nmax; e0 += 32) {
      __syncwarp();
#pragma unroll 8
      for (int q = 0; q < 32; q++) {
        const int64_t bq = __shfl_sync(FULL, b0, q);
        const bool in = e0 + lane < __shfl_sync(FULL, f.n0, q);
        tf[q * FT_TILE + lane] = in ? __int_as_float(ev_frame[bq + e0 + lane]) : 0.f;
        tv[q * FT_TILE + lane] = in ? ev_val[bq + e0 + lane] : 0.f;
      }
      __syncwarp();
#pragma unroll 4
      for (int s = 0; s < 32; s++) {
        const uint32_t fr = __float_as_uint(tf[lane * FT_TILE + s]);
        float v = tv[lane * FT_TILE + s];
        if (e0 + s < f.n0) {
          // normalize_by_framesum: v / (frameSum[f] / mean) (main.cpp:330-333)
          if (fscale) v = __fdiv_rn(v, fscale[fr]);
          f.S[(e0 + s) * 32] = make_uint2(fr, __float_as_uint(v));
        }
      }
    }
    __syncwarp();
    f.tail_sorted = f.sorted = true;
    f.tail0 = INT_MAX;
    float *out = stage + (mine ? (size_t)p * 3 * Dp : 0);
    ft_run_level<KA>(f, pl, ar, 0, ref, mine, out, Dp);
    for (int gi = 1; gi < pl->nlev; gi++) ft_run_level<KB>(f, pl, ar, gi, ref, mine, out, Dp);
    __syncwarp();
  }
}

// The kernel's results [pixel][G2, IP, IF][Dp] into G2 / IP / IF [D][P]: 32 x
// 32 tiles through shared memory.  A warp's lanes hold pixels from all over
// their window, and storing each delay's 32 values where they belong took 1.8
// of 5.6 ms (960 x 960 pixels, 70 delays); with whole sectors per pixel and
// this pass over them (0.41 ms) all of it takes 4.5 ms.
__global__ void __launch_bounds__(256)
k_ft_out(int32_t P, int32_t D, int32_t Dp, const uint8_t *__restrict__ pclass,
         const float *__restrict__ stage, float *__restrict__ G2, float *__restrict__ IP,
         float *__restrict__ IF) {
  __shared__ float tile[8][32][33];  // a warp each: no barrier, all loads in flight
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p0 = blockIdx.x * 32;
  const bool mine = p0 + lane < P && pclass[p0 + lane] == PCLASS_FTHREAD;
  const unsigned rows = __ballot_sync(FULL, mine);
  if (!rows) return;
  const float *src = stage + (size_t)p0 * 3 * Dp + lane;
  for (int c0 = w * 32; c0 < 3 * Dp; c0 += 8 * 32) {
    const bool in = c0 + lane < 3 * Dp;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 32; q++)
      tile[w][q][lane] = in && (rows >> q & 1u) ? src[(size_t)q * 3 * Dp + c0] : 0.f;
    __syncwarp();
    int which = c0 / Dp, d = c0 - which * Dp;
#pragma unroll 8
    for (int r = 0; r < 32; r++) {
      if (mine && which < 3 && d < D) {
        float *o = which == 0 ? G2 : (which == 1 ? IP : IF);
        o[(size_t)d * P + p0 + lane] = tile[w][lane][r];
      }
      if (++d == Dp) {
        d = 0;
        which++;
      }
    }
  }
}

// Host-side plan: level groups of the delay schedule with the lastframe each
// sees and whether the reference compacts before it (corr.cpp:341-391).
std::vector<uint8_t> make_plan(const Series &s, int mode) {
  const int D = s.D;
  std::vector<uint8_t> buf(mc_plan_bytes(D), 0);
  McPlan *pl = (McPlan *)buf.data();
  int32_t *base = (int32_t *)(buf.data() + sizeof(McPlan));
  int32_t *tau_lvl = base;
  float *denom = (float *)(base + D);
  int32_t *tau_abs = base + 2 * D, *t_ip = base + 3 * D, *gi = base + 4 * D;
  float *rcp = (float *)(base + 5 * D);
  pl->P = s.P;
  pl->D = D;
  pl->F = s.F;
  pl->mode = mode;
  int ll = 0, lastframe = s.F, nlev = 0, acc = 1;
  for (int k = 0; k < D; k++) {
    int level = s.delays.level[k];
    bool newgroup = (k == 0) || level != s.delays.level[k - 1];
    int compact = 0;
    if (ll != level) {
      if (lastframe % 2) lastframe -= 1;
      lastframe = lastframe / 2;
      compact = 1;
    }
    // tau / pow(2, level) truncated to int (corr.cpp:393-394)
    int tau = level > 0 ? (int)(s.delays.tau[k] / std::pow(2.0, level)) : s.delays.tau[k];
    tau_lvl[k] = tau;
    tau_abs[k] = s.delays.tau[k];
    denom[k] = (lastframe - tau) > 0 ? (float)(lastframe - tau) : 0.f;
    rcp[k] = denom[k] > 0.f ? recip_rn((int32_t)(lastframe - tau)) : 0.f;
    t_ip[k] = (int32_t)std::max<int64_t>(0, (int64_t)(lastframe - tau) << level);
    if (newgroup) {
      if (nlev >= MAX_LEVELS) throw Error(XPCS_ERR_INVALID_ARGUMENT, "too many multi-tau levels");
      McLevel &L = pl->lv[nlev++];
      L.level = level;
      L.first = k;
      L.count = 0;
      L.lastframe = lastframe;
      L.tau_lo = tau;
      L.compact = compact;
      L.t_end = (int32_t)((int64_t)lastframe << level);
    }
    McLevel &L = pl->lv[nlev - 1];
    if (tau != L.tau_lo + L.count)
      throw Error(XPCS_ERR_INVALID_ARGUMENT, "non-consecutive delays within a level");
    L.count++;
    acc = std::max(acc, L.count);
    gi[k] = nlev - 1;
    ll = level;
  }
  pl->nlev = nlev;
  pl->acc = acc;
  pl->scr = std::max(std::max(acc, nlev), MT_MIN_SCR) + std::max(0, s.scr_extra);
  for (int k = 1; k < D; k++)
    if (t_ip[k] >= t_ip[k - 1] || tau_abs[k] <= tau_abs[k - 1])
      throw Error(XPCS_ERR_INVALID_ARGUMENT, "delay thresholds are not monotone");
  for (int g = 1; g < nlev; g++)
    if (pl->lv[g].t_end > pl->lv[g - 1].t_end)
      throw Error(XPCS_ERR_INVALID_ARGUMENT, "level end thresholds are not monotone");
  return buf;
}

size_t thread_smem(int scr, int cap) {
  return (size_t)MT_WARPS * (cap + scr) * 32 * sizeof(uint32_t);
}

using ThreadKernel = void (*)(const uint8_t *, const int64_t *, const int32_t *, const uint8_t *,
                              const int32_t *, const float *, float *, float *, float *);

ThreadKernel thread_kernel(int cap) {
  switch (cap) {
    case 32: return k_mt_thread<32>;
    case 48: return k_mt_thread<48>;
    case 64: return k_mt_thread<64>;
    case 80: return k_mt_thread<80>;
    case 112: return k_mt_thread<112>;
  }
  throw Error(XPCS_ERR_INVALID_ARGUMENT, "unsupported thread-kernel row capacity");
}
size_t warp_smem(int D, int acc, int cap, int warps) {
  return mc_plan_bytes(D) + (size_t)warps * (2 * cap + 32 * acc) * sizeof(int32_t);
}

// The kernels' row counters, before the first kernel that uses one.
void reset_counters(Series &s, cudaStream_t st) {
  constexpr size_t first = offsetof(DevStats, wnext), end = offsetof(DevStats, events);
  XG_CUDA(cudaMemsetAsync((char *)s.stats.p + first, 0, end - first, st));
}

// Blocks of k_mt_fthread, the slots within FT_SLOT_BYTES, and its scratch.
struct FtScratch {
  int blocks;
  size_t slots, list, out;  // bytes, pixels, floats
};
FtScratch ft_scratch(const Series &s, int32_t cap, int sms, int per_sm) {
  const size_t block_bytes = (size_t)FT_WARPS * 32 * cap * sizeof(uint2);
  per_sm = std::min(per_sm, (int)(FT_SLOT_BYTES / (block_bytes * (size_t)sms)));
  const int windows = (s.P + FT_WIN_PIX - 1) / FT_WIN_PIX;
  const int blocks = std::min(sms * std::max(1, per_sm), windows * (FT_WIN_PIX / 32 / FT_WARPS));
  return {blocks, blocks * block_bytes, (size_t)windows * FT_WIN_PIX,
          (size_t)s.P * 3 * ((s.D + 3) & ~3)};
}

// Given back: a captured batch graph that holds the addresses is stale with it.
void release_float_thread(Series &s, cudaStream_t st) {
  if (s.ft_slots.p || s.ft_list.p || s.ft_out.p) s.generation++;
  s.ft_slots.release(st);
  s.ft_list.release(st);
  s.ft_out.release(st);
}

// The scratch of k_mt_fthread, up to 3 GB of slots and as much as G2, IP and IF
// together; false where it is not to be had (the rows then go to the warp-per-row
// kernel, which needs none).  A captured graph allocates nothing.
bool reserve_float_thread(Series &s, cudaStream_t st, const FtScratch &f) {
  if (f.slots <= s.ft_slots.cap && f.list <= s.ft_list.cap && f.out <= s.ft_out.cap) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  XG_CUDA(cudaStreamIsCapturing(st, &cap));
  if (cap != cudaStreamCaptureStatusNone) return false;
  if (s.ft_slots.try_reserve(f.slots, st) && s.ft_list.try_reserve(f.list, st) &&
      s.ft_out.try_reserve(f.out, st))
    return true;
  release_float_thread(s, st);
  return false;
}

// The rows of the thread-per-pixel float kernel moved to the list of the
// warp-per-row one.
__global__ void k_ft_to_warps(int32_t P, const uint8_t *__restrict__ pclass,
                              int32_t *__restrict__ flist, DevStats *__restrict__ stats) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool mine = p < P && pclass[p] == PCLASS_FTHREAD;
  const unsigned m = __ballot_sync(0xffffffffu, mine);
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0 && m) {
    base = atomicAdd(&stats->nfloat, __popc(m));
    atomicSub(&stats->nfthread, __popc(m));
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  if (mine) flist[base + __popc(m & ((1u << lane) - 1u))] = (int32_t)p;
}

// The float rows of a series (flatfield, average, hot pixels, dense data,
// normalize_by_framesum) on st: the thread-per-pixel kernel's rows, and for the
// others the warp-per-row replay when the schedule allows it (beside the last
// rows of the kernel before: 8.68 -> 8.32 ms at 960 x 960 x 2,000 dense frames),
// else the thread-per-row one.
void launch_float_rows(Series &s, const McPlan &hp, cudaStream_t st, int sms) {
  const int P = s.P;
  size_t ne = s.raw_events > 0 ? (size_t)s.raw_events : 1;
  s.sc_frame.reserve(ne, st);
  s.sc_val.reserve(ne, st);
  int grid = std::max(1, std::min((P + 127) / 128, sms * 8));
  const float *fscale = nullptr;
  if (s.desc.normalize_by_framesum) {
    prepare_framesum_scale(s);
    fscale = s.d_fscale.p;
  }
  bool thread_rows = s.float_cap > 0;
  const int Dp = (s.D + 3) & ~3;  // padded delays of k_mt_fthread's staged results
  if (thread_rows) {
    const auto kernel = s.desc.delays_per_level <= 4 ? k_mt_fthread<8, 4> : k_mt_fthread<16, 8>;
    int per_sm = 0;
    XG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, FT_WARPS * 32, 0));
    const FtScratch f = ft_scratch(s, s.float_cap, sms, per_sm);
    thread_rows = reserve_float_thread(s, st, f);
    if (thread_rows) {
      k_ft_sort<<<(unsigned)(f.list / FT_WIN_PIX), 256, 0, st>>>(P, s.row_len.p, s.pclass.p,
                                                                s.ft_list.p);
      XG_CHECK_LAUNCH();
      kernel<<<f.blocks, FT_WARPS * 32, 0, st>>>(
          s.plan.p, s.float_cap, (uint2 *)s.ft_slots.p, s.ft_list.p, s.row_ptr.p, s.row_len.p,
          s.ev_frame.p, s.ev_val.p, fscale, s.stats.p, Dp, s.ft_out.p);
    } else {
      k_ft_to_warps<<<(P + 255) / 256, 256, 0, st>>>(P, s.pclass.p, s.flist.p, s.stats.p);
    }
    XG_CHECK_LAUNCH();
  }
  if (mt_float_rows_warp(hp)) {
    const size_t smf = FW_WARPS * fw_warp_bytes(hp.acc);
    allow_smem(k_mt_fwarp);
    int per_sm = 0;
    XG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mt_fwarp, FW_WARPS * 32,
                                                          smf));
    const int blocks = sms * std::max(1, per_sm);
    if (thread_rows) {
      launch_overlapped(k_mt_fwarp, blocks, FW_WARPS * 32, smf, st, s.plan.p, s.flist.p, s.stats.p,
                        s.row_ptr.p, s.row_len.p, s.ev_frame.p, s.ev_val.p, fscale, s.sc_frame.p,
                        s.sc_val.p, s.G2.p, s.IP.p, s.IF.p);
    } else {
      k_mt_fwarp<<<blocks, FW_WARPS * 32, smf, st>>>(
          s.plan.p, s.flist.p, s.stats.p, s.row_ptr.p, s.row_len.p, s.ev_frame.p, s.ev_val.p,
          fscale, s.sc_frame.p, s.sc_val.p, s.G2.p, s.IP.p, s.IF.p);
      XG_CHECK_LAUNCH();
    }
  } else {
    k_mt_float<<<grid, 128, 0, st>>>(s.plan.p, s.flist.p, s.stats.p, s.row_ptr.p, s.row_len.p,
                                     s.ev_frame.p, s.ev_val.p, fscale, s.sc_frame.p, s.sc_val.p,
                                     s.G2.p, s.IP.p, s.IF.p);
    XG_CHECK_LAUNCH();
  }
  if (thread_rows) {
    k_ft_out<<<(P + 31) / 32, 256, 0, st>>>(P, s.D, Dp, s.pclass.p, s.ft_out.p, s.G2.p, s.IP.p,
                                            s.IF.p);
    XG_CHECK_LAUNCH();
    // under a memory limit the scratch is the call's alone: what follows, and
    // other handles, have what they had without this kernel
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    XG_CUDA(cudaStreamIsCapturing(st, &cap));
    if (cap == cudaStreamCaptureStatusNone && dev_limited()) release_float_thread(s, st);
  }
}

}  // namespace

// The float nearest to 1/b (ties to even) for an integer b in [1, 2^24]:
// candidates around the double quotient compared by their exact residuals
// (g*b has at most 48 significant bits, so 1 - g*b is exact in double).
float recip_rn(int32_t b) {
  const float f = (float)(1.0 / (double)b);
  float best = f;
  double be = std::fabs(1.0 - (double)f * b);
  for (float g : {std::nextafter(f, 0.f), std::nextafter(f, 2.f * f)}) {
    const double e = std::fabs(1.0 - (double)g * b);
    uint32_t gb, bb;
    std::memcpy(&gb, &g, 4);
    std::memcpy(&bb, &best, 4);
    if (e < be || (e == be && (gb & 1u) == 0 && (bb & 1u) != 0)) {
      best = g;
      be = e;
    }
  }
  return best;
}

// Row capacity of the thread-per-pixel float kernel.  It serves series whose
// values are floats as a rule (flatfield, averaging, dense frames,
// normalize_by_framesum) with at most 16 delays a level.  Longer rows go to
// the warp-per-row kernel: one of them would keep a warp busy longer than the
// rest of the series takes.  Dense frames' rows differ most (the threshold
// passes much of some pixels' noise): at 960 x 960 x 2,000 frames the float
// rows take 6.2 / 5.6 / 5.1 / 4.5 / 4.5 ms with 2 / 3 / 4 / 6 / 9 times the
// mean; photon counting series do not depend on it (0.72 ms at 509 x 387 x
// 1,500 frames from 2 to 9 times the mean).  The kernel's time is at least the
// longest row's (about 1.1 us an event) and the other kernel's grows with all
// events (0.08 ns each), so the longest row is limited to a multiple of the
// mean that falls with the pixel count, and below 90,000 pixels the kernel is
// not used: at 320 x 320 dense pixels, rows of 736 events, 6 times the mean
// takes 6.0 ms, this rule 4.5 and the warp-per-row kernel alone 4.7.  Rows of
// 4,000 events on average gain nothing any more (320^2 x 60,000 frames).
int32_t mt_float_cap(const Series &s, double mean) {
  if (!(s.has_flat || s.desc.avg_frames > 1 || s.desc.dense || s.desc.normalize_by_framesum))
    return 0;
  const int dpl = s.desc.delays_per_level;
  if (s.D == 0 || dpl < 1 || 2 * dpl > FT_MAXC || mean > FT_MEAN_MAX) return 0;
  static_assert(FT_MAXC == FT_MAXD, "a level's largest delay is at most 2 dpl bins");
  const double factor = std::min(s.desc.dense ? 6.0 : 3.0, FT_PIX_FACTOR * s.P);
  return factor < 1.25 ? 0 : (int32_t)std::min<double>(s.F, factor * mean + 64.0);
}

size_t mt_float_bytes(const Series &s, int32_t float_cap, int sms) {
  if (float_cap <= 0) return 0;
  // as many blocks on an SM as their shared memory lets there be
  const FtScratch f =
      ft_scratch(s, float_cap, sms, (int)(SMEM_MAX / (sizeof(float) * FT_WARPS * FT_WORDS)));
  return f.slots + sizeof(int32_t) * f.list + sizeof(float) * f.out;
}

std::vector<uint8_t> prepare_multitau(Series &s, int mode) {
  cudaStream_t st = s.stream;
  // the plan depends on the series' shape and the mode only; it is uploaded
  // once per mode (a captured batch graph must not copy from host memory)
  std::vector<uint8_t> plan = make_plan(s, mode);
  const McPlan *hp = (const McPlan *)plan.data();
  if (s.plan_mode != mode || s.plan_scr != hp->scr) {
    s.plan.reserve(plan.size(), st);
    XG_CUDA(cudaMemcpyAsync(s.plan.p, plan.data(), plan.size(), cudaMemcpyHostToDevice, st));
    XG_CUDA(cudaStreamSynchronize(st));
    s.plan_mode = mode;
    s.plan_scr = hp->scr;
  }
  const size_t nD = (size_t)s.D * s.P;
  s.G2.reserve(nD ? nD : 1, st);
  s.IP.reserve(nD ? nD : 1, st);
  s.IF.reserve(nD ? nD : 1, st);
  return plan;
}

void run_multitau(Series &s, int mode) {
  cudaStream_t st = s.stream;
  const int D = s.D, P = s.P;
  const std::vector<uint8_t> plan = prepare_multitau(s, mode);
  const McPlan *hp = (const McPlan *)plan.data();
  if (D == 0 || P == 0) return;
  const int scr = std::max(hp->acc, hp->nlev);
  const ThreadKernel ktt = thread_kernel(s.thread_cap);
  const size_t smt = thread_smem(hp->scr, s.thread_cap),
               smw = warp_smem(D, scr, MT_WARP_CAP, WP_WARPS);
  const size_t smm = warp_smem(D, scr, MT_MID_CAP, MID_WARPS);
  const size_t sml = warp_smem(D, scr, MT_LONG_CAP, LONG_WARPS);
  if (smt > SMEM_MAX || smw > SMEM_MAX || smm > SMEM_MAX || sml > SMEM_MAX)
    throw Error(XPCS_ERR_INVALID_ARGUMENT, "delay schedule too large for the multi-tau kernels");
  allow_smem(ktt);
  allow_smem(k_mt_warp);
  int sms = 0;
  XG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.device));
  XG_CUDA(cudaEventRecord(s.ev[4], st));
  reset_counters(s, st);
  DevStats *ds = s.stats.p;
  // long rows in two launches over one list: up to 1024 events with 4 warps per
  // block, longer ones, first, with 2 warps per block; rows of 81-256 events;
  // the thread kernel's pixels
  k_mt_warp<<<sms * (int)(SMEM_MAX / sml), LONG_WARPS * 32, sml, st>>>(
      s.plan.p, s.llist.p, &ds->nlong, MT_MID_CAP, MT_LONG_CAP, s.row_ptr.p, s.row_len.p,
      s.ev_frame.p, s.ev_val.p, s.G2.p, s.IP.p, s.IF.p, &ds->wnext[0]);
  XG_CHECK_LAUNCH();
  launch_overlapped(k_mt_warp, sms * (int)(SMEM_MAX / smm), MID_WARPS * 32, smm, st,
                    s.plan.p, s.llist.p, &ds->nlong, MT_WARP_CAP, MT_MID_CAP, s.row_ptr.p,
                    s.row_len.p, s.ev_frame.p, s.ev_val.p, s.G2.p, s.IP.p, s.IF.p,
                    &ds->wnext[1]);
  launch_overlapped(k_mt_warp, sms * (int)(SMEM_MAX / smw), WP_WARPS * 32, smw, st,
                    s.plan.p, s.wlist.p, &ds->nwarp, 0, MT_WARP_CAP, s.row_ptr.p, s.row_len.p,
                    s.ev_frame.p, s.ev_val.p, s.G2.p, s.IP.p, s.IF.p, &ds->wnext[2]);
  const int per_block = MT_WARPS * 32;
  launch_overlapped(ktt, (P + per_block - 1) / per_block, per_block, smt, st, s.plan.p,
                    s.row_ptr.p, s.row_len.p, s.pclass.p, s.ev_frame.p, s.ev_val.p, s.G2.p,
                    s.IP.p, s.IF.p);
  XG_CUDA(cudaEventRecord(s.ev[5], st));
  launch_float_rows(s, *hp, st, sms);
  XG_CUDA(cudaEventRecord(s.ev[6], st));
}

void mt_queue_build(const std::vector<Series *> &ss, MtQueue &q, cudaStream_t st) {
  std::vector<MtQueueMember> tab;
  q.cap_first.assign(MT_THREAD_NCAPS, 0);
  q.cap_count.assign(MT_THREAD_NCAPS, 0);
  q.cap_groups.assign(MT_THREAD_NCAPS, 0);
  q.scr_max = q.acc_max = 1;
  for (int c = 0; c < MT_THREAD_NCAPS; c++) {
    q.cap_first[c] = (int32_t)tab.size();
    int32_t groups = 0;
    for (Series *sp : ss) {
      Series &s = *sp;
      if (s.thread_cap != MT_THREAD_CAPS[c] || s.D == 0 || s.P == 0) continue;
      const McPlan hp = *(const McPlan *)make_plan(s, s.plan_mode).data();
      q.scr_max = std::max(q.scr_max, hp.scr);
      q.acc_max = std::max(q.acc_max, std::max(hp.acc, hp.nlev));
      MtQueueMember m{s.plan.p, s.row_ptr.p, s.row_len.p, s.pclass.p, s.ev_frame.p, s.ev_val.p,
                      s.G2.p, s.IP.p, s.IF.p, s.wlist.p, s.llist.p, s.stats.p, groups,
                      (s.P + 31) / 32};
      groups += m.groups;
      tab.push_back(m);
    }
    q.cap_count[c] = (int32_t)tab.size() - q.cap_first[c];
    q.cap_groups[c] = groups;
  }
  q.tab.reserve(std::max<size_t>(tab.size(), 1), st);
  if (!tab.empty())
    XG_CUDA(cudaMemcpyAsync(q.tab.p, tab.data(), sizeof(MtQueueMember) * tab.size(),
                            cudaMemcpyHostToDevice, st));
  q.next.reserve(MT_THREAD_NCAPS + 3, st);
  XG_CUDA(cudaStreamSynchronize(st));
}

void mt_queue_run(const std::vector<Series *> &ss, MtQueue &q, cudaStream_t st) {
  const int32_t n = q.cap_first.empty() ? 0 : q.cap_first.back() + q.cap_count.back();
  if (n == 0) return;
  int dev = 0, sms = 0;
  XG_CUDA(cudaGetDevice(&dev));
  XG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  XG_CUDA(cudaMemsetAsync(q.next.p, 0, sizeof(int32_t) * (MT_THREAD_NCAPS + 3), st));
  // the warp-per-pixel tiers over every member, longest rows first: rows of
  // 1025-4096, 257-1024 and 81-256 events; then the thread kernels
  const int tiers[3][4] = {{1, MT_MID_CAP, MT_LONG_CAP, LONG_WARPS},
                           {1, MT_WARP_CAP, MT_MID_CAP, MID_WARPS},
                           {0, 0, MT_WARP_CAP, WP_WARPS}};
  const size_t pref_bytes = mc_align16(sizeof(int32_t) * (size_t)(n + 1));
  for (int t = 0; t < 3; t++) {
    const int cap = tiers[t][2], warps = tiers[t][3];
    const size_t sm = pref_bytes + (size_t)warps * (2 * cap + 32 * q.acc_max) * sizeof(int32_t);
    if (sm > SMEM_MAX)
      throw Error(XPCS_ERR_INVALID_ARGUMENT, "delay schedule too large for the multi-tau kernels");
    allow_smem(k_mt_warp_queue);
    int per_sm = 0;
    XG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mt_warp_queue, warps * 32,
                                                          sm));
    const int grid = sms * std::max(1, per_sm);
    int32_t *next = q.next.p + MT_THREAD_NCAPS + t;
    if (t == 0) {
      k_mt_warp_queue<<<grid, warps * 32, sm, st>>>(q.tab.p, n, tiers[t][0], tiers[t][1], cap,
                                                    q.acc_max, next);
      XG_CHECK_LAUNCH();
    } else {
      launch_overlapped(k_mt_warp_queue, grid, warps * 32, sm, st, q.tab.p, n, tiers[t][0],
                        tiers[t][1], cap, q.acc_max, next);
    }
  }
  using QueueKernel = void (*)(const MtQueueMember *, int32_t, int32_t, int32_t, int32_t *);
  const QueueKernel kq[MT_THREAD_NCAPS] = {k_mt_thread_queue<32>, k_mt_thread_queue<48>,
                                           k_mt_thread_queue<64>, k_mt_thread_queue<80>,
                                           k_mt_thread_queue<112>};
  for (int c = 0; c < MT_THREAD_NCAPS; c++) {
    if (!q.cap_count[c]) continue;
    const size_t smt = thread_smem(q.scr_max, MT_THREAD_CAPS[c]);
    if (smt > SMEM_MAX)
      throw Error(XPCS_ERR_INVALID_ARGUMENT, "delay schedule too large for the multi-tau kernels");
    allow_smem(kq[c]);
    int per_sm = 0;
    XG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kq[c], MT_WARPS * 32, smt));
    const int blocks = std::min(sms * std::max(1, per_sm), (q.cap_groups[c] + MT_WARPS - 1) /
                                                               MT_WARPS);
    launch_overlapped(kq[c], std::max(1, blocks), MT_WARPS * 32, smt, st,
                      q.tab.p + q.cap_first[c], q.cap_count[c], q.cap_groups[c], q.scr_max,
                      q.next.p + c);
  }
  for (Series *sp : ss) {  // float rows, member by member (none in integer data)
    Series &s = *sp;
    if (s.D == 0 || s.P == 0) continue;
    const McPlan hp = *(const McPlan *)make_plan(s, s.plan_mode).data();
    reset_counters(s, st);
    launch_float_rows(s, hp, st, sms);
  }
}

// Loads the kernels of mt_noalloc_rows on the current device and lifts their
// shared-memory limit, so that later calls find them in place.
cudaError_t mt_noalloc_setup() {
  const void *k[] = {(const void *)k_na_thread<32>, (const void *)k_na_thread<80>,
                     (const void *)k_na_warp, (const void *)k_na_fwarp};
  for (const void *f : k) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, f);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)SMEM_MAX - (int)a.sharedSizeBytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Whether the row kernels take the schedule: shared memory, at most 32 delays
// a level (the warp kernels' lanes), consecutive delays and monotone
// thresholds, as make_plan requires.
bool mt_noalloc_supported(const McPlan &hp, const McArrays &ar) {
  const int scr = std::max(hp.acc, hp.nlev);
  if (hp.D <= 0 || hp.P > (1 << 30) || hp.acc > 32 || thread_smem(hp.scr, 80) > SMEM_MAX ||
      warp_smem(0, scr, MT_WARP_CAP, WP_WARPS) > SMEM_MAX ||
      warp_smem(0, scr, MT_MID_CAP, MID_WARPS) > SMEM_MAX ||
      warp_smem(0, scr, MT_LONG_CAP, LONG_WARPS) > SMEM_MAX)
    return false;
  for (int k = 1; k < hp.D; k++)
    if (ar.t_ip[k] >= ar.t_ip[k - 1] || ar.tau_abs[k] <= ar.tau_abs[k - 1]) return false;
  for (int g = 0; g < hp.nlev; g++) {
    const McLevel &L = hp.lv[g];
    if (g > 0 && L.t_end > hp.lv[g - 1].t_end) return false;
    for (int k = 0; k < L.count; k++)
      if (ar.tau_lvl[L.first + k] != L.tau_lo + k) return false;
  }
  return true;
}

// Whether float rows go to the warp-per-row kernel (else the replay).
bool mt_float_rows_warp(const McPlan &hp) {
  int kmax = 0;
  for (int g = 0; g < hp.nlev; g++) kmax = std::max(kmax, hp.lv[g].tau_lo + hp.lv[g].count - 1);
  return kmax <= FW_MAXC && hp.acc <= FW_MAXC;
}

// Enqueues the row kernels over the caller's rows: outputs of every regular
// row (and zeros for the others); status[1] then holds the kinds of rows left.
cudaError_t mt_noalloc_rows(const McPlan &hp, const NaRows &v, int sms, cudaStream_t st) {
  const int scr = std::max(hp.acc, hp.nlev);
  const unsigned blocks = (unsigned)(((int64_t)v.P + MT_WARPS * 32 - 1) / (MT_WARPS * 32));
  // rows of about 1.5 times the mean fit the thread kernel (default_knobs has
  // more steps; two keep the kernels loaded at set-up few)
  const int cap = 1.5 * (double)v.events <= 32.0 * (double)v.P ? 32 : 80;
  if (cap == 32)
    k_na_thread<32><<<blocks, MT_WARPS * 32, thread_smem(hp.scr, 32), st>>>(v);
  else
    k_na_thread<80><<<blocks, MT_WARPS * 32, thread_smem(hp.scr, 80), st>>>(v);
  const int tiers[3][3] = {{cap, MT_WARP_CAP, WP_WARPS},
                           {MT_WARP_CAP, MT_MID_CAP, MID_WARPS},
                           {MT_MID_CAP, MT_LONG_CAP, LONG_WARPS}};
  for (int t = 0; t < 3; t++) {
    const size_t sm = warp_smem(0, scr, tiers[t][1], tiers[t][2]);
    k_na_warp<<<sms * std::max(1, (int)(SMEM_MAX / sm)), tiers[t][2] * 32, sm, st>>>(
        v, 1 << t, tiers[t][0], tiers[t][1], v.status + 2 + t);
  }
  if (mt_float_rows_warp(hp))
    k_na_fwarp<<<sms * 7, FW_WARPS * 32, FW_WARPS * fw_warp_bytes(hp.acc), st>>>(v, v.status + 5);
  return cudaGetLastError();
}

}  // namespace xg
