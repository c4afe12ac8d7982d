// F3: two-time correlation C2T(t1, t2) per q bin, with the reference's
// smoothing and its one-time reductions g2full / g2partials.
//
// Replaces Corr::twotime (src/xpcs/corr.cpp:560-924) with SmoothingStaticMap /
// SmoothingSymmetric (:433-547) and ComputeSG* (:1166-1305).  REFERENCE mode
// reproduces the reference's float32 operations in its order:
//   - the pixels of the processed q bins are rows in mapping order (q, static
//     bin, pixel), as event lists (photon counting) or as a dense matrix
//     V [rows][F], zero where a pixel has no event;
//   - sg[g][f] = the float sum over the rows of smoothing group g (a static
//     bin, or a q bin for the symmetric method) in mapping order, / pixels;
//     with the average filter, the float mean over frames;
//   - every event value is divided by its sg;
//   - C_q[f0][f1] (f0 <= f1) = the float sum over the q bin's rows, in
//     mapping order (ascending pixel index with frame threading), of
//     v(f0) * v(f1) over pairs of events, then / pixels: one separate multiply
//     and add per pair (no fused multiply-add), in row order, products with a
//     missing event skipped as the reference never forms them.  Event lists:
//     a warp per column f1 walks the column's events in row order
//     (k_tt_gram_events); dense rows: a tiled CUDA-core Gram whose reduction
//     runs over the rows in order (k_tt_gram);
//   - g2full[ff] = the float mean of diagonal ff in order; g2partials[ff][w]
//     the float sum of window w (`window` entries) of diagonal ff / window.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <utility>

#include "xpcs_internal.h"

namespace xg {
namespace {

constexpr int TT_TILE = 64;  // Gram tile (frames x frames)
constexpr int TT_KC = 32;    // rows per shared-memory chunk

__global__ void k_tt_scatter(int32_t R, int32_t F, const int32_t *__restrict__ row_pix,
                             const int64_t *__restrict__ row_ptr,
                             const int32_t *__restrict__ row_len,
                             const int32_t *__restrict__ ev_frame,
                             const float *__restrict__ ev_val, float *__restrict__ V) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const int p = row_pix[r];
  const int64_t b = row_ptr[p];
  const int n = row_len[p];
  for (int i = 0; i < n; i++) {
    const int f = ev_frame[b + i];
    if (f >= 0 && f < F) V[(size_t)r * F + f] = ev_val[b + i];
  }
}

// sg[g][f]: float sum over the group's rows in order, / pixels
__global__ void k_tt_sg(int32_t G, int32_t F, const int32_t *__restrict__ grp_ptr,
                        const float *__restrict__ V, float *__restrict__ sg) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x, g = blockIdx.y;
  if (f >= F || g >= G) return;
  float acc = 0.f;
  for (int r = grp_ptr[g]; r < grp_ptr[g + 1]; r++) acc = __fadd_rn(acc, V[(size_t)r * F + f]);
  sg[(size_t)g * F + f] = __fdiv_rn(acc, (float)(grp_ptr[g + 1] - grp_ptr[g]));
}

__global__ void k_tt_sg_avg(int32_t G, int32_t F, const float *__restrict__ sg,
                            float *__restrict__ sga) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G) return;
  float acc = 0.f;
  for (int f = 0; f < F; f++) acc = __fadd_rn(acc, sg[(size_t)g * F + f]);
  sga[g] = __fdiv_rn(acc, (float)F);
}

__global__ void k_tt_smooth(int32_t R, int32_t F, int32_t average,
                            const int32_t *__restrict__ row_grp, const float *__restrict__ sg,
                            float *__restrict__ V) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)R * F) return;
  const int r = (int)(i / F), f = (int)(i % F);
  const float v = V[i];
  if (v == 0.f) return;  // no event
  const int g = row_grp[r];
  V[i] = __fdiv_rn(v, average ? sg[g] : sg[(size_t)g * F + f]);
}

// One block per upper-triangle 64x64 tile of one q bin; 256 threads x 4x4 cells.
__global__ void __launch_bounds__(256)
k_tt_gram(int32_t F, int32_t nrows, const int32_t *__restrict__ order,
          const float *__restrict__ V, float *__restrict__ C) {
  __shared__ float As[TT_KC][TT_TILE];
  __shared__ float Bs[TT_KC][TT_TILE];
  // linear block id -> (bi <= bj)
  const int T = (F + TT_TILE - 1) / TT_TILE;
  int id = blockIdx.x, bi = 0;
  while (id >= T - bi) {
    id -= T - bi;
    bi++;
  }
  const int bj = bi + id;
  const int f0 = bi * TT_TILE, f1 = bj * TT_TILE;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < nrows; k0 += TT_KC) {
    for (int e = threadIdx.x; e < TT_KC * TT_TILE; e += 256) {
      const int kk = e / TT_TILE, c = e % TT_TILE;
      const bool in = k0 + kk < nrows;
      const size_t row = in ? (size_t)order[k0 + kk] * F : 0;
      As[kk][c] = (in && f0 + c < F) ? V[row + f0 + c] : 0.f;
      Bs[kk][c] = (in && f1 + c < F) ? V[row + f1 + c] : 0.f;
    }
    __syncthreads();
    const int kn = min(TT_KC, nrows - k0);
    for (int kk = 0; kk < kn; kk++) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float pr = __fmul_rn(a[i], b[j]);
          acc[i][j] = (a[i] != 0.f && b[j] != 0.f) ? __fadd_rn(acc[i][j], pr) : acc[i][j];
        }
    }
    __syncthreads();
  }
  const float den = (float)nrows;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int r = f0 + ty * 4 + i, c = f1 + tx * 4 + j;
      if (r < F && c < F && r <= c) C[(size_t)r * F + c] = __fdiv_rn(acc[i][j], den);
    }
}

// ------------------------------------------------------------ event lists
//
// Smoothing group of every row.
__global__ void k_tt_groups(int32_t R, int32_t G, const int32_t *__restrict__ grp_ptr,
                            int32_t *__restrict__ row_grp) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  int lo = 0, hi = G - 1;  // the last group that starts at or before r
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (grp_ptr[mid] <= r) lo = mid;
    else hi = mid - 1;
  }
  row_grp[r] = lo;
}

// The Gram of sparse rows: of the F (F + 1) / 2 products of a row only those
// of its events exist, and a column f1 of C needs, in row order, the rows
// with an event at f1 and each one's earlier events.  The rows' events are
// sorted by (q, frame), stably from row order, which gives every column's
// rows in the order its sums take them.

// Events of row order[j] (order null: row j) in build order, and the rows' ordered
// pairs of events, sum n (n - 1).
__global__ void __launch_bounds__(256)
k_tt_lens(int32_t R, const int32_t *__restrict__ order, const int32_t *__restrict__ row_pix,
          const int32_t *__restrict__ row_len, int32_t *__restrict__ len,
          unsigned long long *__restrict__ pairs) {
  __shared__ unsigned long long s_pairs[8];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = j < R ? row_len[row_pix[order ? order[j] : j]] : 0;
  if (j < R) len[j] = n;
  unsigned long long x = (unsigned long long)n * (unsigned)max(n - 1, 0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if ((threadIdx.x & 31) == 0) s_pairs[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) x += s_pairs[w];
    if (x) atomicAdd(pairs, x);
  }
}

// One warp per row in build order: (key = q F + frame, a = row, b = the
// event's position in its row).
__global__ void k_tt_build(int32_t R, int32_t F, int32_t Q, const int32_t *__restrict__ order,
                           const int32_t *__restrict__ q_ptr, const int32_t *__restrict__ row_pix,
                           const int64_t *__restrict__ row_ptr,
                           const int32_t *__restrict__ row_len,
                           const int32_t *__restrict__ ev_frame, const int64_t *__restrict__ cpos,
                           uint32_t *__restrict__ key, int32_t *__restrict__ a,
                           float *__restrict__ b) {
  const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= R) return;
  const int r = order ? order[j] : (int)j;
  int q = 0, hi = Q - 1;  // the last q bin whose rows start at or before r
  while (q < hi) {
    const int mid = (q + hi + 1) >> 1;
    if (q_ptr[mid] <= r) q = mid;
    else hi = mid - 1;
  }
  const int p = row_pix[r], n = row_len[p];
  const int64_t src = row_ptr[p], dst = cpos[j];
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    key[dst + i] = (uint32_t)q * (uint32_t)F + (uint32_t)ev_frame[src + i];
    a[dst + i] = r;
    b[dst + i] = __int_as_float(i);
  }
}

// col_ptr[c] = first event of column c = q F + frame
__global__ void k_tt_cols(int64_t ncol, int64_t n, const uint32_t *__restrict__ key,
                          int64_t *__restrict__ col_ptr) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ncol) return;
  int64_t first = 0, len = n;
  while (len > 0) {
    const int64_t h = len >> 1;
    if (key[first + h] < (uint64_t)c) {
      first += h + 1;
      len -= h + 1;
    } else {
      len = h;
    }
  }
  col_ptr[c] = first;
}

// sg[g][f] as k_tt_sg forms it (a row without an event at f adds 0): one warp
// per (group, frame) over the column's events of the group's rows, in row
// order (the lists sorted from mapping order).
__global__ void k_tt_sg_events(int32_t F, const int32_t *__restrict__ grp_ptr,
                               const int32_t *__restrict__ grp_q,
                               const int64_t *__restrict__ col_ptr, const int32_t *__restrict__ a,
                               const float *__restrict__ b, const int32_t *__restrict__ row_pix,
                               const int64_t *__restrict__ row_ptr,
                               const float *__restrict__ ev_val, float *__restrict__ sg) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int f = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), g = blockIdx.y;
  if (f >= F) return;
  const int r0 = grp_ptr[g], r1 = grp_ptr[g + 1];
  const int64_t c = (int64_t)grp_q[g] * F + f, end = col_ptr[c + 1];
  int64_t lo = col_ptr[c], len = end - lo;
  while (len > 0) {  // the group's first row in the column
    const int64_t h = len >> 1;
    if (a[lo + h] < r0) {
      lo += h + 1;
      len -= h + 1;
    } else {
      len = h;
    }
  }
  float acc = 0.f;
  for (int64_t e0 = lo;; e0 += 32) {
    const int64_t e = e0 + lane;
    const int r = e < end ? a[e] : r1;
    const bool in = r < r1;
    const float v = in ? ev_val[row_ptr[row_pix[r]] + __float_as_int(b[e])] : 0.f;
    const int n = __popc(__ballot_sync(FULL, in));
    for (int k = 0; k < n; k++) acc = __fadd_rn(acc, __shfl_sync(FULL, v, k));
    if (n < 32) break;
  }
  if (lane == 0) sg[(size_t)g * F + f] = __fdiv_rn(acc, (float)(r1 - r0));
}

// Smoothed values of the rows' events, beside their frames (one warp per row).
__global__ void k_tt_smooth_events(int32_t R, int32_t F, int32_t average,
                                   const int32_t *__restrict__ row_pix,
                                   const int32_t *__restrict__ row_grp,
                                   const int64_t *__restrict__ row_ptr,
                                   const int32_t *__restrict__ row_len,
                                   const int32_t *__restrict__ ev_frame,
                                   const float *__restrict__ ev_val, const float *__restrict__ sg,
                                   float *__restrict__ sv) {
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= R) return;
  const int p = row_pix[r], n = row_len[p], g = row_grp[r];
  const int64_t base = row_ptr[p];
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    const float v = ev_val[base + i];
    sv[base + i] =
        v == 0.f ? v : __fdiv_rn(v, average ? sg[g] : sg[(size_t)g * F + ev_frame[base + i]]);
  }
}

__device__ __forceinline__ void tt_add(float &acc, float x, float y) {
  acc = __fadd_rn(acc, __fmul_rn(x, y));
}
__device__ __forceinline__ void tt_add(int32_t &acc, int32_t x, int32_t y) { acc += x * y; }
__device__ __forceinline__ void tt_value(float v, float &x) { x = v; }
__device__ __forceinline__ void tt_value(float v, int32_t &x) { x = __float2int_rn(v); }

// The events [lo, hi) of column f1, in row order, by one warp: each one's row
// contributes v(f0) v(f1) to acc[f0] for its events up to f1, one f0 per lane,
// so no two lanes of a step share a sum and every sum takes its rows in order.
// A lane each looks up 32 events' rows at a time, and the next event's first
// 32 row entries are loaded while the current one's are added: the steps'
// latency bounds it.
template <class T>
__device__ __forceinline__ void tt_column(int64_t lo, int64_t hi, const int32_t *__restrict__ a,
                                          const float *__restrict__ b,
                                          const int32_t *__restrict__ row_pix,
                                          const int64_t *__restrict__ row_ptr,
                                          const int32_t *__restrict__ ev_frame,
                                          const float *__restrict__ val, T *acc) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int64_t e0 = lo; e0 < hi; e0 += 32) {
    const int64_t e = e0 + lane;
    int64_t my_base = 0;
    int my_i = -1;  // position of the event in its row: entries 0 .. i reach up to f1
    T my_v = 0;
    if (e < hi) {
      my_base = row_ptr[row_pix[a[e]]];
      my_i = __float_as_int(b[e]);
      tt_value(val[my_base + my_i], my_v);
    }
    const int n = (int)min((int64_t)32, hi - e0);
    int64_t base = __shfl_sync(FULL, my_base, 0);
    int i = __shfl_sync(FULL, my_i, 0);
    int f = lane <= i ? ev_frame[base + lane] : 0;
    float v = lane <= i ? val[base + lane] : 0.f;
    for (int k = 0; k < n; k++) {
      const int64_t bk = base;
      const int ik = i, fk = f;
      T vk;
      tt_value(v, vk);
      const T v1 = __shfl_sync(FULL, my_v, k);
      const int nk = min(k + 1, 31);
      base = __shfl_sync(FULL, my_base, nk);
      i = k + 1 < n ? __shfl_sync(FULL, my_i, nk) : -1;
      f = lane <= i ? ev_frame[base + lane] : 0;
      v = lane <= i ? val[base + lane] : 0.f;
      if (v1 == 0) continue;  // no event (a smoothed value of 0 forms no product)
      if (vk != 0) tt_add(acc[fk], vk, v1);
      for (int j = lane + 32; j <= ik; j += 32) {
        T x;
        tt_value(val[bk + j], x);
        if (x != 0) tt_add(acc[ev_frame[bk + j]], x, v1);
      }
      __syncwarp();
    }
  }
}

// One warp per column f1 of one q bin, W columns a block: the column's sums
// over f0 <= f1 in the warp's shared memory (F floats).  Long columns first;
// the block writes its columns side by side (32-byte sectors at W = 8).
// Measured (256 x 256 pixels, 701 frames, 6 q bins, 2 % of the pixels hit per
// frame): the two-time call 0.84 ms against 11.3 ms with the dense matrix,
// 9.75 ms of it in the tiled Gram.
__global__ void __launch_bounds__(256)
k_tt_gram_events(int32_t F, const int32_t *__restrict__ q_ptr,
                 const int64_t *__restrict__ col_ptr, const int32_t *__restrict__ a,
                 const float *__restrict__ b, const int32_t *__restrict__ row_pix,
                 const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ ev_frame,
                 const float *__restrict__ sv, float *__restrict__ C) {
  extern __shared__ float tt_acc[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int q = blockIdx.y, c0 = (gridDim.x - 1 - blockIdx.x) * W, f1 = c0 + w;
  float *acc = tt_acc + (size_t)w * F;
  if (f1 < F) {
    for (int f = lane; f <= f1; f += 32) acc[f] = 0.f;
    __syncwarp();
    const int64_t *cp = col_ptr + (int64_t)q * F + f1;
    tt_column<float>(cp[0], cp[1], a, b, row_pix, row_ptr, ev_frame, sv, acc);
  }
  __syncthreads();
  const float den = (float)(q_ptr[q + 1] - q_ptr[q]);
  float *Cq = C + (size_t)q * F * F;
  const int last = min(c0 + W, F) - 1;
  for (int idx = threadIdx.x; idx < (last + 1) * W; idx += blockDim.x) {
    const int f0 = idx / W, cw = idx % W, c = c0 + cw;
    if (c < F && f0 <= c) Cq[(size_t)f0 * F + c] = __fdiv_rn(tt_acc[(size_t)cw * F + f0], den);
  }
}

// ----------------------------------------- EXACT mode from the event lists
//
// The counts' Gram products are integers, so the lists give EXACT mode's
// matrices as well, and for sparse counts with less work than the dense Gram
// on the tensor cores, which multiplies (and first stores) mostly zeros:
// int32 sums in shared memory, exact while sum over a group's rows of (max
// count)^2 < 2^31, then the same double operations on them as after the
// tensor-core Gram (k_twotime_tc.cu).

// Per group: sum over its rows of (max |count|)^2; flag 1: a value that is not
// an integer count.  One warp per row.
__global__ void k_tt_check(int32_t R, const int32_t *__restrict__ row_pix,
                           const int32_t *__restrict__ row_grp,
                           const int64_t *__restrict__ row_ptr,
                           const int32_t *__restrict__ row_len, const float *__restrict__ ev_val,
                           unsigned long long *__restrict__ bound, int32_t *__restrict__ flags) {
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= R) return;
  const int lane = threadIdx.x & 31, p = row_pix[r], n = row_len[p];
  const int64_t base = row_ptr[p];
  unsigned mx = 0;
  bool bad = false;
  for (int i = lane; i < n; i += 32) {
    const float v = ev_val[base + i];
    const bool ok = v == truncf(v) && fabsf(v) <= 65536.f;
    bad = bad || !ok;
    mx = max(mx, ok ? (unsigned)fabsf(v) : 0u);
  }
  bad = __any_sync(0xffffffffu, bad);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) {
    if (bad) atomicOr(flags, 1);
    if (mx) atomicAdd(&bound[row_grp[r]], (unsigned long long)mx * mx);
  }
}

// The part of column c's events whose rows lie in [r0, r1) (ascending rows).
__device__ __forceinline__ int64_t tt_first_row(const int32_t *__restrict__ a, int64_t lo,
                                                int64_t hi, int32_t r) {
  int64_t len = hi - lo;
  while (len > 0) {
    const int64_t h = len >> 1;
    if (a[lo + h] < r) {
      lo += h + 1;
      len -= h + 1;
    } else {
      len = h;
    }
  }
  return lo;
}

// sg[g][f] = (sum of the group's counts at f) / pixels in double, and its
// reciprocal; sg as float.  One warp per (group, frame).
__global__ void k_tt_sg_counts(int32_t F, const int32_t *__restrict__ grp_ptr,
                               const int32_t *__restrict__ grp_q,
                               const int64_t *__restrict__ col_ptr, const int32_t *__restrict__ a,
                               const float *__restrict__ b, const int32_t *__restrict__ row_pix,
                               const int64_t *__restrict__ row_ptr,
                               const float *__restrict__ ev_val, double *__restrict__ sgd,
                               double *__restrict__ isg, float *__restrict__ sg) {
  const int lane = threadIdx.x & 31;
  const int nb = (F + 7) / 8;  // blocks of 8 frames; any number of groups in one dimension
  const int f = (int)(blockIdx.x % nb) * 8 + (threadIdx.x >> 5), g = (int)(blockIdx.x / nb);
  if (f >= F) return;
  const int r0 = grp_ptr[g], r1 = grp_ptr[g + 1];
  const int64_t c = (int64_t)grp_q[g] * F + f;
  const int64_t lo = tt_first_row(a, col_ptr[c], col_ptr[c + 1], r0);
  const int64_t hi = tt_first_row(a, lo, col_ptr[c + 1], r1);
  long long s = 0;
  for (int64_t e = lo + lane; e < hi; e += 32)
    s += (long long)ev_val[row_ptr[row_pix[a[e]]] + __float_as_int(b[e])];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const double v = (double)s / (r1 - r0);
    sgd[(size_t)g * F + f] = v;
    isg[(size_t)g * F + f] = 1.0 / v;
    sg[(size_t)g * F + f] = (float)v;
  }
}

// The averaged form: the mean over the frames, in order; one thread per group.
__global__ void k_tt_sg_counts_avg(int32_t G, int32_t F, const double *__restrict__ sgd,
                                   double *__restrict__ isg, float *__restrict__ sga) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= G) return;
  double mean = 0.0;
  for (int f = 0; f < F; f++) mean += sgd[(size_t)g * F + f];
  mean /= F;
  isg[(size_t)g * F] = 1.0 / mean;
  sga[g] = (float)mean;
}

// One warp per column as k_tt_gram_events, on the counts: the int32 sums of
// every smoothing group of the q bin in turn, folded into double sums where
// there are several (multi), C and its double form Cq as k_tc_single /
// k_tc_accum and k_tc_final give them.
// Measured (512 x 512 pixels, 1,536 frames, 9 q bins, 1 % of the pixels hit per
// frame, one group per q bin): the call 1.05 ms against 3.58 with the
// tensor-core Gram (1.45 in the Gram, the rest in building, clearing and
// scaling its matrices and in a synchronisation per group).
__global__ void __launch_bounds__(256)
k_tt_gram_counts(int32_t F, int32_t q0, int32_t multi, int32_t average,
                 const int32_t *__restrict__ q_ptr, const int32_t *__restrict__ q_grp,
                 const int32_t *__restrict__ grp_ptr, const int64_t *__restrict__ col_ptr,
                 const int32_t *__restrict__ a, const float *__restrict__ b,
                 const int32_t *__restrict__ row_pix, const int64_t *__restrict__ row_ptr,
                 const int32_t *__restrict__ ev_frame, const float *__restrict__ ev_val,
                 const double *__restrict__ isg, double *__restrict__ Cd, float *__restrict__ C) {
  extern __shared__ __align__(16) uint8_t tt_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int q = q0 + blockIdx.y, c0 = (gridDim.x - 1 - blockIdx.x) * W, f1 = c0 + w;
  double *dsum = (double *)tt_raw;  // [W][F] when multi
  int32_t *isum = (int32_t *)(dsum + (multi ? (size_t)W * F : 0));
  int32_t *acc = isum + (size_t)w * F;
  double *dac = dsum + (size_t)w * F;
  const int g0 = q_grp[q], g1 = q_grp[q + 1];
  if (f1 < F) {
    const int64_t lo = col_ptr[(int64_t)q * F + f1], hi = col_ptr[(int64_t)q * F + f1 + 1];
    if (multi)
      for (int f = lane; f <= f1; f += 32) dac[f] = 0.0;
    for (int g = g0; g < g1; g++) {
      for (int f = lane; f <= f1; f += 32) acc[f] = 0;
      __syncwarp();
      const int64_t l = multi ? tt_first_row(a, lo, hi, grp_ptr[g]) : lo;
      const int64_t h = multi ? tt_first_row(a, l, hi, grp_ptr[g + 1]) : hi;
      tt_column<int32_t>(l, h, a, b, row_pix, row_ptr, ev_frame, ev_val, acc);
      if (!multi) break;
      const double *ig = isg + (size_t)g * F;
      const double y = average ? ig[0] : ig[f1];
      for (int f = lane; f <= f1; f += 32)
        if (acc[f]) dac[f] += (double)acc[f] * (average ? ig[0] : ig[f]) * y;
      __syncwarp();
    }
  }
  __syncthreads();
  const int32_t npix = q_ptr[q + 1] - q_ptr[q];
  const double inv = npix ? 1.0 / npix : 0.0;
  const double *ig = isg + (size_t)g0 * F;
  double *Cdq = Cd + (size_t)blockIdx.y * F * F;
  float *Cq = C + (size_t)q * F * F;
  const int last = min(c0 + W, F) - 1;
  for (int idx = threadIdx.x; idx < (last + 1) * W; idx += blockDim.x) {
    const int f0 = idx / W, cw = idx % W, c = c0 + cw;
    if (c >= F || f0 > c) continue;
    double v;
    if (multi) {
      v = dsum[(size_t)cw * F + f0] * inv;
    } else {
      const int32_t n = isum[(size_t)cw * F + f0];
      v = n ? (double)n * (average ? ig[0] : ig[f0]) * (average ? ig[0] : ig[c]) * inv : 0.0;
    }
    Cdq[(size_t)f0 * F + c] = v;
    Cq[(size_t)f0 * F + c] = (float)v;
  }
}

// Columns per block of the event Grams, of `bytes` per frame: 8 while two
// blocks fit on an SM, fewer for longer columns; 0 when not even one fits.
int tt_columns(int32_t F, size_t bytes) {
  const size_t col = bytes * (size_t)F;
  for (int w : {8, 4, 2, 1})
    if (w * col <= 110 * 1024) return w;
  return col <= 220 * 1024 ? 1 : 0;
}

// one thread per (q, diagonal ff): g2full and, for ff < window, g2partials
__global__ void k_tt_diag(int32_t Q, int32_t F, int32_t window, int32_t tp,
                          const float *__restrict__ C, float *__restrict__ g2full,
                          float *__restrict__ g2part) {
  const int ff = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (ff >= F || q >= Q) return;
  const float *Cq = C + (size_t)q * F * F;
  float acc = 0.f;
  int fx = 0;
  for (; fx + 16 <= F - ff; fx += 16) {  // the loads first, in flight together
    float x[16];
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = Cq[(size_t)(fx + j) * F + fx + j + ff];
#pragma unroll
    for (int j = 0; j < 16; j++) acc = __fadd_rn(acc, x[j]);
  }
  for (; fx < F - ff; fx++) acc = __fadd_rn(acc, Cq[(size_t)fx * F + fx + ff]);
  g2full[(size_t)ff * Q + q] = __fdiv_rn(acc, (float)(F - ff));
  if (ff < window) {
    for (int w = 0; w < tp; w++) {
      float s = 0.f;
      for (int fx = w * window; fx < (w + 1) * window && fx < F - ff; fx++)
        s = __fadd_rn(s, Cq[(size_t)fx * F + fx + ff]);
      g2part[((size_t)ff * tp + w) * Q + q] = __fdiv_rn(s, (float)window);
    }
  }
}

// Device memory that the event lists and their tables would still have to
// allocate.
size_t lists_bytes(const Series &s, int32_t R, int32_t G, int32_t Q) {
  const size_t n = (size_t)std::max<int64_t>(s.raw_events, 1);
  return s.keyA.more(n) + s.keyB.more(n) + s.frA.more(n) + s.frB.more(n) + s.vA.more(n) +
         s.vB.more(n) + s.hist.more(radix_hist_words(n)) + s.tt_len.more(R) +
         s.tt_cpos.more((size_t)R + 2) + s.tt_cols.more((size_t)Q * s.F + 1) +
         s.tt_qptr.more(2 * (size_t)Q + G + 2) + s.scan_tmp.more(scan_workspace_bytes(R));
}

// The density of rows with the given ordered pairs of events, as if every frame of
// every row had it: what the lists' work, which is in pairs, goes by where some
// of the processed rows are far brighter than the detector.
double pair_density(int64_t pairs, int32_t R, int32_t F) {
  return std::sqrt((double)pairs / R) / F;
}

// The density up to which the event Gram is taken, of the mapped pixels before its
// lists are made and of the processed rows' pairs then (events per pixel and frame,
// d).  Its work grows as d^2, the tiled Gram's
// not at all, and short columns are cheap at any density.  Whole calls in ms,
// event lists / tiled (random events, 3 q bins):
//   pixels  frames   d = 0.05      0.1         0.2         0.4
//   128^2      100  0.38/2.52   0.49/2.53   0.70/2.57   1.41/2.58   (0.7: 3.1/2.6)
//   128^2      700  0.53/2.73   0.98/2.78   2.70/2.85   9.5/3.0
//   128^2    2,000  1.10/6.61   2.50/6.74   7.95/7.02   28.5/7.5
//   256^2      700  1.20/12.5   3.03/12.6   10.1/12.8   36.8/13.2
//   64^2     4,096  1.58/5.60   3.10/5.75   9.03/6.09   32.0/7.0
// Under a memory limit the form that takes less more of it is chosen, so that
// no call is refused for the lists.
double tt_events_most(int32_t F) { return std::min(0.4, std::max(0.15, 40.0 / F)); }
bool tt_use_events(Series &s, int32_t R, int32_t G, int32_t Q) {
  if (tt_columns(s.F, sizeof(float)) == 0) return false;
  if (dev_limited() && lists_bytes(s, R, G, Q) + s.tt_V.more(s.raw_events) >
                           s.tt_V.more((size_t)R * s.F))
    return false;
  return (double)s.raw_events <=
         tt_events_most(s.F) * (double)s.qmap.pix.size() * s.R_in * s.F;
}

// Warps of 256-thread blocks for k units of one warp.
unsigned tt_warps(int64_t k) { return (unsigned)((k * 32 + 255) / 256); }

struct EventLists {
  const int32_t *q_ptr, *grp_q, *q_grp;  // rows of each q bin; q bin of each group; groups of each
  int64_t n;                             // events of the rows
};

// Row counts for the lists, and the tables of q bins and groups; enqueues the
// copy of the rows' events and ordered pairs of events to n[0] and n[1] (valid
// after a synchronisation).
EventLists lists_prepare(Series &s, const TwoTimeLayout &lay, int32_t R, int32_t G, int32_t Q,
                         const int32_t *order, int64_t *n) {
  cudaStream_t st = s.stream;
  std::vector<int32_t> tab(lay.q_ptr);
  for (int32_t g = 0, q = 0; g < G; g++) {
    while (q + 1 < Q && lay.grp_ptr[g] >= lay.q_ptr[q + 1]) q++;
    tab.push_back(q);
  }
  tab.push_back(0);
  tab.insert(tab.end(), lay.q_grp_end.begin(), lay.q_grp_end.end());
  s.tt_qptr.reserve(tab.size(), st);
  XG_CUDA(cudaMemcpyAsync(s.tt_qptr.p, tab.data(), 4 * tab.size(), cudaMemcpyHostToDevice, st));
  s.tt_len.reserve(R, st);
  s.tt_cpos.reserve((size_t)R + 2, st);
  s.tt_cols.reserve((size_t)Q * s.F + 1, st);
  s.scan_tmp.reserve(scan_workspace_bytes(R), st);
  XG_CUDA(cudaMemsetAsync(s.tt_cpos.p + R + 1, 0, sizeof(int64_t), st));
  k_tt_lens<<<(R + 255) / 256, 256, 0, st>>>(R, order, s.tt_row_pix.p, s.row_len.p, s.tt_len.p,
                                             (unsigned long long *)s.tt_cpos.p + R + 1);
  XG_CHECK_LAUNCH();
  exclusive_scan_i32_i64(s.tt_len.p, s.tt_cpos.p, R, s.scan_tmp.p, st);
  if (n) XG_CUDA(cudaMemcpyAsync(n, s.tt_cpos.p + R, 2 * sizeof(*n), cudaMemcpyDeviceToHost, st));
  const int32_t *q_ptr = s.tt_qptr.p;
  return {q_ptr, q_ptr + Q + 1, q_ptr + Q + 1 + G, 0};
}

// The lists are not taken after all: under a memory limit their tables give way to
// the other form's buffers.
bool lists_refused(Series &s) {
  if (dev_limited()) {
    s.tt_len.release(s.stream);
    s.tt_cpos.release(s.stream);
    s.tt_cols.release(s.stream);
  }
  return false;
}

// Sorts the rows' events by (q, frame) from the given row order (null: mapping
// order); the sorted (row, position) pairs, and the columns' first events in
// tt_cols.
std::pair<const int32_t *, const float *> lists_build(Series &s, const EventLists &l, int32_t R,
                                                      int32_t Q, const int32_t *order) {
  cudaStream_t st = s.stream;
  const int32_t F = s.F;
  const int64_t ncol = (int64_t)Q * F;
  const size_t ne = std::max<int64_t>(l.n, 1);
  s.keyA.reserve(ne, st);
  s.frA.reserve(ne, st);
  s.vA.reserve(ne, st);
  s.keyB.reserve(ne, st);
  s.frB.reserve(ne, st);
  s.vB.reserve(ne, st);
  k_tt_build<<<tt_warps(R), 256, 0, st>>>(R, F, Q, order, l.q_ptr, s.tt_row_pix.p, s.row_ptr.p,
                                          s.row_len.p, s.ev_frame.p, s.tt_cpos.p, s.keyA.p,
                                          s.frA.p, s.vA.p);
  XG_CHECK_LAUNCH();
  const int bits = ncol > 1 ? 64 - __builtin_clzll((unsigned long long)ncol - 1) : 1;
  const bool in_b =
      radix_sort_triples(s, s.keyA.p, s.frA.p, s.vA.p, s.keyB.p, s.frB.p, s.vB.p, l.n, bits);
  k_tt_cols<<<(unsigned)((ncol + 256) / 256), 256, 0, st>>>(ncol, l.n, in_b ? s.keyB.p : s.keyA.p,
                                                            s.tt_cols.p);
  XG_CHECK_LAUNCH();
  return {in_b ? s.frB.p : s.frA.p, in_b ? s.vB.p : s.vA.p};
}

// C, sg and sga from event lists; false when the processed rows are too dense.
bool gram_events(Series &s, const TwoTimeReq &req, const TwoTimeLayout &lay, int32_t R, int32_t G,
                 int32_t Q) {
  cudaStream_t st = s.stream;
  const int32_t F = s.F;
  int64_t n[2] = {0, 0};
  EventLists l = lists_prepare(s, lay, R, G, Q, nullptr, n);
  XG_CUDA(cudaStreamSynchronize(st));
  if (pair_density(n[1], R, F) > tt_events_most(F)) return lists_refused(s);
  l.n = n[0];
  auto ab = lists_build(s, l, R, Q, nullptr);  // mapping order
  k_tt_sg_events<<<dim3(tt_warps(F), G), 256, 0, st>>>(F, s.tt_grp_ptr.p, l.grp_q, s.tt_cols.p,
                                                       ab.first, ab.second, s.tt_row_pix.p,
                                                       s.row_ptr.p, s.ev_val.p, s.tt_sg.p);
  XG_CHECK_LAUNCH();
  if (req.average) {
    k_tt_sg_avg<<<(G + 127) / 128, 128, 0, st>>>(G, F, s.tt_sg.p, s.tt_sga.p);
    XG_CHECK_LAUNCH();
  }
  s.tt_V.reserve((size_t)std::max<int64_t>(s.raw_events, 1), st);  // as long as the event lists
  k_tt_smooth_events<<<tt_warps(R), 256, 0, st>>>(R, F, req.average, s.tt_row_pix.p,
                                                  s.tt_row_grp.p, s.row_ptr.p, s.row_len.p,
                                                  s.ev_frame.p, s.ev_val.p,
                                                  req.average ? s.tt_sga.p : s.tt_sg.p, s.tt_V.p);
  XG_CHECK_LAUNCH();
  if (req.frame_threading) {
    lists_prepare(s, lay, R, G, Q, s.tt_order.p, nullptr);
    ab = lists_build(s, l, R, Q, s.tt_order.p);
  }
  const int W = tt_columns(F, sizeof(float));
  const size_t smem = sizeof(float) * (size_t)F * W;
  allow_smem(k_tt_gram_events);
  k_tt_gram_events<<<dim3((F + W - 1) / W, Q), 32 * W, smem, st>>>(
      F, l.q_ptr, s.tt_cols.p, ab.first, ab.second, s.tt_row_pix.p, s.row_ptr.p, s.ev_frame.p,
      s.tt_V.p, s.tt_C.p);
  XG_CHECK_LAUNCH();
  return true;
}

// EXACT mode from the counts' event lists; false when the series takes the
// other forms: pixels, or the processed rows by their pairs of events, too dense
// for the lists, or counts too large for int32 sums.  The lists' work grows with the square of the events per pixel and
// frame, d, and the tensor-core Gram's hardly at all; longer columns leave the
// lists fewer warps per SM.  Whole calls in ms, lists / tensor cores:
//   pixels  frames  q bins   d = 0.01       0.02        0.03        0.05
//   256^2      300       3  0.38/0.85   0.50/0.89   0.58/0.88   0.77/0.94  (0.1: 1.35/1.13)
//   512^2    1,536       9  1.05/3.58   1.54/3.74   2.37/4.04   4.50/4.62
//     (two groups a q bin)  1.55/4.54   2.39/4.83   3.61/5.22   7.02/6.04
//   1024^2     700       9  2.13/9.83   3.14/10.3   4.10/11.4   7.87/13.3
//   512^2    4,096       9  4.02/6.50   8.57/7.08   15.7/8.02   38.1/9.72
bool gram_counts(Series &s, const TwoTimeReq &req, const TwoTimeLayout &lay, int32_t R, int32_t G,
                 int32_t Q) {
  cudaStream_t st = s.stream;
  const int32_t F = s.F;
  const double most = std::min(0.06, 65.0 / F);
  if (F > 65535 || (int64_t)(F + 7) / 8 * G > INT32_MAX ||
      (double)s.raw_events > most * (double)s.qmap.pix.size() * s.R_in * F)
    return false;
  const bool multi = G > Q;
  const size_t col = sizeof(int32_t) + (multi ? sizeof(double) : 0);
  const int W = tt_columns(F, col);
  if (W == 0) return false;
  const size_t F2 = (size_t)F * F;
  // q bins at a time: their double matrices within 2 GB, and a grid's rows
  int32_t step = (int32_t)std::max<size_t>(
      1, std::min<size_t>(std::min(Q, 65535), (2ull << 30) / (8 * F2)));
  if (dev_limited()) {  // as in tt_use_events
    step = 1;
    if (lists_bytes(s, R, G, Q) + s.tt_Cq.more(F2) + s.tt_sgd.more(2 * (size_t)G * F) +
            s.tt_bound.more(G) >
        twotime_exact_bytes(s, lay))
      return false;
  }
  int64_t n[2] = {0, 0};
  int32_t flags = 0;
  std::vector<unsigned long long> bound(G);
  s.tt_bound.reserve(std::max(G, 2), st);
  s.tt_flags.reserve(1, st);
  XG_CUDA(cudaMemsetAsync(s.tt_bound.p, 0, sizeof(unsigned long long) * G, st));
  XG_CUDA(cudaMemsetAsync(s.tt_flags.p, 0, sizeof(int32_t), st));
  k_tt_check<<<tt_warps(R), 256, 0, st>>>(R, s.tt_row_pix.p, s.tt_row_grp.p, s.row_ptr.p,
                                          s.row_len.p, s.ev_val.p, s.tt_bound.p, s.tt_flags.p);
  XG_CHECK_LAUNCH();
  EventLists l = lists_prepare(s, lay, R, G, Q, nullptr, n);
  XG_CUDA(cudaMemcpyAsync(bound.data(), s.tt_bound.p, sizeof(unsigned long long) * G,
                          cudaMemcpyDeviceToHost, st));
  XG_CUDA(cudaMemcpyAsync(&flags, s.tt_flags.p, sizeof(flags), cudaMemcpyDeviceToHost, st));
  XG_CUDA(cudaStreamSynchronize(st));
  l.n = n[0];
  if (flags & 1) tt_not_counts();
  if (pair_density(n[1], R, F) > most) return lists_refused(s);
  for (unsigned long long b : bound)
    if (b >= (1ull << 31)) return lists_refused(s);
  const auto ab = lists_build(s, l, R, Q, nullptr);
  s.tt_sgd.reserve(2 * (size_t)G * F, st);
  double *sgd = s.tt_sgd.p, *isg = sgd + (size_t)G * F;
  k_tt_sg_counts<<<(unsigned)((F + 7) / 8) * (unsigned)G, 256, 0, st>>>(
      F, s.tt_grp_ptr.p, l.grp_q, s.tt_cols.p, ab.first, ab.second, s.tt_row_pix.p, s.row_ptr.p,
      s.ev_val.p, sgd, isg, s.tt_sg.p);
  XG_CHECK_LAUNCH();
  if (req.average) {
    k_tt_sg_counts_avg<<<(G + 31) / 32, 32, 0, st>>>(G, F, sgd, isg, s.tt_sga.p);
    XG_CHECK_LAUNCH();
  }
  const size_t smem = col * (size_t)F * W;
  allow_smem(k_tt_gram_counts);
  s.tt_Cq.reserve(F2 * step, st);
  for (int32_t q = 0; q < Q; q += step) {
    const int32_t nq = std::min(step, Q - q);
    k_tt_gram_counts<<<dim3((F + W - 1) / W, nq), 32 * W, smem, st>>>(
        F, q, multi, req.average, l.q_ptr, l.q_grp, s.tt_grp_ptr.p, s.tt_cols.p, ab.first,
        ab.second, s.tt_row_pix.p, s.row_ptr.p, s.ev_frame.p, s.ev_val.p, isg, s.tt_Cq.p,
        s.tt_C.p);
    XG_CHECK_LAUNCH();
    twotime_exact_diag(s, req.window, Q, q, nq);
  }
  return true;
}

// The same from the dense matrix V.
void gram_dense(Series &s, const TwoTimeReq &req, const TwoTimeLayout &lay, int32_t R, int32_t G,
                int32_t Q) {
  cudaStream_t st = s.stream;
  const int32_t F = s.F;
  const std::vector<int32_t> &q_ptr = lay.q_ptr;
  const size_t nV = (size_t)R * F;
  s.tt_V.reserve(nV, st);
  XG_CUDA(cudaMemsetAsync(s.tt_V.p, 0, 4 * nV, st));
  k_tt_scatter<<<(R + 127) / 128, 128, 0, st>>>(R, F, s.tt_row_pix.p, s.row_ptr.p, s.row_len.p,
                                                s.ev_frame.p, s.ev_val.p, s.tt_V.p);
  XG_CHECK_LAUNCH();
  k_tt_sg<<<dim3((F + 127) / 128, G), 128, 0, st>>>(G, F, s.tt_grp_ptr.p, s.tt_V.p, s.tt_sg.p);
  XG_CHECK_LAUNCH();
  if (req.average) {
    k_tt_sg_avg<<<(G + 127) / 128, 128, 0, st>>>(G, F, s.tt_sg.p, s.tt_sga.p);
    XG_CHECK_LAUNCH();
  }
  k_tt_smooth<<<(unsigned)((nV + 255) / 256), 256, 0, st>>>(R, F, req.average, s.tt_row_grp.p,
                                                           req.average ? s.tt_sga.p : s.tt_sg.p,
                                                           s.tt_V.p);
  XG_CHECK_LAUNCH();
  const int T = (F + TT_TILE - 1) / TT_TILE;
  for (int32_t q = 0; q < Q; q++) {
    const int32_t nr = q_ptr[q + 1] - q_ptr[q];
    if (nr == 0) continue;
    k_tt_gram<<<T * (T + 1) / 2, 256, 0, st>>>(F, nr, s.tt_order.p + q_ptr[q], s.tt_V.p,
                                               s.tt_C.p + (size_t)q * F * F);
    XG_CHECK_LAUNCH();
  }
}

}  // namespace

void run_twotime(Series &s, const TwoTimeReq &req, int mode, bool force_i64) {
  cudaStream_t st = s.stream;
  const QMap &qm = s.qmap;
  const int32_t F = s.F;
  TwoTimeOut &o = s.tt;
  o = TwoTimeOut{};
  o.frames = F;
  o.window = req.window;
  o.partials = req.window > 0 ? std::max(0, (F - req.window) / req.window) : 0;
  // rows of the processed q bins in mapping order (ranges of the mapping's
  // pixel list, which is on the device already); smoothing groups; q row ranges
  TwoTimeLayout lay;
  int32_t R = 0;
  std::vector<std::pair<int32_t, int32_t>> runs;  // [first, end) of the pixel list
  for (int32_t i = 0; i < qm.nq(); i++) {
    const int32_t q = qm.q_ids[i];
    if (std::find(req.qbins.begin(), req.qbins.end(), q) == req.qbins.end()) continue;
    const int32_t k0 = qm.entry_pix_ptr[qm.q_entry_ptr[i]];
    const int32_t k1 = qm.entry_pix_ptr[qm.q_entry_ptr[i + 1]];
    if (req.static_map)
      for (int32_t e = qm.q_entry_ptr[i]; e < qm.q_entry_ptr[i + 1]; e++)
        lay.grp_ptr.push_back(R + qm.entry_pix_ptr[e + 1] - k0);
    else
      lay.grp_ptr.push_back(R + k1 - k0);
    R += k1 - k0;
    if (!runs.empty() && runs.back().second == k0)
      runs.back().second = k1;
    else
      runs.push_back({k0, k1});
    lay.q_ptr.push_back(R);
    lay.q_grp_end.push_back((int32_t)lay.grp_ptr.size() - 1);
    o.qbins.push_back(q);
  }
  const std::vector<int32_t> &grp_ptr = lay.grp_ptr, &q_ptr = lay.q_ptr;
  const int32_t G = (int32_t)grp_ptr.size() - 1, Q = (int32_t)o.qbins.size();
  o.sg_rows = G;
  o.sg_cols = req.average ? 1 : F;
  o.averaged = req.average != 0;
  auto up = [&](DBuf<int32_t> &b, const std::vector<int32_t> &v) {
    b.reserve(v.size() ? v.size() : 1, st);
    if (!v.empty())
      XG_CUDA(cudaMemcpyAsync(b.p, v.data(), 4 * v.size(), cudaMemcpyHostToDevice, st));
  };
  s.tt_row_pix.reserve(R ? R : 1, st);
  int32_t at = 0;
  for (const auto &r : runs) {
    if (r.second > r.first)
      XG_CUDA(cudaMemcpyAsync(s.tt_row_pix.p + at, s.n_pix.p + r.first,
                              4 * (size_t)(r.second - r.first), cudaMemcpyDeviceToDevice, st));
    at += r.second - r.first;
  }
  up(s.tt_grp_ptr, grp_ptr);
  s.tt_row_grp.reserve(R ? R : 1, st);
  if (R > 0) {
    k_tt_groups<<<(R + 255) / 256, 256, 0, st>>>(R, G, s.tt_grp_ptr.p, s.tt_row_grp.p);
    XG_CHECK_LAUNCH();
  }
  s.tt_sg.reserve((size_t)(G ? G : 1) * (F ? F : 1), st);
  s.tt_sga.reserve(G ? G : 1, st);
  s.tt_C.reserve((size_t)(Q ? Q : 1) * F * F + 1, st);
  s.tt_full.reserve((size_t)F * (Q ? Q : 1) + 1, st);
  s.tt_part.reserve((size_t)req.window * o.partials * (Q ? Q : 1) + 1, st);
  XG_CUDA(cudaMemsetAsync(s.tt_C.p, 0, 4 * ((size_t)Q * F * F + 1), st));
  if (mode == XPCS_MODE_EXACT) {
    if (R > 0 && F > 0 && (force_i64 || !gram_counts(s, req, lay, R, G, Q)))
      run_twotime_exact(s, req, lay, force_i64);
    o.ready = true;
    return;
  }
  // Gram order of every q bin's rows
  const auto upload_order = [&] {
    std::vector<int32_t> order(R);
    std::iota(order.begin(), order.end(), 0);
    if (req.frame_threading) {
      std::vector<int32_t> row_pix;
      for (const auto &r : runs)
        row_pix.insert(row_pix.end(), qm.pix.begin() + r.first, qm.pix.begin() + r.second);
      for (int32_t q = 0; q < Q; q++)
        std::sort(order.begin() + q_ptr[q], order.begin() + q_ptr[q + 1],
                  [&](int32_t a, int32_t b) { return row_pix[a] < row_pix[b]; });
    }
    up(s.tt_order, order);
  };
  if (R > 0 && F > 0) {
    if (req.frame_threading) upload_order();  // event lists take the mapping order as it is
    if (!tt_use_events(s, R, G, Q) || !gram_events(s, req, lay, R, G, Q)) {
      if (!req.frame_threading) upload_order();
      gram_dense(s, req, lay, R, G, Q);
    }
    k_tt_diag<<<dim3((F + 127) / 128, Q), 128, 0, st>>>(Q, F, req.window, o.partials, s.tt_C.p,
                                                       s.tt_full.p, s.tt_part.p);
    XG_CHECK_LAUNCH();
  }
  o.ready = true;
}

void get_twotime(Series &s, int32_t *qbins, float *sg, float *c2t, float *g2full,
                 float *g2part) {
  cudaStream_t st = s.stream;
  const TwoTimeOut &o = s.tt;
  const size_t Q = o.qbins.size(), F = (size_t)o.frames;
  if (qbins) std::copy(o.qbins.begin(), o.qbins.end(), qbins);
  if (sg && o.sg_rows)
    XG_CUDA(cudaMemcpyAsync(sg, o.averaged ? s.tt_sga.p : s.tt_sg.p,
                            4 * (size_t)o.sg_rows * o.sg_cols, cudaMemcpyDeviceToHost, st));
  if (c2t) populate_host(c2t, 4 * Q * F * F);
  if (c2t && Q) XG_CUDA(cudaMemcpyAsync(c2t, s.tt_C.p, 4 * Q * F * F, cudaMemcpyDeviceToHost, st));
  if (g2full && Q) XG_CUDA(cudaMemcpyAsync(g2full, s.tt_full.p, 4 * F * Q, cudaMemcpyDeviceToHost, st));
  if (g2part && Q && o.partials)
    XG_CUDA(cudaMemcpyAsync(g2part, s.tt_part.p, 4 * (size_t)o.window * o.partials * Q,
                            cudaMemcpyDeviceToHost, st));
  XG_CUDA(cudaStreamSynchronize(st));
}

}  // namespace xg
