// F1: side statistics of the filters, bit-identical to the reference.
//
// SparseFilter::Apply / DenseFilter::Apply accumulate, per filter frame and
// in ascending pixel order (sparse_filter.cpp:160-192, dense_filter.cpp:176-
// 208), with float adds:
//   pixels_sum_[pix]                       += v   (frame order per pixel)
//   f_sum                                  += v   -> frames_sum_[F + k] = f_sum / P
//   partitions_mean_[sbin]                 += v   (frame-major, pixel order)
//   partial_partitions_mean_[win][sbin]    += v
// and main.cpp:321-411 divides pixelSum by the frame count and the partition
// means by pixels_per_bin * window (or * frames).  The float sums depend on
// the order, so they are replayed in it where it matters: pixel sums come from
// the merge pass (rows are in frame order).  Photon counts whose sums stay
// below 2^24 are added as integers, in any order (the integer series section
// below).  Otherwise the event lists are stably re-sorted by frame
// (giving frame-major, pixel-ascending order), summed per frame, then stably
// re-sorted by static bin (keeping that order inside each bin) and summed per
// bin and per (window, bin).  Pixel-major dense series, whose finishing pass
// skips the pixel sums, get them here from their rows.
#include <algorithm>
#include <climits>
#include <vector>

#include "xpcs_internal.h"

namespace xg {
namespace {

__device__ __forceinline__ int64_t lower_bound_u32(const uint32_t *a, int64_t n, uint32_t x) {
  int64_t first = 0, len = n;
  while (len > 0) {
    int64_t half = len >> 1;
    if (a[first + half] < x) {
      first += half + 1;
      len -= half + 1;
    } else {
      len = half;
    }
  }
  return first;
}

// rows (pixel-major) -> compact triples (key = frame, a = pixel, b = value);
// one warp per row, so that its events are read and written coalesced (one
// thread per row took 344 us at 640 x 480 x 2,000 frames, 11.4 M events)
__global__ void k_side_build(int32_t P, const int64_t *__restrict__ row_ptr,
                             const int32_t *__restrict__ row_len, const int64_t *__restrict__ cpos,
                             const int32_t *__restrict__ fr, const float *__restrict__ val,
                             uint32_t *__restrict__ key, int32_t *__restrict__ a,
                             float *__restrict__ b) {
  const int p = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (p >= P) return;
  const int64_t src = row_ptr[p], dst = cpos[p];
  const int n = row_len[p];
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    key[dst + i] = (uint32_t)fr[src + i];
    a[dst + i] = p;
    b[dst + i] = val[src + i];
  }
}

// ((b[lo] + b[lo + 1]) + ...) + b[hi - 1] from 0, in that order, by one warp
// (every lane returns it).  Bound by the chain of dependent additions, about
// 4 cycles each: the lanes load 256 values at a time, one chunk ahead, into
// the warp's shared memory, and every lane adds them in order from 16-byte
// broadcast reads that do not wait on the chain.  The partition sums of
// 11.4 M events in 24 bins: 3.2 ms (6.3 ms with the values passed by
// shuffle, 71 ms with one thread per sum and a dependent load each).
constexpr int OS_CHUNK = 256;
__device__ __forceinline__ float ordered_sum(const float *__restrict__ b, int64_t lo, int64_t hi,
                                             float *sm) {
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
  float x[OS_CHUNK / 32];
  auto load = [&](int64_t i) {
#pragma unroll
    for (int h = 0; h < OS_CHUNK / 32; h++)
      x[h] = i + h * 32 + lane < hi ? b[i + h * 32 + lane] : 0.f;
  };
  load(lo);
  for (int64_t i = lo; i < hi; i += OS_CHUNK) {
    __syncwarp();
#pragma unroll
    for (int h = 0; h < OS_CHUNK / 32; h++) sm[h * 32 + lane] = x[h];
    __syncwarp();
    load(i + OS_CHUNK);
    const int n = (int)min((int64_t)OS_CHUNK, hi - i);
    const float4 *s4 = (const float4 *)sm;
    if (n == OS_CHUNK) {
#pragma unroll 16
      for (int q = 0; q < OS_CHUNK / 4; q++) {
        const float4 y = s4[q];
        acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, y.x), y.y), y.z), y.w);
      }
    } else {
      for (int j = 0; j < n; j++) acc = __fadd_rn(acc, sm[j]);
    }
  }
  return acc;
}

// one warp per frame
__global__ void k_frame_sums(int32_t F, int32_t P, int64_t n, const uint32_t *__restrict__ key,
                             const float *__restrict__ b, float *__restrict__ frame_sum) {
  __shared__ __align__(16) float sm[8][OS_CHUNK];  // at most 8 warps a block
  const int k = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= F) return;
  const int64_t lo = lower_bound_u32(key, n, (uint32_t)k), hi = lower_bound_u32(key, n, (uint32_t)k + 1);
  const float f = ordered_sum(b, lo, hi, sm[threadIdx.x >> 5]);
  if ((threadIdx.x & 31) == 0) {
    frame_sum[k] = (float)(k + 1.0);
    frame_sum[F + k] = __fdiv_rn(f, (float)P);
  }
}

// key <- static bin of the pixel in a; a <- frame (the old key)
__global__ void k_sbin_keys(int64_t n, const int32_t *__restrict__ sbin, uint32_t *__restrict__ key,
                            int32_t *__restrict__ a) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t f = key[i];
  key[i] = (uint32_t)sbin[a[i]];
  a[i] = (int32_t)f;
}

// First of the events [lo, hi), frames ascending, with a frame >= f.
__device__ __forceinline__ int64_t first_frame(const int32_t *__restrict__ frame, int64_t lo,
                                               int64_t hi, int64_t f) {
  int64_t a = lo, len = hi - lo;
  while (len > 0) {
    const int64_t h = len >> 1;
    if (frame[a + h] < f) {
      a += h + 1;
      len -= h + 1;
    } else {
      len = h;
    }
  }
  return a;
}

// One warp (block) per static bin for the whole-series sum (the longest
// chains, in the first S blocks of the grid), then one per (window, static
// bin): each sum in event order.  Frames ascend inside a bin's segment.
__global__ void k_part_sums(int32_t S, int32_t nwin, int32_t sw, int32_t F, int64_t n,
                            const uint32_t *__restrict__ key, const int32_t *__restrict__ frame,
                            const float *__restrict__ b, const int32_t *__restrict__ ppb,
                            float *__restrict__ total, float *__restrict__ partial) {
  __shared__ __align__(16) float sm[OS_CHUNK];  // one warp a block
  const int64_t wid = blockIdx.x;
  const int w = (int)(wid / S) - 1, sb = (int)(wid % S);
  int64_t lo = lower_bound_u32(key, n, (uint32_t)sb), hi = lower_bound_u32(key, n, (uint32_t)sb + 1);
  if (w >= 0) {
    const int64_t end = hi;
    lo = first_frame(frame, lo, end, (int64_t)w * sw);
    hi = first_frame(frame, lo, end, (int64_t)(w + 1) * sw);
  }
  const float acc = ordered_sum(b, lo, hi, sm);
  if ((threadIdx.x & 31) != 0) return;
  if (w < 0)
    total[sb] = __fdiv_rn(acc, __fmul_rn((float)ppb[sb], (float)F));
  else
    partial[(size_t)w * S + sb] = __fdiv_rn(acc, __fmul_rn((float)ppb[sb], (float)sw));
}

// ------------------------------------------------------------ integer series
//
// Photon counts without flatfield or averaging: while every value is a
// non-negative integer and every sum stays below 2^24, each partial float sum
// of the reference is an integer below 2^24 and exact, so the order does not
// matter and integer sums give the same bits.  One pass over the pixel-major
// rows then replaces the two sorts and the ordered sums; k_side_int_out checks
// the conditions and sets `bad`, after which the ordered path runs.  32-bit
// sums cannot wrap while the series' total is below 2^32 (checked as well).
// Measured (640 x 480 x 2,000 frames, 11.4 M events; the whole call): 0.31 ms
// against 3.90 ms on the ordered path and 64 ms before.
struct SideInt {
  unsigned long long total;
  int32_t bad;
  int32_t pad;
};
constexpr int SI_THREADS = 512;
constexpr int SI_SMEM = 100 * 1024;  // frame and partition counters of a block: 2 blocks per SM

// A warp takes 32 rows in turn, its lanes over a row's events, with the next
// chunk's loads in flight.  The per-frame and per-(window, bin) counters live
// in shared memory where they fit (fs_in / pt_in) and are added to the global
// ones at the end; a row's events of one window are summed over the warp
// first.  175 us for 11.4 M events in 292 k rows, about 134 warp instructions
// a chunk at 38 % issue.  Window nwin collects the frames after the last whole
// window.
__global__ void __launch_bounds__(SI_THREADS)
k_side_int(int32_t P, int32_t F, int32_t S, int32_t nwin, int32_t sw, int32_t fs_in,
           int32_t pt_in, const int64_t *__restrict__ row_ptr,
           const int32_t *__restrict__ row_len, const int32_t *__restrict__ sbin,
           const int32_t *__restrict__ fr, const float *__restrict__ val,
           uint32_t *__restrict__ fs_g, uint32_t *__restrict__ pt_g, SideInt *__restrict__ si) {
  extern __shared__ uint32_t si_smem[];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int nfs = fs_in ? F : 0, npt = pt_in ? (nwin + 1) * S : 0;
  for (int k = threadIdx.x; k < nfs + npt; k += blockDim.x) si_smem[k] = 0;
  __syncthreads();
  uint32_t *fs = fs_in ? si_smem : fs_g;
  uint32_t *pt = pt_in ? si_smem + nfs : pt_g;
  unsigned long long total = 0;
  bool bad = false;
  const int64_t groups = ((int64_t)P + 31) / 32;
  for (int64_t g = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); g < groups;
       g += (int64_t)gridDim.x * warps) {
    const int64_t p = g * 32 + lane;
    const int my_n = p < P ? row_len[p] : 0;
    const int64_t my_b = my_n ? row_ptr[p] : 0;
    const int my_sb = my_n ? sbin[p] : 0;
    unsigned rows = __ballot_sync(FULL, my_n > 0);
    // the next chunk's events are loaded while this one is added up
    int q = rows ? __ffs(rows) - 1 : 0, i0 = 0;
    int n = __shfl_sync(FULL, my_n, q);
    int64_t b = __shfl_sync(FULL, my_b, q);
    int sb = __shfl_sync(FULL, my_sb, q);
    int f = lane < n ? fr[b + lane] : 0;
    float x = lane < n ? val[b + lane] : 0.f;
    while (rows) {
      const bool in = i0 + lane < n;
      const int fc = f, sbc = sb;
      const float xc = x;
      i0 += 32;
      if (i0 >= n) {
        rows &= rows - 1u;
        q = rows ? __ffs(rows) - 1 : 0;
        i0 = 0;
        n = rows ? __shfl_sync(FULL, my_n, q) : 0;
        b = __shfl_sync(FULL, my_b, q);
        sb = __shfl_sync(FULL, my_sb, q);
      }
      f = i0 + lane < n ? fr[b + i0 + lane] : 0;
      x = i0 + lane < n ? val[b + i0 + lane] : 0.f;
      const bool ok = xc >= 0.f && xc < 16777216.f && xc == truncf(xc);
      bad = bad || (in && !ok);
      const uint32_t v = in && ok ? (uint32_t)xc : 0u;
      total += v;
      if (v) atomicAdd(&fs[fc], v);
      // frames ascend, so a window's lanes are one run: its sum is the
      // difference of the inclusive prefix sum between the ends of runs
      const int w = in ? min(fc / sw, nwin) : INT_MAX;
      uint32_t s = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, s, o);
        if (lane >= o) s += y;
      }
      const int wn = __shfl_down_sync(FULL, w, 1);
      const bool end = in && (lane == 31 || w != wn);
      const unsigned ends = __ballot_sync(FULL, end) & ((1u << lane) - 1u);
      const uint32_t sp = __shfl_sync(FULL, s, ends ? 31 - __clz(ends) : 0);
      if (end) atomicAdd(&pt[(size_t)w * S + sbc], ends ? s - sp : s);
    }
  }
  if (total) atomicAdd(&si->total, total);
  if (bad) atomicOr(&si->bad, 1);
  __syncthreads();
  for (int k = threadIdx.x; k < nfs; k += blockDim.x)
    if (si_smem[k]) atomicAdd(&fs_g[k], si_smem[k]);
  for (int k = threadIdx.x; k < npt; k += blockDim.x)
    if (si_smem[nfs + k]) atomicAdd(&pt_g[k], si_smem[nfs + k]);
}

__global__ void k_side_int_out(int32_t P, int32_t F, int32_t S, int32_t nwin, int32_t sw,
                               const uint32_t *__restrict__ fs, const uint32_t *__restrict__ pt,
                               const int32_t *__restrict__ ppb,
                               const DevStats *__restrict__ stats, SideInt *__restrict__ si,
                               float *__restrict__ frame_sum, float *__restrict__ total,
                               float *__restrict__ partial) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool bad = i == 0 && si->total >= (1ull << 32);
  if (i < F) {
    bad = bad || fs[i] >= (1u << 24);
    frame_sum[i] = (float)((double)i + 1.0);
    frame_sum[F + i] = __fdiv_rn((float)fs[i], (float)P);
  }
  if (stats->events == 0) return;  // no events: the partition means stay 0, empty bins' too
  if (i < S) {
    unsigned long long t = 0;
    for (int w = 0; w <= nwin; w++) t += pt[(size_t)w * S + i];
    bad = bad || t >= (1ull << 24);
    total[i] = __fdiv_rn((float)t, __fmul_rn((float)ppb[i], (float)F));
  }
  if (i < (int64_t)S * nwin)
    partial[i] = __fdiv_rn((float)pt[i], __fmul_rn((float)ppb[i % S], (float)sw));
  if (bad) atomicOr(&si->bad, 1);
}

// pixels_sum_[pix] += v over a row in frame order, for rows whose finishing
// pass does not form the sums (pixel-major dense series).
__global__ void k_row_sums(int32_t P, const int64_t *__restrict__ row_ptr,
                           const int32_t *__restrict__ row_len, const float *__restrict__ val,
                           float *__restrict__ ps) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  const int64_t b = row_ptr[p];
  float a = 0.f;
  for (int32_t i = 0; i < row_len[p]; i++) a = __fadd_rn(a, val[b + i]);
  ps[p] = a;
}

__global__ void k_pixel_sums(int32_t P, int32_t F, const float *__restrict__ ps,
                             float *__restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < P) out[p] = __fdiv_rn(ps[p], (float)F);
}

}  // namespace

namespace {

// The ordered sums of frameSum and the partition means (any values), into the
// device results: the events re-sorted by frame, then by static bin.
void side_ordered(Series &s, int32_t nwin, float *d_fs, float *d_tot, float *d_part) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P, F = s.F, S = s.qmap.total_static, sw = s.desc.static_window;
  DevStats stats{};
  XG_CUDA(cudaMemcpyAsync(&stats, s.stats.p, sizeof(stats), cudaMemcpyDeviceToHost, st));
  XG_CUDA(cudaStreamSynchronize(st));
  const int64_t n = (int64_t)stats.events;
  const int bs = 256;
  if (n > 0) {
    s.side_pos.reserve((size_t)P + 1, st);
    s.scan_tmp.reserve(scan_workspace_bytes(P), st);
    exclusive_scan_i32_i64(s.row_len.p, s.side_pos.p, P, s.scan_tmp.p, st);
    s.keyA.reserve(n, st);
    s.frA.reserve(n, st);
    s.vA.reserve(n, st);
    s.keyB.reserve(n, st);
    s.frB.reserve(n, st);
    s.vB.reserve(n, st);
    const auto warps = [&](int64_t k) { return (unsigned)((k * 32 + bs - 1) / bs); };
    k_side_build<<<warps(P), bs, 0, st>>>(P, s.row_ptr.p, s.row_len.p, s.side_pos.p, s.ev_frame.p,
                                          s.ev_val.p, s.keyA.p, s.frA.p, s.vA.p);
    XG_CHECK_LAUNCH();
    const int fbits = 32 - __builtin_clz((unsigned)(F > 1 ? F - 1 : 1));
    const bool in_b = radix_sort_triples(s, s.keyA.p, s.frA.p, s.vA.p, s.keyB.p, s.frB.p, s.vB.p, n,
                                         fbits);
    uint32_t *k1 = in_b ? s.keyB.p : s.keyA.p, *k2 = in_b ? s.keyA.p : s.keyB.p;
    int32_t *a1 = in_b ? s.frB.p : s.frA.p, *a2 = in_b ? s.frA.p : s.frB.p;
    float *b1 = in_b ? s.vB.p : s.vA.p, *b2 = in_b ? s.vA.p : s.vB.p;
    k_frame_sums<<<warps(F), bs, 0, st>>>(F, P, n, k1, b1, d_fs);
    XG_CHECK_LAUNCH();
    k_sbin_keys<<<(unsigned)((n + bs - 1) / bs), bs, 0, st>>>(n, s.d_sbin.p, k1, a1);
    XG_CHECK_LAUNCH();
    const int sbits = 32 - __builtin_clz((unsigned)(S > 1 ? S - 1 : 1));
    const bool in2 = radix_sort_triples(s, k1, a1, b1, k2, a2, b2, n, sbits);
    // one warp per block: the long chains of the whole-series sums get SMs of their own
    k_part_sums<<<(unsigned)((int64_t)S * (nwin + 1)), 32, 0, st>>>(
        S, nwin, sw, F, n, in2 ? k2 : k1, in2 ? a2 : a1, in2 ? b2 : b1, s.d_ppb.p, d_tot, d_part);
    XG_CHECK_LAUNCH();
  } else {
    // no events: frame numbers still fill the first row of frameSum
    std::vector<float> fs(2 * (size_t)F, 0.f);
    for (int k = 0; k < F; k++) fs[k] = (float)(k + 1.0);
    if (F) XG_CUDA(cudaMemcpyAsync(d_fs, fs.data(), sizeof(float) * fs.size(), cudaMemcpyHostToDevice, st));
    XG_CUDA(cudaStreamSynchronize(st));
  }
}

}  // namespace

void run_side_stats(Series &s, const SideOut &out) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P, F = s.F, S = s.qmap.total_static;
  const int32_t sw = s.desc.static_window, nwin = sw > 0 ? F / sw : 0;
  // device results: [P] pixel sums, [2F] frame sums, [S] totals, [nwin*S] partials
  const size_t nout = (size_t)P + 2 * (size_t)F + S + (size_t)nwin * S;
  s.side_out.reserve(nout ? nout : 1, st);
  float *d_pix = s.side_out.p, *d_fs = d_pix + P, *d_tot = d_fs + 2 * (size_t)F,
        *d_part = d_tot + S;
  XG_CUDA(cudaMemsetAsync(s.side_out.p, 0, sizeof(float) * nout, st));
  const int bs = 256;
  if (s.dense_px) {
    k_row_sums<<<(P + bs - 1) / bs, bs, 0, st>>>(P, s.row_ptr.p, s.row_len.p, s.ev_val.p,
                                                  s.pixels_sum.p);
    XG_CHECK_LAUNCH();
  }
  k_pixel_sums<<<(P + bs - 1) / bs, bs, 0, st>>>(P, F, s.pixels_sum.p, d_pix);
  XG_CHECK_LAUNCH();
  // values that can only be photon counts take the integer pass; whether they
  // are is checked on the device
  const bool ints = F > 0 && !s.has_flat && s.desc.avg_frames == 1 &&
                    !(s.desc.dense && s.has_dark);
  SideInt si{};
  if (ints) {
    const size_t nfs = (size_t)F, npt = (size_t)(nwin + 1) * S;
    constexpr size_t head = sizeof(SideInt) / sizeof(uint32_t);
    s.side_cnt.reserve(head + nfs + npt, st);
    XG_CUDA(cudaMemsetAsync(s.side_cnt.p, 0, sizeof(uint32_t) * (head + nfs + npt), st));
    SideInt *dsi = (SideInt *)s.side_cnt.p;
    uint32_t *fs = s.side_cnt.p + head, *pt = fs + nfs;
    const bool pt_in = sizeof(uint32_t) * npt <= SI_SMEM / 4;
    const bool fs_in = sizeof(uint32_t) * (nfs + (pt_in ? npt : 0)) <= SI_SMEM;
    const size_t sm = sizeof(uint32_t) * ((fs_in ? nfs : 0) + (pt_in ? npt : 0));
    XG_CUDA(cudaFuncSetAttribute(k_side_int, cudaFuncAttributeMaxDynamicSharedMemorySize, SI_SMEM));
    int sms = 0;
    XG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.device));
    const int rows = SI_THREADS / 32;
    k_side_int<<<std::max(1, std::min(2 * sms, (P + rows - 1) / rows)), SI_THREADS, sm, st>>>(
        P, F, S, nwin, std::max(sw, 1), fs_in, pt_in, s.row_ptr.p, s.row_len.p, s.d_sbin.p,
        s.ev_frame.p, s.ev_val.p, fs, pt, dsi);
    XG_CHECK_LAUNCH();
    const int64_t no = std::max<int64_t>(F, std::max<int64_t>(S, (int64_t)S * nwin));
    k_side_int_out<<<(unsigned)((no + bs - 1) / bs), bs, 0, st>>>(P, F, S, nwin, std::max(sw, 1),
                                                                 fs, pt, s.d_ppb.p, s.stats.p, dsi,
                                                                 d_fs, d_tot, d_part);
    XG_CHECK_LAUNCH();
    XG_CUDA(cudaMemcpyAsync(&si, dsi, sizeof(si), cudaMemcpyDeviceToHost, st));
    XG_CUDA(cudaStreamSynchronize(st));
  }
  if (!ints || si.bad) side_ordered(s, nwin, d_fs, d_tot, d_part);
  if (out.pixel_sum)
    XG_CUDA(cudaMemcpyAsync(out.pixel_sum, d_pix, sizeof(float) * P, cudaMemcpyDeviceToHost, st));
  if (out.frame_sum)
    XG_CUDA(cudaMemcpyAsync(out.frame_sum, d_fs, sizeof(float) * 2 * (size_t)F, cudaMemcpyDeviceToHost, st));
  if (out.part_total)
    XG_CUDA(cudaMemcpyAsync(out.part_total, d_tot, sizeof(float) * S, cudaMemcpyDeviceToHost, st));
  if (out.part_partial && nwin)
    XG_CUDA(cudaMemcpyAsync(out.part_partial, d_part, sizeof(float) * (size_t)nwin * S,
                            cudaMemcpyDeviceToHost, st));
  XG_CUDA(cudaStreamSynchronize(st));
}

// normalize_by_framesum (main.cpp:314-337): divisor frameSum[F+f] / mean per
// frame, mean = the float sum of frameSum[F..2F) in frame order / F, computed
// in float on the host exactly as the reference does; the float multi-tau
// kernel divides every value by it when it loads the rows.
void prepare_framesum_scale(Series &s) {
  const int32_t F = s.F;
  std::vector<float> fs(2 * (size_t)F + 1);
  run_side_stats(s, SideOut{nullptr, fs.data(), nullptr, nullptr});
  float acc = 0.f;
  for (int32_t f = 0; f < F; f++) acc += fs[(size_t)F + f];
  const float mean = acc / (float)F;
  std::vector<float> q((size_t)F + 1, 1.f);
  for (int32_t f = 0; f < F; f++) q[f] = fs[(size_t)F + f] / mean;
  s.d_fscale.reserve(q.size(), s.stream);
  XG_CUDA(cudaMemcpyAsync(s.d_fscale.p, q.data(), sizeof(float) * q.size(),
                          cudaMemcpyHostToDevice, s.stream));
  XG_CUDA(cudaStreamSynchronize(s.stream));
}

}  // namespace xg
