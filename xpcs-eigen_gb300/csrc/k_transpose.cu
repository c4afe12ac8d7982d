// K-a: sparse-frame filter and pixel-major transpose.
//
// Replaces SparseFilter::Apply (src/xpcs/filter/sparse_filter.cpp:115-193),
// which walks every frame and pushes (frame, value) onto per-pixel std::vector
// rows.  Here the raw frame-major event stream (int32 pixel index, int16 value)
// is filtered and stably sorted by pixel with an LSD radix sort, so that every
// pixel's events come out contiguous and in stream order (frame order).
//
//   pass 0   reads the raw events directly: per event it derives the filter
//            frame (raw frame / (stride*avg), from a per-warp-chunk table of
//            raw frames and a per-raw-frame table of filter frames), drops
//            unused stride sub-frames and frames past the end (key = P, sorts
//            last), and forms v = (float)(value * flatfield) as the reference
//            does (sparse_filter.cpp:149-153).
//   pass k   7- or 8-bit digit k of the pixel index: tile histograms -> digit-major
//            exclusive scan -> stable scatter.  Ranking inside a tile uses
//            per-bit warp ballots + per-warp digit counters, so equal digits
//            keep stream order (tile, warp, round, lane).
//   merge    one warp per 32 pixels: events of the same filter frame are
//            summed in stream order and divided by avg (sparse_filter.cpp:
//            160-172), pixelSum is accumulated in frame order, pixels outside
//            the mask (sparse_filter.cpp:147) get empty rows, and every pixel
//            is classified for the multi-tau kernels.
#include <algorithm>
#include <cstddef>

#include "f64emu.cuh"
#include "classify.cuh"
#include "overlap.cuh"
#include "xpcs_internal.h"

namespace xg {
namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
// Items per lane: 8 (tiles of 2048) keeps more blocks resident; above
// RS_BIG_N events 16 (tiles of 4096) halves the tile histograms.
constexpr int64_t RS_BIG_N = (int64_t)1 << 27;
// Digits of 7 or 8 bits (DB): 7 wherever they need no pass more (keys of 9-14,
// 17-21 or 25-28 bits).  Half the digits halve the tile histograms and their
// scan, take a ballot less per item to rank and double a tile's runs of
// consecutive addresses.  A downsweep of 52 M items takes 312 / 269 / 254 us in
// the three passes (353 / 305 / 281 with 8 bits).
constexpr int RS_DIGITS_MAX = 256;
static_assert(RS_DIGITS_MAX <= RS_THREADS, "a thread per digit in the downsweep scan");

// The raw frames [r0, r0 + nframes) of a series: idx/val/valf start at their
// first event e0, frame_off/frame_map at r0, and frame_off holds absolute
// event offsets, so an event's index relative to e0 is compared with
// frame_off[r] - e0.
struct RawCfg {
  const int32_t *idx;
  const int16_t *val;   // sparse series: raw values (flatfield applied here)
  const float *valf;    // dense series: values already filtered by K-b
  const int64_t *frame_off;  // [nframes+1]
  const int32_t *frame_map;  // [nframes]: filter frame of a raw frame, -1 if unused
  const int32_t *chunk_frame;  // [ceil(n / chunk)]: raw frame of item chunk * c
  int32_t nframes;
  int64_t e0;
  int64_t n;
  int32_t P, F, R_in, stride;
  const double *flat;  // may be null
  DevStats *stats;
};

struct PassCfg {
  const uint32_t *key_in;
  const int32_t *fr_in;
  const float *v_in;
  uint32_t *key_out;  // null on the last pass
  int32_t *fr_out;
  float *v_out;
  int64_t n;
  int shift;
  int ntiles;       // tiles, and the row length of the digit-major histogram
  int hstride;      // (a multiple of 4)
  uint32_t sentinel;
};

// Per-pass workspace after the histogram: the digits' totals, then their
// first positions, then the count of scanned digits.
struct DigitSums {
  uint32_t total[RS_DIGITS_MAX], base[RS_DIGITS_MAX];
  uint32_t done;
};

// Raw frame of the first item of every chunk of 32 * IPT items (one warp's
// share of a tile): chunk c starts in frame r when off[r] - e0 <= chunk c <
// off[r + 1] - e0.
__global__ void k_chunk_frames(int32_t nframes, const int64_t *__restrict__ off, int64_t e0,
                               int64_t nchunks, int32_t chunk, int32_t *__restrict__ chunk_frame) {
  overlap_after();
  const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nframes) return;
  const int64_t c0 = (off[r] - e0 + chunk - 1) / chunk;
  const int64_t c1 = min((off[r + 1] - e0 + chunk - 1) / chunk, nchunks);
  for (int64_t c = c0; c < c1; c++) chunk_frame[c] = r;
}

// The raw loads of item i (pixel index and value), issued before any of the
// per-item work so that a lane's loads are in flight together.
__device__ __forceinline__ void raw_load(const RawCfg &c, int64_t i, int32_t &p, float &v) {
  p = c.idx[i];
  v = c.valf ? c.valf[i] : (float)c.val[i];
}

// Filter frame, sort key and filtered value of item i.  r is the raw frame of
// this lane's previous item, nb = frame_off[r + 1] and k = frame_map[r], kept
// in registers so that the common case (no frame boundary crossed) loads
// nothing.  Masked pixels keep their own key here; their rows are emptied by
// the merge, which reads the mask once per pixel instead of once per event.
__device__ __forceinline__ bool raw_frame_key(const RawCfg &c, int64_t i, int32_t &r, int64_t &nb,
                                              int32_t &k, int32_t p, uint32_t &key,
                                              int32_t &frame) {
  while (nb <= i) {
    r++;
    nb = c.frame_off[r + 1] - c.e0;
    k = c.frame_map[r];
  }
  frame = k;
  if (p < 0 || p >= c.P) {
    c.stats->error |= DEVERR_PIXEL_INDEX;
    key = (uint32_t)c.P;
    return false;
  }
  key = k >= 0 ? (uint32_t)p : (uint32_t)c.P;
  return true;
}

// (float)((double)v * g) as the reference forms a flat-fielded value,
// exactly, in integer arithmetic (f64emu.cuh)
__device__ __forceinline__ float flat_value(float v, double g) {
  float w;
  return f32_mul_f64(v, g, w) ? w : __double2float_rn(__dmul_rn((double)v, g));
}

__device__ __forceinline__ void raw_key(const RawCfg &c, int64_t i, int32_t &r, int64_t &nb,
                                        int32_t &k, int32_t p, float &v, uint32_t &key,
                                        int32_t &frame) {
  if (!raw_frame_key(c, i, r, nb, k, p, key, frame)) {
    v = 0.f;
    return;
  }
  if (!c.valf && c.flat) v = flat_value(v, c.flat[p]);
}

// Packed items (sparse series with fewer than 65,536 filter frames): filter
// frame in the high half, the raw int16 value in the low half.  The flatfield
// is applied when the last pass writes the events out.
__device__ __forceinline__ int32_t pack_item(int32_t frame, float raw) {
  return (int32_t)(((uint32_t)frame << 16) | ((uint32_t)(int32_t)raw & 0xffffu));
}

// Item i of a tile in warp-striped order: warp w owns [w*32*IPT, (w+1)*32*IPT),
// round k, lane l -> w*32*IPT + k*32 + l.
template <int IPT>
__device__ __forceinline__ int64_t item_index(int tile, int w, int k, int lane) {
  return (int64_t)tile * (RS_THREADS * IPT) + (int64_t)w * 32 * IPT + k * 32 + lane;
}

template <int IPT, int DB, bool FIRST>
__global__ void __launch_bounds__(RS_THREADS)
k_upsweep(RawCfg rc, PassCfg pc, uint32_t *__restrict__ hist, DigitSums *__restrict__ ds) {
  overlap_after();
  constexpr int RS_DIGITS = 1 << DB;
  __shared__ uint32_t h[RS_DIGITS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tile = blockIdx.x;
  if (tile == 0 && threadIdx.x == 0) ds->done = 0;  // for the pass's digit scan
  for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS) h[d] = 0;
  __syncthreads();
  uint32_t key[IPT];
  // all loads first, so that they are in flight together
  if (FIRST) {
    const int64_t nch = (rc.n + 32 * IPT - 1) / (32 * IPT);
    int32_t r = rc.chunk_frame[min((int64_t)tile * RS_WARPS + w, nch - 1)];
    int64_t nb = rc.frame_off[r + 1] - rc.e0;
    int32_t kf = rc.frame_map[r];
    int32_t pix[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      const int64_t i = item_index<IPT>(tile, w, k, lane);
      pix[k] = i < pc.n ? rc.idx[i] : 0;
    }
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      int64_t i = item_index<IPT>(tile, w, k, lane);
      key[k] = 0xffffffffu;
      if (i < pc.n) {
        while (nb <= i) {
          r++;
          nb = rc.frame_off[r + 1] - rc.e0;
          kf = rc.frame_map[r];
        }
        const int32_t p = pix[k];
        key[k] = (p < 0 || p >= rc.P || kf < 0) ? (uint32_t)rc.P : (uint32_t)p;
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      int64_t i = item_index<IPT>(tile, w, k, lane);
      key[k] = i < pc.n ? pc.key_in[i] : 0xffffffffu;
    }
  }
  int dropped = 0;  // items that sort last: their count gives the kept total
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    if (key[k] == 0xffffffffu) continue;
    if (FIRST && key[k] == pc.sentinel) dropped++;
    atomicAdd(&h[(key[k] >> pc.shift) & (RS_DIGITS - 1)], 1u);
  }
  if (FIRST) {
    dropped = __reduce_add_sync(0xffffffffu, dropped);
    if (lane == 0 && dropped) atomicAdd(&rc.stats->dropped, (unsigned long long)dropped);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS)
    hist[(int64_t)d * pc.hstride + tile] = h[d];
}

// One block per digit: the exclusive scan of its tile counts, in place, and
// its total; the last block to finish turns the totals into the digits' first
// positions.  One launch per pass instead of the three of a device-wide scan:
// 12 us at 25,469 tiles (42 before, with twice the digits), 5 us at 1,204 (12).
constexpr int DSC_THREADS = 1024;
constexpr int DSC_IPT = 8;
__global__ void __launch_bounds__(DSC_THREADS)
k_digit_scan(int digits, int ntiles, int hstride, uint32_t *__restrict__ hist,
             DigitSums *__restrict__ ds) {
  overlap_after();
  __shared__ uint32_t wsum[DSC_THREADS / 32];
  __shared__ bool last;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t *row = hist + (int64_t)blockIdx.x * hstride;
  uint32_t carry = 0;
  for (int base = 0; base < ntiles; base += DSC_THREADS * DSC_IPT) {
    const int i = base + threadIdx.x * DSC_IPT;
    uint32_t v[DSC_IPT];
#pragma unroll
    for (int k = 0; k < DSC_IPT; k += 4) {  // rows are 16-byte aligned, hstride a multiple of 4
      const uint4 x = i + k < hstride ? *(const uint4 *)(row + i + k) : make_uint4(0u, 0u, 0u, 0u);
      v[k] = x.x;
      v[k + 1] = x.y;
      v[k + 2] = x.z;
      v[k + 3] = x.w;
    }
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < DSC_IPT; k++) {
      if (i + k >= ntiles) v[k] = 0;  // the row's padding is not written by the upsweep
      const uint32_t c = v[k];
      v[k] = s;
      s += c;
    }
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t y = wsum[lane];  // DSC_THREADS / 32 == 32 warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t z = __shfl_up_sync(FULL, y, o);
      if (lane >= o) y += z;
    }
    const uint32_t before = w ? __shfl_sync(FULL, y, w - 1) : 0u;
    const uint32_t all = __shfl_sync(FULL, y, 31);
    const uint32_t off = carry + before + x - s;
#pragma unroll
    for (int k = 0; k < DSC_IPT; k += 4)
      if (i + k < hstride)
        *(uint4 *)(row + i + k) =
            make_uint4(off + v[k], off + v[k + 1], off + v[k + 2], off + v[k + 3]);
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    ds->total[blockIdx.x] = carry;
    __threadfence();
    last = atomicAdd(&ds->done, 1u) == (uint32_t)digits - 1u;
  }
  __syncthreads();
  if (!last || w != 0) return;
  __threadfence();
  uint32_t run = 0;
  for (int d0 = 0; d0 < digits; d0 += 32) {
    const uint32_t c = ((volatile uint32_t *)ds->total)[d0 + lane];
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    ds->base[d0 + lane] = run + x - c;
    run += __shfl_sync(FULL, x, 31);
  }
}

// Shared memory of the downsweep: per-warp digit counters, the tile's global
// and local digit offsets, and the tile staged in digit order.
template <int IPT, int DB, bool PK>
struct DsSmem {
  uint32_t wcnt[RS_WARPS][1 << DB];
  uint32_t toff[1 << DB];
  uint32_t tstart[1 << DB];
  uint32_t wtot[RS_THREADS / 32];
  uint32_t key[RS_THREADS * IPT];
  int32_t fr[RS_THREADS * IPT];      // frame, or the packed item
  float v[PK ? 1 : RS_THREADS * IPT];
};

template <int IPT, int DB, bool FIRST, bool LAST, bool PK>
__global__ void __launch_bounds__(RS_THREADS)
k_downsweep(RawCfg rc, PassCfg pc, const uint32_t *__restrict__ offsets,
            const DigitSums *__restrict__ dsum) {
  overlap_after();
  constexpr int RS_DIGITS = 1 << DB;
  extern __shared__ __align__(16) uint8_t ds_raw[];
  DsSmem<IPT, DB, PK> &sm = *reinterpret_cast<DsSmem<IPT, DB, PK> *>(ds_raw);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tile = blockIdx.x;
  for (int d = lane; d < RS_DIGITS; d += 32) sm.wcnt[w][d] = 0;
  for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS)
    sm.toff[d] = offsets[(int64_t)d * pc.hstride + tile] + dsum->base[d];
  __syncwarp();

  uint32_t key[IPT];
  int32_t fr[IPT];
  float v[IPT];
  uint32_t rank[IPT];
  const unsigned lt = (1u << lane) - 1u;
  // all loads first, so that they are in flight together
  if (FIRST) {
    const int64_t nch = (rc.n + 32 * IPT - 1) / (32 * IPT);
    int32_t r = rc.chunk_frame[min((int64_t)tile * RS_WARPS + w, nch - 1)];
    int64_t nb = rc.frame_off[r + 1] - rc.e0;
    int32_t kf = rc.frame_map[r];
    int32_t pix[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      const int64_t i = item_index<IPT>(tile, w, k, lane);
      pix[k] = 0;
      v[k] = 0.f;
      if (i < pc.n) raw_load(rc, i, pix[k], v[k]);
    }
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      const int64_t i = item_index<IPT>(tile, w, k, lane);
      key[k] = 0xffffffffu;
      fr[k] = 0;
      if (i < pc.n) {
        if (PK) {
          raw_frame_key(rc, i, r, nb, kf, pix[k], key[k], fr[k]);
          fr[k] = pack_item(fr[k], v[k]);
        } else {
          raw_key(rc, i, r, nb, kf, pix[k], v[k], key[k], fr[k]);
        }
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < IPT; k++) {
      int64_t i = item_index<IPT>(tile, w, k, lane);
      key[k] = 0xffffffffu;
      fr[k] = 0;
      v[k] = 0.f;
      if (i < pc.n) {
        key[k] = pc.key_in[i];
        fr[k] = pc.fr_in[i];
        if (!PK) v[k] = pc.v_in[i];
      }
    }
  }
  // stable rank within the warp: equal digits keep (round, lane) order
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    const bool ok = key[k] != 0xffffffffu;
    uint32_t d = ok ? ((key[k] >> pc.shift) & (RS_DIGITS - 1)) : RS_DIGITS;
    // lanes with the same digit (and the invalid marker's bit), one ballot per
    // bit: cheaper here than match_any
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b <= DB; b++) {
      const bool bit = (d >> b) & 1u;
      const unsigned bal = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? bal : ~bal;
    }
    int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (ok && lane == leader) {
      base = sm.wcnt[w][d];
      sm.wcnt[w][d] = base + __popc(peers);
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    rank[k] = base + __popc(peers & lt);
  }
  __syncthreads();
  // per digit: exclusive over warps; tile total -> tile-local digit starts
  {
    const int d = threadIdx.x;  // whole warps of digits
    uint32_t run = 0, x = 0;
    if (d < RS_DIGITS) {
#pragma unroll
      for (int ww = 0; ww < RS_WARPS; ww++) {
        uint32_t c = sm.wcnt[ww][d];
        sm.wcnt[ww][d] = run;
        run += c;
      }
      x = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
    }
    if (lane == 31) sm.wtot[w] = x;  // 0 past the digits
    __syncthreads();
    uint32_t before = 0;
    for (int ww = 0; ww < w; ww++) before += sm.wtot[ww];
    if (d < RS_DIGITS) sm.tstart[d] = before + x - run;
  }
  __syncthreads();
  // stage the tile in digit order
#pragma unroll
  for (int k = 0; k < IPT; k++) {
    if (key[k] == 0xffffffffu) continue;
    const uint32_t d = (key[k] >> pc.shift) & (RS_DIGITS - 1);
    const uint32_t q = sm.tstart[d] + sm.wcnt[w][d] + rank[k];
    sm.key[q] = key[k];
    sm.fr[q] = fr[k];
    if (!PK) sm.v[q] = v[k];
  }
  __syncthreads();
  // write out: consecutive staged elements of a digit go to consecutive addresses
  uint32_t nvalid = 0;
#pragma unroll
  for (int ww = 0; ww < RS_THREADS / 32; ww++) nvalid += sm.wtot[ww];
  for (uint32_t q = threadIdx.x; q < nvalid; q += RS_THREADS) {
    const uint32_t kq = sm.key[q];
    if (LAST && kq == pc.sentinel) continue;
    const uint32_t d = (kq >> pc.shift) & (RS_DIGITS - 1);
    const uint32_t pos = sm.toff[d] + (q - sm.tstart[d]);
    if (!LAST || pc.key_out) pc.key_out[pos] = kq;
    if (PK && LAST) {
      const uint32_t it = (uint32_t)sm.fr[q];
      const float raw = (float)(int16_t)(it & 0xffffu);
      pc.fr_out[pos] = (int32_t)(it >> 16);
      pc.v_out[pos] = rc.flat ? flat_value(raw, rc.flat[kq]) : raw;
    } else {
      pc.fr_out[pos] = sm.fr[q];
      if (!PK) pc.v_out[pos] = sm.v[q];
    }
  }
}

// Row pointers from the sorted keys: row_ptr[p] = the first position whose key
// is >= p (std::lower_bound over the kept items), row_ptr[P] = the kept total.
// One pass over the keys, 512 per warp in four 16-byte loads a lane: where the
// key changes, the rows up to it start there; a warp fills longer gaps (rows
// without events) together.  Bound by HBM: 4 B per event read.  One binary
// search per pixel took 64 us at 49.6 M events in 1 Mi pixels and 12 at 2.5 M
// in 512^2, this pass 64 and 9.
// One warp fills 7,600 rows of a gap in a microsecond, too few where most of a
// large detector is one gap (events in one corner, or none kept): the filter of
// 20,000 events on 4,096 x 4,096 pixels took 2.84 ms so, 0.65 with the events
// all over the detector, and as long as that now.  So the grid's first gap_blocks take the rows in
// aligned spans of RP_SPAN, a warp each, and fill those that lie in one gap
// (two binary searches tell); the warp that finds the gap leaves them out.
constexpr int RP_U = 4;
constexpr int RP_SPAN = 4096;
__device__ __forceinline__ int64_t first_key(const uint32_t *__restrict__ keys, int64_t n,
                                             int32_t p) {  // the first that is >= p
  int64_t first = 0;
  while (n > 0) {
    const int64_t h = n >> 1;
    if ((int32_t)keys[first + h] < p) {
      first += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return first;
}
__global__ void __launch_bounds__(256)
k_row_ptr(const uint32_t *__restrict__ keys, int64_t n, const DevStats *__restrict__ stats,
          int32_t P, int32_t gap_blocks, int64_t *__restrict__ row_ptr) {
  overlap_after();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t nv = n - (int64_t)stats->dropped;
  if ((int)blockIdx.x < gap_blocks) {
    const int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RP_SPAN;
    if (p0 + RP_SPAN - 1 > P) return;  // rows 0 .. P
    const int64_t at = first_key(keys, nv, (int32_t)p0 + (lane & 1) * (RP_SPAN - 1));
    const int64_t pos = __shfl_sync(FULL, at, 0);
    if (pos != __shfl_sync(FULL, at, 1)) return;
    for (int k = lane; k < RP_SPAN; k += 32) row_ptr[p0 + k] = pos;
    return;
  }
  // the warp's first key; position nv is the end of the last rows
  const int64_t w0 =
      (((int64_t)(blockIdx.x - gap_blocks) * blockDim.x + threadIdx.x) >> 5) * (RP_U * 128);
  if (w0 > nv) return;
  int32_t key[RP_U][5];  // keys i0 - 1 .. i0 + 3 of a group: -1 before the first, P past the end
#pragma unroll
  for (int u = 0; u < RP_U; u++) {
    const int64_t i0 = w0 + u * 128 + lane * 4;
    if (i0 + 3 < nv) {
      const uint4 x = *(const uint4 *)(keys + i0);
      key[u][1] = (int32_t)x.x;
      key[u][2] = (int32_t)x.y;
      key[u][3] = (int32_t)x.z;
      key[u][4] = (int32_t)x.w;
    } else {
#pragma unroll
      for (int k = 1; k < 5; k++) key[u][k] = i0 - 1 + k < nv ? (int32_t)keys[i0 - 1 + k] : P;
    }
  }
  int32_t before = w0 > 0 ? (int32_t)keys[w0 - 1] : -1;
#pragma unroll
  for (int u = 0; u < RP_U; u++) {
    const int64_t i0 = w0 + u * 128 + lane * 4;
    key[u][0] = __shfl_up_sync(FULL, key[u][4], 1);
    if (lane == 0) key[u][0] = before;
    before = __shfl_sync(FULL, key[u][4], 31);
    // rows (key[k - 1], key[k]] start at position i0 - 1 + k; most lanes see no
    // change
    if (key[u][4] != key[u][0]) {
#pragma unroll
      for (int k = 1; k < 5; k++)
        if (key[u][k] - key[u][k - 1] <= 8)
          for (int32_t p = key[u][k - 1] + 1; p <= key[u][k]; p++) row_ptr[p] = i0 - 1 + k;
    }
    if (!__any_sync(FULL, key[u][4] - key[u][0] > 8)) continue;
#pragma unroll
    for (int k = 1; k < 5; k++) {
      unsigned big = __ballot_sync(FULL, key[u][k] - key[u][k - 1] > 8);
      while (big) {
        const int l = __ffs(big) - 1;
        big &= big - 1u;
        const int32_t a = __shfl_sync(FULL, key[u][k - 1], l);
        const int32_t e = __shfl_sync(FULL, key[u][k], l);
        const int64_t pos = __shfl_sync(FULL, i0 - 1 + k, l);
        // whole spans [s0, s1) of the gap's rows a + 1 .. e are the gap blocks'
        int32_t s0 = e + 1, s1 = e + 1;
        if (gap_blocks) {
          s0 = min((a + RP_SPAN) / RP_SPAN * RP_SPAN, e + 1);
          s1 = max((e + 1) / RP_SPAN * RP_SPAN, s0);
        }
        for (int32_t p = a + 1 + lane; p < s0; p += 32) row_ptr[p] = pos;
        for (int32_t p = s1 + lane; p <= e; p += 32) row_ptr[p] = pos;
      }
    }
  }
}

// The events of one row (b, n) merged in place by a warp: events of the same
// filter frame summed in stream order as pixels_value_[pix] += v, then / avg
// (sparse_filter.cpp:146-172); psum: the merged values summed in frame order.
// A group that reaches the end of a 32-event chunk stays open (its frame and
// sum so far) until the next chunk.  The same results in every lane, except
// total, which each lane holds its share of (saturating at 2^24).
__device__ __forceinline__ void merge_row(int64_t b, int32_t n, float favg,
                                          int32_t *__restrict__ fr, float *__restrict__ val,
                                          int32_t &out, bool &integral, uint32_t &total,
                                          float &psum) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  out = 0;
  integral = true;
  total = 0;
  psum = 0.f;
  int32_t cf = -1;  // the open group
  float ca = 0.f;
  const auto count = [&](float x, bool mine) {
    if (!mine) return;
    if (x == truncf(x) && fabsf(x) < 16777216.f)
      total = min(total + (uint32_t)fabsf(x), 1u << 24);
    else
      integral = false;
  };
  int32_t f_nx = lane < n ? fr[b + lane] : -1;
  float x_nx = lane < n ? val[b + lane] : 0.f;
  for (int32_t i0 = 0; i0 < n; i0 += 32) {
    const int32_t f = f_nx;
    float x = x_nx;
    const bool in = i0 + lane < n;
    f_nx = i0 + 32 + lane < n ? fr[b + i0 + 32 + lane] : -1;
    x_nx = i0 + 32 + lane < n ? val[b + i0 + 32 + lane] : 0.f;
    const int cnt = min(32, n - i0);
    // the open group's events at the chunk's start
    const unsigned other = __ballot_sync(FULL, !in || f != cf);
    const int lead = other ? __ffs(other) - 1 : 32;
    for (int k = 0; k < lead; k++) ca = __fadd_rn(ca, __shfl_sync(FULL, x, k));
    if (lead == cnt) continue;  // only possible with events left in the group or row
    if (cf >= 0) {
      const float v = __fdiv_rn(ca, favg);
      if (lane == 0) {
        fr[b + out] = cf;
        val[b + out] = v;
      }
      count(v, lane == 0);
      psum = __fadd_rn(psum, v);
      out++;
    }
    // groups that start in this chunk
    const int32_t fp = __shfl_up_sync(FULL, f, 1);
    const bool head = in && lane >= lead && (lane == lead || f != fp);
    const unsigned heads = __ballot_sync(FULL, head);
    const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
    const int run = head ? (after ? __ffs(after) : cnt - lane) : 0;
    const int longest = __reduce_max_sync(FULL, run);
    float acc = __fadd_rn(0.f, x);
    for (int k = 1; k < longest; k++) {
      const float y = __shfl_down_sync(FULL, x, k);
      if (k < run) acc = __fadd_rn(acc, y);
    }
    const int last = 31 - __clz(heads);  // stays open
    cf = __shfl_sync(FULL, f, last);
    ca = __shfl_sync(FULL, acc, last);
    const unsigned done = heads & ~(1u << last);
    const float v = __fdiv_rn(acc, favg);
    const bool emit = done >> lane & 1u;
    __syncwarp();
    if (emit) {
      const int32_t o = out + __popc(done & ((1u << lane) - 1u));
      fr[b + o] = f;
      val[b + o] = v;
    }
    count(v, emit);
    for (unsigned m = done; m; m &= m - 1u)
      psum = __fadd_rn(psum, __shfl_sync(FULL, v, __ffs(m) - 1));
    out += __popc(done);
  }
  if (cf >= 0) {
    const float v = __fdiv_rn(ca, favg);
    if (lane == 0) {
      fr[b + out] = cf;
      val[b + out] = v;
    }
    count(v, lane == 0);
    psum = __fadd_rn(psum, v);
    out++;
  }
  integral = __all_sync(FULL, integral);
}

constexpr int MC_WARPS = 4;             // warps per block of 32 pixels
constexpr int MC_ROWS = 32 / MC_WARPS;  // rows per warp

// Long rows, and rows to merge.  One block per 32 consecutive pixels, 8 rows
// per warp, a warp's lanes over a row's events: repeated frames, whether every
// value is an integer, sum |v| and sum v are found in one pass (the next
// chunk, of this row or the next, in flight), reduced once per row.  Without
// duplicates and with avg == 1 the row is final as sorted, and for integer
// rows with sum |v| < 2^24 every float partial sum of pixelSum is exact, so
// pixelSum = (float)sum v; otherwise the row is merged / summed in frame
// order.  Pixels outside the mask get empty rows.  The block's first warp
// classifies the 32 pixels.
__global__ void __launch_bounds__(MC_WARPS * 32)
k_merge_rows(int32_t P, int32_t F, int32_t avg, int32_t tcap, int32_t fcap,
                 int32_t force_float,
                 const int64_t *__restrict__ row_ptr, const uint8_t *__restrict__ mask,
                 int32_t *__restrict__ fr, float *__restrict__ val, int32_t *__restrict__ row_len,
                 uint8_t *__restrict__ pclass, ClassLists cl, float *__restrict__ pixels_sum,
                 DevStats *__restrict__ stats) {
  overlap_after();
  __shared__ int32_t s_len[32];
  __shared__ uint8_t s_cls[32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int pb = blockIdx.x * 32, p0 = pb + w * MC_ROWS;
  int64_t my_b = 0;
  int32_t my_n = 0;
  if (lane < MC_ROWS && p0 + lane < P && mask[p0 + lane]) {
    my_b = row_ptr[p0 + lane];
    my_n = (int32_t)(row_ptr[p0 + lane + 1] - my_b);
  }
  if (lane < MC_ROWS) {  // rows without events
    s_len[w * MC_ROWS + lane] = 0;
    s_cls[w * MC_ROWS + lane] = PCLASS_EMPTY;
    if (p0 + lane < P && my_n == 0) pixels_sum[p0 + lane] = 0.f;
  }
  __syncwarp();
  unsigned rows = __ballot_sync(FULL, my_n > 0);
  int q = rows ? __ffs(rows) - 1 : 0;
  int64_t b = __shfl_sync(FULL, my_b, q);
  int32_t n = __shfl_sync(FULL, my_n, q), i0 = 0;
  int32_t f = lane < n ? fr[b + lane] : -1;
  float x = lane < n ? val[b + lane] : 0.f;
  int32_t last_f = -1;  // the previous chunk's last frame
  bool dup = false, nonint = false;
  uint32_t total = 0;  // this lane's share, saturating at 2^24
  int32_t sum = 0;     // exact while the total is below 2^24
  while (rows) {
    const bool in = i0 + lane < n;
    const int32_t fc = f;
    const float xc = x;
    const int32_t nc = n;
    const int64_t bc = b;
    const int qc = q;
    const bool end = i0 + 32 >= n;  // the row's last chunk
    i0 += 32;
    if (end) {
      rows &= rows - 1u;
      q = rows ? __ffs(rows) - 1 : 0;
      b = __shfl_sync(FULL, my_b, q);
      n = rows ? __shfl_sync(FULL, my_n, q) : 0;
      i0 = 0;
    }
    f = i0 + lane < n ? fr[b + i0 + lane] : -1;
    x = i0 + lane < n ? val[b + i0 + lane] : 0.f;
    int32_t fp = __shfl_up_sync(FULL, fc, 1);
    if (lane == 0) fp = last_f;
    if (in) {
      dup = dup || fc == fp;
      const bool ni = !(xc == truncf(xc) && fabsf(xc) < 16777216.f);
      nonint = nonint || ni;
      if (!ni) {
        total = min(total + (uint32_t)fabsf(xc), 1u << 24);
        sum += (int32_t)xc;
      }
    }
    if (!end) {
      last_f = __shfl_sync(FULL, fc, 31);
      continue;
    }
    int32_t out = nc;
    bool integral = !__any_sync(FULL, nonint);
    float psum = 0.f;
    if (__any_sync(FULL, dup) || avg != 1) {
      merge_row(bc, nc, (float)avg, fr, val, out, integral, total, psum);
      total = __reduce_add_sync(FULL, total);
    } else {
      total = __reduce_add_sync(FULL, total);
      if (integral && total < 16777216u) {
        psum = (float)__reduce_add_sync(FULL, sum);
      } else {
        for (int32_t j0 = 0; j0 < nc; j0 += 32) {
          const float y = j0 + lane < nc ? val[bc + j0 + lane] : 0.f;
          const int m = min(32, nc - j0);
          if (m == 32) {
#pragma unroll
            for (int k = 0; k < 32; k++) psum = __fadd_rn(psum, __shfl_sync(FULL, y, k));
          } else {
            for (int k = 0; k < m; k++) psum = __fadd_rn(psum, __shfl_sync(FULL, y, k));
          }
        }
      }
    }
    if (lane == 0) {
      uint8_t c = pixel_class(out, integral, total, F, tcap);
      if (force_float && c != PCLASS_EMPTY) c = PCLASS_FLOAT;  // values rescaled after the filter
      s_len[w * MC_ROWS + qc] = out;
      s_cls[w * MC_ROWS + qc] = float_class(c, out, fcap);
      pixels_sum[p0 + qc] = psum;
    }
    last_f = -1;
    dup = nonint = false;
    total = 0;
    sum = 0;
  }
  __syncthreads();
  if (w == 0) {
    const int p = pb + lane;
    const bool has = p < P;
    if (has) row_len[p] = s_len[lane];
    record_class_warp(has, p, s_cls[lane], s_len[lane], pclass, cl, stats);
  }
}

// Short rows.  One warp per 32 consecutive pixels, whose rows are contiguous:
// tiles of 1,024 events are read coalesced, repeated frames are found between
// neighbouring events (a bit per row start tells which neighbours share a
// row), and the values go to shared memory, where each lane adds up its own
// row in order: the running sum is pixelSum as the reference forms it, and
// sum |v|, exact below 2^24, classifies the row.  A warp that finds a repeated
// frame merges its rows one by one.  Pixels outside the mask get empty rows.
// Bound by instruction issue, about 6 per event and row of a lane; a warp's
// former walk of the events in chunks that straddle rows searched every
// event's row and reduced three sums per run, 155 instructions a chunk (times
// at merge_classify).
constexpr int MS_TILE = 1024;
constexpr int MS_WARPS = 8;
constexpr double MS_MEAN_MAX = 256.0;  // see merge_classify
__global__ void __launch_bounds__(MS_WARPS * 32)
k_merge_short(int32_t P, int32_t F, int32_t tcap, int32_t fcap, int32_t force_float,
              const int64_t *__restrict__ row_ptr, const uint8_t *__restrict__ mask,
              int32_t *__restrict__ fr, float *__restrict__ val, int32_t *__restrict__ row_len,
              uint8_t *__restrict__ pclass, ClassLists cl, float *__restrict__ pixels_sum,
              DevStats *__restrict__ stats) {
  overlap_after();
  __shared__ float s_val[MS_WARPS][MS_TILE];
  __shared__ uint32_t s_start[MS_WARPS][MS_TILE / 32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p0 = (blockIdx.x * MS_WARPS + w) * 32;
  if (p0 >= P) return;
  const int p = p0 + lane;
  const bool has = p < P, keep = has && mask[p] != 0;
  const int64_t e0 = row_ptr[p0], e1 = row_ptr[min(p0 + 32, P)];
  const int64_t my_b = has ? row_ptr[p] : e1;
  const int64_t my_e = has ? row_ptr[p + 1] : e1;
  float *tile = s_val[w];
  uint32_t *start = s_start[w];
  float total = 0.f, psum = 0.f;
  bool dup = false, nonint = false;
  int32_t last_f = -1;
  for (int64_t t0 = e0; t0 < e1; t0 += MS_TILE) {
    const int n = (int)min((int64_t)MS_TILE, e1 - t0);
    __syncwarp();
    start[lane] = 0u;
    __syncwarp();
    if (my_b >= t0 && my_b < t0 + n)
      atomicOr(&start[(int)(my_b - t0) >> 5], 1u << ((int)(my_b - t0) & 31));
    __syncwarp();
    for (int c0 = 0; c0 * 32 < n; c0 += 4) {
      int32_t f[4];
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {  // the loads first, in flight together
        const int i = (c0 + u) * 32 + lane;
        f[u] = i < n ? fr[t0 + i] : -1;
        x[u] = i < n ? val[t0 + i] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int i = (c0 + u) * 32 + lane;
        int32_t fp = __shfl_up_sync(FULL, f[u], 1);
        if (lane == 0) fp = last_f;
        last_f = __shfl_sync(FULL, f[u], 31);
        if (i < n) {
          dup = dup || (f[u] == fp && !(start[c0 + u] >> lane & 1u));
          tile[i] = x[u];
        }
      }
    }
    __syncwarp();
    const int i0 = (int)(max(my_b, t0) - t0), i1 = (int)(min(my_e, t0 + n) - t0);
    for (int i = i0; i < i1; i++) {
      const float x = tile[i];
      total = __fadd_rn(total, fabsf(x));
      psum = __fadd_rn(psum, x);
      nonint = nonint || x != truncf(x);
    }
  }
  int32_t out = keep ? (int32_t)(my_e - my_b) : 0;
  bool integral = !nonint;
  // sum |v| as an integer: exact below 2^24, and only compared with less above
  long long tot = total < 16777216.f ? (long long)total : 1ll << 24;
  if (__any_sync(FULL, dup)) {
    unsigned rows = __ballot_sync(FULL, out > 0);
    while (rows) {
      const int q = __ffs(rows) - 1;
      rows &= rows - 1u;
      int32_t o;
      bool in;
      uint32_t share;
      float ps;
      merge_row(__shfl_sync(FULL, my_b, q), __shfl_sync(FULL, out, q), 1.f, fr, val, o, in, share,
                ps);
      share = __reduce_add_sync(FULL, share);
      if (lane == q) {
        out = o;
        integral = in;
        tot = share;
        psum = ps;
      }
    }
  }
  if (has) {
    row_len[p] = out;
    pixels_sum[p] = keep ? psum : 0.f;
  }
  uint8_t c = keep ? pixel_class(out, integral, tot, F, tcap) : (uint8_t)PCLASS_EMPTY;
  if (force_float && c != PCLASS_EMPTY) c = PCLASS_FLOAT;  // values rescaled after the filter
  record_class_warp(has, p, float_class(c, out, fcap), out, pclass, cl, stats);
}

template <int IPT, int DB, bool FIRST, bool LAST, bool PK>
void launch_downsweep(Series &s, int ntiles, const RawCfg &rc, const PassCfg &pc,
                      const DigitSums *ds) {
  const size_t smem = sizeof(DsSmem<IPT, DB, PK>);
  XG_CUDA(cudaFuncSetAttribute(k_downsweep<IPT, DB, FIRST, LAST, PK>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_overlapped(k_downsweep<IPT, DB, FIRST, LAST, PK>, ntiles, RS_THREADS, smem, s.stream, rc,
                    pc, s.hist.p, ds);
}

// One radix pass: tile histograms, digit-major scan, stable scatter.
template <int IPT, int DB, bool PK>
void radix_pass(Series &s, bool first, bool last, const RawCfg &rc, PassCfg pc) {
  cudaStream_t st = s.stream;
  const int ntiles = pc.ntiles;
  pc.hstride = (ntiles + 3) & ~3;
  DigitSums *ds = (DigitSums *)(s.hist.p + ((size_t)pc.hstride << DB));
  launch_overlapped(first ? k_upsweep<IPT, DB, true> : k_upsweep<IPT, DB, false>, ntiles,
                    RS_THREADS, 0, st, rc, pc, s.hist.p, ds);
  launch_overlapped(k_digit_scan, 1 << DB, DSC_THREADS, 0, st, 1 << DB, ntiles, pc.hstride,
                    s.hist.p, ds);
  if (first && last)
    launch_downsweep<IPT, DB, true, true, PK>(s, ntiles, rc, pc, ds);
  else if (first)
    launch_downsweep<IPT, DB, true, false, PK>(s, ntiles, rc, pc, ds);
  else if (last)
    launch_downsweep<IPT, DB, false, true, PK>(s, ntiles, rc, pc, ds);
  else
    launch_downsweep<IPT, DB, false, false, PK>(s, ntiles, rc, pc, ds);
  XG_CHECK_LAUNCH();
}

// Passes and digit bits for keys of nbits bits.
struct Digits {
  int passes, bits;
};
Digits digits_for(int nbits) {
  const int passes = (nbits + 7) / 8;
  return {passes, nbits <= 7 * passes ? 7 : 8};
}

void radix_pass(Series &s, int ipt, int bits, bool packed, bool first, bool last, const RawCfg &rc,
                const PassCfg &pc) {
  if (packed) {
    if (ipt == 16)
      bits == 7 ? radix_pass<16, 7, true>(s, first, last, rc, pc)
                : radix_pass<16, 8, true>(s, first, last, rc, pc);
    else
      bits == 7 ? radix_pass<8, 7, true>(s, first, last, rc, pc)
                : radix_pass<8, 8, true>(s, first, last, rc, pc);
  } else {
    if (ipt == 16)
      bits == 7 ? radix_pass<16, 7, false>(s, first, last, rc, pc)
                : radix_pass<16, 8, false>(s, first, last, rc, pc);
    else
      bits == 7 ? radix_pass<8, 7, false>(s, first, last, rc, pc)
                : radix_pass<8, 8, false>(s, first, last, rc, pc);
  }
}

int items_per_lane(int64_t n) { return n >= RS_BIG_N ? 16 : 8; }

}  // namespace

// The histogram of a pass over n items, its rows padded to 16 bytes, and the
// digits' sums: sized for 8-bit digits and tiles of 8 items per lane whichever
// a sort takes.  A series' sorts by other keys (side statistics, two-time
// lists) have their own digits and tiles but never more items than its
// transpose, so that none of them moves the buffer under a captured batch.
size_t radix_hist_words(int64_t n) {
  const int64_t tiles = (n + RS_THREADS * 8 - 1) / (RS_THREADS * 8);
  return (size_t)((tiles + 3) & ~(int64_t)3) * RS_DIGITS_MAX +
         sizeof(DigitSums) / sizeof(uint32_t);
}

// Stable LSD radix sort of (key, a, b) triples by the low `key_bits` bits of
// key, with the passes above; (key2, a2, b2) is scratch of the same length.
// Returns true when the sorted triples ended in the scratch arrays.
bool radix_sort_triples(Series &s, uint32_t *key, int32_t *a, float *b, uint32_t *key2,
                        int32_t *a2, float *b2, int64_t n, int key_bits) {
  if (n <= 0 || key_bits <= 0) return false;
  const Digits dg = digits_for(key_bits);
  const int passes = dg.passes;
  const int ipt = items_per_lane(n);
  const int ntiles = (int)((n + RS_THREADS * ipt - 1) / (RS_THREADS * ipt));
  s.hist.reserve(radix_hist_words(n), s.stream);
  RawCfg rc{};
  uint32_t *kb[2] = {key, key2};
  int32_t *ab[2] = {a, a2};
  float *bb[2] = {b, b2};
  for (int pass = 0; pass < passes; pass++) {
    PassCfg pc{};
    pc.n = n;
    pc.shift = dg.bits * pass;
    pc.ntiles = ntiles;
    pc.sentinel = 0xfffffffeu;
    pc.key_in = kb[pass & 1];
    pc.fr_in = ab[pass & 1];
    pc.v_in = bb[pass & 1];
    pc.key_out = kb[(pass + 1) & 1];
    pc.fr_out = ab[(pass + 1) & 1];
    pc.v_out = bb[(pass + 1) & 1];
    radix_pass(s, ipt, dg.bits, false, false, false, rc, pc);
  }
  return (passes & 1) != 0;
}

namespace {

// Device copies of the per-raw-frame tables (event offsets, filter frame of
// every raw frame) after frames were ingested.
void upload_frame_tables(Series &s) {
  cudaStream_t st = s.stream;
  if (!s.frame_off_dirty) return;
  s.d_frame_off.reserve(s.frame_off.size(), st);
  XG_CUDA(cudaMemcpyAsync(s.d_frame_off.p, s.frame_off.data(),
                          sizeof(int64_t) * s.frame_off.size(), cudaMemcpyHostToDevice, st));
  s.frame_map.resize(s.raw_frames);
  for (int32_t r = 0; r < s.raw_frames; r++) {  // stride*avg raw frames per filter frame
    const int32_t k = r / s.R_in;
    s.frame_map[r] = (k < s.F && ((r - k * s.R_in) % s.desc.stride_frames) == 0) ? k : -1;
  }
  s.d_frame_map.reserve(s.frame_map.size() ? s.frame_map.size() : 1, st);
  if (!s.frame_map.empty())
    XG_CUDA(cudaMemcpyAsync(s.d_frame_map.p, s.frame_map.data(),
                            sizeof(int32_t) * s.frame_map.size(), cudaMemcpyHostToDevice, st));
  s.frame_off_dirty = false;
}

// Filter and stable radix transpose of the raw frames [r0, r1): pixel-major
// events into ev_fr / ev_val and their row pointers (relative to ev_fr) into
// row_ptr [P+1].  Needs the frame tables on the device.
void transpose_range(Series &s, int32_t r0, int32_t r1, int32_t *ev_fr, float *ev_val,
                     int64_t *row_ptr) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P;
  const int64_t e0 = s.frame_off[r0], n = s.frame_off[r1] - e0;
  if (n <= 0) {
    XG_CUDA(cudaMemsetAsync(row_ptr, 0, sizeof(int64_t) * ((size_t)P + 1), st));
    return;
  }
  // the count of items sorted last, read by the row pointers, is per range
  XG_CUDA(cudaMemsetAsync(&s.stats.p->dropped, 0, sizeof(unsigned long long), st));
  const int nbits = 32 - __builtin_clz((unsigned)P);  // bits to hold P (the drop key)
  const Digits dg = digits_for(nbits);
  const int passes = dg.passes;
  const int ipt = s.radix_ipt == 8 || s.radix_ipt == 16 ? s.radix_ipt : items_per_lane(n);
  const int ntiles = (int)((n + RS_THREADS * ipt - 1) / (RS_THREADS * ipt));
  s.hist.reserve(radix_hist_words(n), s.stream);
  // sparse series below 65,536 filter frames carry one packed word per item
  // (frame, raw value) through the passes instead of a frame and a value
  const bool dense = s.desc.dense != 0;
  const bool packed = !dense && s.F <= 65536;
  // the last pass also writes the kept items' keys, for the row pointers
  s.keyA.reserve(n, st);
  if (passes > 1) {
    s.keyB.reserve(n, st);
    s.frA.reserve(n, st);
    if (!packed) s.vA.reserve(n, st);
  }
  if (passes > 2) {
    s.frB.reserve(n, st);
    if (!packed) s.vB.reserve(n, st);
  }
  const int chunk = 32 * ipt;
  const int64_t nch = (n + chunk - 1) / chunk;
  const int32_t nfr = r1 - r0;
  s.d_chunk_frame.reserve((size_t)nch, st);
  launch_overlapped(k_chunk_frames, (nfr + 255) / 256, 256, 0, st, nfr, s.d_frame_off.p + r0, e0,
                    nch, chunk, s.d_chunk_frame.p);
  RawCfg rc{s.raw_idx.p + e0, dense ? nullptr : s.raw_val.p + e0,
            dense ? s.raw_valf.p + e0 : nullptr, s.d_frame_off.p + r0, s.d_frame_map.p + r0,
            s.d_chunk_frame.p, nfr, e0, n, P, s.F, s.R_in, s.desc.stride_frames,
            s.has_flat ? s.d_flat.p : nullptr, s.stats.p};
  uint32_t *kbuf[2] = {s.keyA.p, s.keyB.p};
  int32_t *fbuf[2] = {s.frA.p, s.frB.p};
  float *vbuf[2] = {s.vA.p, s.vB.p};
  for (int pass = 0; pass < passes; pass++) {
    bool first = pass == 0, last = pass == passes - 1;
    PassCfg pc{};
    pc.n = n;
    pc.shift = dg.bits * pass;
    pc.ntiles = ntiles;
    pc.sentinel = (uint32_t)P;
    if (!first) {
      pc.key_in = kbuf[(pass - 1) & 1];
      pc.fr_in = fbuf[(pass - 1) & 1];
      pc.v_in = vbuf[(pass - 1) & 1];
    }
    if (last) {
      pc.key_out = kbuf[pass & 1];  // not the pass's input
      pc.fr_out = ev_fr;
      pc.v_out = ev_val;
    } else {
      pc.key_out = kbuf[pass & 1];
      pc.fr_out = fbuf[pass & 1];
      pc.v_out = vbuf[pass & 1];
    }
    radix_pass(s, ipt, dg.bits, packed, first, last, rc, pc);
  }
  const uint32_t *keys = (passes % 2 == 0) ? s.keyB.p : s.keyA.p;  // written by the last pass
  // smaller detectors' gaps take a warp at most 17 us, no longer than the searches
  const int gaps = P >= 1 << 17 ? (int)(((int64_t)P + 1 + 8 * RP_SPAN - 1) / (8 * RP_SPAN)) : 0;
  launch_overlapped(k_row_ptr, (unsigned)(gaps + (n + 1 + RP_U * 1024 - 1) / (RP_U * 1024)), 256, 0,
                    st, keys, n, s.stats.p, P, gaps, row_ptr);
}

void reserve_lists(Series &s) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P;
  s.row_ptr.reserve((size_t)P + 1, st);
  s.row_len.reserve(P, st);
  s.pclass.reserve(P, st);
  s.flist.reserve(P, st);
  s.wlist.reserve(P, st);
  s.llist.reserve(P, st);
  s.pixels_sum.reserve(P, st);
  s.stats.reserve(1, st);
}

// The lane-per-row form while rows are short (mean raw events per mapped
// pixel); to merge (avg != 1) or for long rows, which leave its lanes idle and
// its warps few, the warp-per-row form.  The whole filter stage in ms, short
// form / long form / before both (MS_MEAN_MAX lies between the two):
//   512^2 x 1,000 frames,     9 events a row  0.168 / 0.189 / 0.189
//   1024^2 x 10,000,         47               1.510 / 1.633 / 1.630
//   256^2 x 16,000,         151               0.395 / 0.399 / 0.443
//   512^2 x 4,000,          181               1.432 / 1.468 / 1.527
//   263^2 x 16,000,         676               1.626 / 1.451 / 1.629
//   509^2 x 1,500, average 2, 55 (to merge)       - / 0.825 / 1.114
void merge_classify(Series &s, int32_t avg) {
  const ClassLists cl{s.wlist.p, s.llist.p, s.flist.p};
  const double mean = (double)s.raw_events / (double)std::max<int64_t>(s.valid_pixels, 1);
  if (avg == 1 && mean < MS_MEAN_MAX)
    launch_overlapped(
        k_merge_short, (s.P + MS_WARPS * 32 - 1) / (MS_WARPS * 32), MS_WARPS * 32, 0, s.stream,
        s.P, s.F, s.class_cap, s.float_cap, s.desc.normalize_by_framesum, s.row_ptr.p, s.d_mask.p,
        s.ev_frame.p, s.ev_val.p, s.row_len.p, s.pclass.p, cl, s.pixels_sum.p, s.stats.p);
  else
    launch_overlapped(
        k_merge_rows, (s.P + 31) / 32, MC_WARPS * 32, 0, s.stream, s.P, s.F, avg, s.class_cap, s.float_cap, s.desc.normalize_by_framesum, s.row_ptr.p,
        s.d_mask.p, s.ev_frame.p, s.ev_val.p, s.row_len.p, s.pclass.p, cl, s.pixels_sum.p,
        s.stats.p);
}

}  // namespace

// ----------------------------------------------------- incremental transposes
//
// With a block size set (xpcs_series_set_block_frames), the frames are
// transposed as they are ingested, block by block (block_frames filter frames
// = block_frames * stride * avg raw frames, so that a filter frame's raw
// frames never straddle two blocks), into a store of block-local pixel-major
// rows that stays on the device.  Each block's rows are merged (events of one
// filter frame summed in stream order, then / avg; masked pixels emptied) as
// the whole-series merge does.  Finishing the series transposes the last,
// partial block and gathers every pixel's segments in block order -- blocks
// follow each other in time, so a row's segments concatenate in frame order --
// into the series' event lists, which are then classified as usual.  The
// result is the same event lists, bit for bit, as one transpose of every frame.

namespace {

// Block merge: one warp per 32 pixels; each lane merges its pixel's row of the
// block in place (when the block's rows hold a repeated frame or avg > 1) and
// records the row's start in the block and its merged length.
__global__ void __launch_bounds__(256)
k_merge_block(int32_t P, int32_t avg, const int64_t *__restrict__ row_ptr,
              const uint8_t *__restrict__ mask, int32_t *__restrict__ fr,
              float *__restrict__ val, int32_t *__restrict__ blk_off,
              int32_t *__restrict__ blk_len) {
  overlap_after();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p - (int)(threadIdx.x & 31) >= P) return;  // whole warp past the end
  const bool has = p < P;
  const int64_t b = has ? row_ptr[p] : 0;
  const int32_t n = has ? (int32_t)(row_ptr[p + 1] - b) : 0;
  int32_t out = 0;
  // one coalesced look at the warp's events: no two equal frames in a row, no
  // repeated frame (equal ones may also be the end of one row and the start of
  // the next, so the lanes then look for themselves)
  const int lane = threadIdx.x & 31;
  const int64_t lo = __shfl_sync(0xffffffffu, b, 0);
  const int64_t hi = row_ptr[min(p - lane + 32, P)];
  bool maybe = false;
  for (int64_t e = lo + 1 + lane; e < hi; e += 32) maybe |= fr[e] == fr[e - 1];
  maybe = __any_sync(0xffffffffu, maybe);
  if (has && mask[p]) {
    bool dup = false;
    for (int32_t i = 1; maybe && i < n && !dup; i++) dup = fr[b + i] == fr[b + i - 1];
    if (dup || avg != 1) {
      const float favg = (float)avg;
      int32_t i = 0;
      while (i < n) {
        const int32_t f = fr[b + i];
        float acc = 0.f;
        do {
          acc = __fadd_rn(acc, val[b + i]);
          i++;
        } while (i < n && fr[b + i] == f);
        fr[b + out] = f;
        val[b + out] = __fdiv_rn(acc, favg);
        out++;
      }
    } else {
      out = n;
    }
  }
  if (has) {
    blk_off[p] = (int32_t)b;
    blk_len[p] = out;
  }
}

// Merged row lengths of every block summed per pixel; pos: the events that a
// pixel has before each block (null: not wanted).
__global__ void k_block_totals(int32_t P, int32_t nblk, const int32_t *__restrict__ blk_len,
                               int32_t *__restrict__ pos, int32_t *__restrict__ tot) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  int32_t t = 0;
#pragma unroll 4
  for (int32_t k = 0; k < nblk; k++) {
    if (pos) pos[(size_t)k * P + p] = t;
    t += blk_len[(size_t)k * P + p];
  }
  tot[p] = t;
}

// Each pixel's block segments, in block order, copied to its row of the
// series' event lists.  One warp per 32 pixels and block: the segments of
// consecutive pixels follow each other in a block (with gaps where the merge
// shortened one), so the lanes take the range's events in order, 4 at a time,
// find each event's pixel among the 32 starts and place it in that pixel's
// row.  Warps of one pixel group follow each other, so that the short runs
// that they write meet in L2.  512 x 512 pixels in 10 blocks, 12.3 M events
// (bandwidth: 30 us): 228 us with one thread a pixel, 134 with one warp for all
// blocks of its pixels, 55 so.  Without pos (4 bytes a pixel and block that a
// memory limit refuses) each warp adds up the lengths before its block.
__global__ void __launch_bounds__(256)
k_gather_blocks(int32_t P, int32_t nblk, const int64_t *__restrict__ blk_base,
                const int32_t *__restrict__ blk_off, const int32_t *__restrict__ blk_len,
                const int32_t *__restrict__ pos, const int32_t *__restrict__ bfr,
                const float *__restrict__ bval, const int64_t *__restrict__ row_ptr,
                int32_t *__restrict__ fr, float *__restrict__ val) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t group = w / nblk;
  if (group * 32 >= P) return;
  const int k = (int)(w - group * nblk), p0 = (int)group * 32, p = p0 + lane;
  const int last = min(31, P - 1 - p0);
  const size_t q = (size_t)k * P + p;
  const int64_t d0 = row_ptr[p0];
  // this lane's segment: its place from the first row's start on, its length
  // and its start in the block
  int32_t before = 0;
  if (p < P && pos) before = pos[q];
  for (int j = 0; p < P && !pos && j < k; j++) before += blk_len[(size_t)j * P + p];
  const int64_t d = p < P ? row_ptr[p] - d0 + before : 0;
  const int32_t n = p < P ? blk_len[q] : 0, off = p < P ? blk_off[q] : INT32_MAX;
  const int64_t base = blk_base[k];
  const int32_t lo = __shfl_sync(FULL, off, 0);
  const int32_t hi = __shfl_sync(FULL, off + n, last);
  for (int32_t e0 = lo; e0 < hi; e0 += 128) {
    int32_t f[4];
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int32_t e = e0 + u * 32 + lane;
      f[u] = e < hi ? bfr[base + e] : 0;
      v[u] = e < hi ? bval[base + e] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int32_t e = e0 + u * 32 + lane;
      int own = 0;  // the last lane whose segment starts at or before e
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(FULL, off, (own + o) & 31) <= e) own += o;
      const int32_t i = e - __shfl_sync(FULL, off, own);
      const int64_t dst = d0 + __shfl_sync(FULL, d, own) + i;
      const int32_t len = __shfl_sync(FULL, n, own);  // by all lanes
      if (e < hi && i < len) {
        fr[dst] = f[u];
        val[dst] = v[u];
      }
    }
  }
}

// Every pixel's block segments gathered into its row of the series' event
// lists (d_blk_base on the device already), then classified (the rows are
// merged already: avg 1 leaves nothing to merge).
void gather_blocks(Series &s) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P, nblk = (int32_t)s.blk_base.size();
  s.blk_tot.reserve(P, st);
  if (nblk > 0) {
    const bool pos = s.blk_pos.try_reserve((size_t)nblk * P, st);
    k_block_totals<<<(P + 255) / 256, 256, 0, st>>>(P, nblk, s.blk_len.p,
                                                    pos ? s.blk_pos.p : nullptr, s.blk_tot.p);
    XG_CHECK_LAUNCH();
    exclusive_scan_i32_i64(s.blk_tot.p, s.row_ptr.p, P, s.scan_tmp.p, st);
    const int64_t warps = (int64_t)((P + 31) / 32) * nblk;  // below 2^31 blocks of 8
    k_gather_blocks<<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(
        P, nblk, s.d_blk_base.p, s.blk_off.p, s.blk_len.p, pos ? s.blk_pos.p : nullptr, s.blk_fr.p,
        s.blk_val.p, s.row_ptr.p, s.ev_frame.p, s.ev_val.p);
    XG_CHECK_LAUNCH();
    if (dev_limited()) s.blk_pos.release(st);  // the call's alone
  } else {
    XG_CUDA(cudaMemsetAsync(s.row_ptr.p, 0, sizeof(int64_t) * ((size_t)P + 1), st));
  }
  merge_classify(s, 1);
}

// Transposes the next block, ending at raw frame r1, into the block store.
void transpose_block(Series &s, int32_t r1) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P, r0 = s.blk_raw_done;
  const int64_t n = s.frame_off[r1] - s.frame_off[r0];
  const int64_t base = s.blk_events;
  s.blk_fr.grow((size_t)(base + std::max<int64_t>(n, 1)), (size_t)base, st);
  s.blk_val.grow((size_t)(base + std::max<int64_t>(n, 1)), (size_t)base, st);
  const size_t k = s.blk_base.size();
  s.blk_off.grow((k + 1) * (size_t)P, k * (size_t)P, st);
  s.blk_len.grow((k + 1) * (size_t)P, k * (size_t)P, st);
  s.blk_rp.reserve((size_t)P + 1, st);
  transpose_range(s, r0, r1, s.blk_fr.p + base, s.blk_val.p + base, s.blk_rp.p);
  launch_overlapped(k_merge_block, (P + 255) / 256, 256, 0, st, P, s.desc.avg_frames, s.blk_rp.p,
                    s.d_mask.p, s.blk_fr.p + base, s.blk_val.p + base,
                    s.blk_off.p + k * (size_t)P, s.blk_len.p + k * (size_t)P);
  s.blk_base.push_back(base);
  s.blk_events = base + n;
  s.blk_raw_done = r1;
}

}  // namespace

void transpose_ready_blocks(Series &s) {
  // pixel-major dense series write their blocks as frames arrive
  if (s.block_frames <= 0 || s.dense_px) return;
  const int32_t step = s.block_frames * s.R_in;
  // raw frames past the series' last filter frame are never used
  const int32_t limit = std::min<int64_t>(s.raw_frames, (int64_t)s.F * s.R_in);
  if (s.blk_raw_done + step > limit) return;
  s.stats.reserve(1, s.stream);
  if (s.blk_base.empty())  // the first block of the series: a clean error word
    XG_CUDA(cudaMemsetAsync(s.stats.p, 0, sizeof(DevStats), s.stream));
  upload_frame_tables(s);
  while (s.blk_raw_done + step <= limit) transpose_block(s, s.blk_raw_done + step);
}

void reset_blocks(Series &s) {
  s.blk_base.clear();
  s.blk_r0.clear();
  s.blk_events = 0;
  s.blk_raw_done = 0;
  s.dn_pend_n = 0;
}

// The thread kernel's row capacity for a series nobody tuned: the smallest
// capacity of at least 1.5 mean rows, which the autotuner also picks for mean
// rows of 25, 52 and 100 events (1 Mi pixels, 5,000-20,000 frames), and the
// extra scratch words it picks from 16,384 frames on.
// Series of few pixels (alone: not beside a batch's other members) give every
// row to a warp: one thread a row leaves most of the chip without work and
// takes as long as its longest row.  At 1,000 frames the integer rows take, with
// a thread / a warp a row, at 4,096 pixels and rows of 3, 10, 30 events 35 / 26,
// 54 / 29 and 84 / 30 us, at 16,384 pixels 36 / 57, 54 / 62 and 117 / 65 us, at
// 36,864 pixels 39 / 102, 58 / 116 and 129 / 125 us; rows of 80 events (4,000
// frames) 190 / 94 us at 16,384 and 197 / 186 us at 36,864 pixels.  The line
// lies where the two meet.  It does not hold for a row capacity that the caller
// chose, and the autotuner times both forms of such a series.
void default_knobs(Series &s, bool alone) {
  if (s.valid_pixels < 0) {
    s.valid_pixels = 0;
    for (uint8_t v : s.qmap.valid) s.valid_pixels += v;
    if (s.qmap.valid.empty()) s.valid_pixels = s.P;  // caller-held rows have no map
  }
  const double mean =
      (double)s.raw_events / ((double)std::max<int64_t>(s.valid_pixels, 1) * s.R_in);
  // raw events of a row that the filter uses: the stride's skipped sub-frames
  // are among a sparse series' events
  s.float_cap = mt_float_cap(s, mean * s.R_in / (s.desc.dense ? 1 : s.desc.stride_frames));
  if (!s.knobs_set) {
    int32_t cap = MT_THREAD_CAPS[MT_THREAD_NCAPS - 1];
    for (int c : MT_THREAD_CAPS)
      if (c >= 1.5 * mean) {
        cap = c;
        break;
      }
    s.thread_cap = cap;
    s.scr_extra = s.F >= 16384 ? 8 : 0;
  }
  const bool few = s.valid_pixels <= std::min(5000.0 + 800.0 * mean, 32000.0);
  s.class_cap = few && alone && !s.by_thread ? 0 : s.thread_cap;
}

void run_filter_transpose(Series &s, bool alone) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P;
  dense_px_flush(s);  // frames still pending become the last block
  default_knobs(s, alone);
  reserve_lists(s);
  const size_t nalloc = s.raw_events > 0 ? (size_t)s.raw_events : 1;
  s.ev_frame.reserve(nalloc, st);
  s.ev_val.reserve(nalloc, st);
  s.scan_tmp.reserve(scan_workspace_bytes(P), st);
  if (s.dense_px) {
    XG_CUDA(cudaMemsetAsync(s.stats.p, 0, sizeof(DevStats), st));
    dense_px_gather(s);  // gathers and classifies
    return;
  }
  if (s.block_frames <= 0) {
    XG_CUDA(cudaMemsetAsync(s.stats.p, 0, sizeof(DevStats), st));
    upload_frame_tables(s);
    transpose_range(s, 0, s.raw_frames, s.ev_frame.p, s.ev_val.p, s.row_ptr.p);
    merge_classify(s, s.desc.avg_frames);
    return;
  }
  // the error word keeps what earlier block transposes found; the counters restart
  if (s.blk_base.empty())
    XG_CUDA(cudaMemsetAsync(s.stats.p, 0, sizeof(DevStats), st));
  else
    XG_CUDA(cudaMemsetAsync(&s.stats.p->nfloat, 0,
                            sizeof(DevStats) - offsetof(DevStats, nfloat), st));
  upload_frame_tables(s);
  if (s.blk_raw_done < s.raw_frames) transpose_block(s, s.raw_frames);  // the last block
  const int32_t nblk = (int32_t)s.blk_base.size();
  s.d_blk_base.reserve((size_t)std::max(nblk, 1), st);
  if (nblk > 0)
    XG_CUDA(cudaMemcpyAsync(s.d_blk_base.p, s.blk_base.data(), sizeof(int64_t) * nblk,
                            cudaMemcpyHostToDevice, st));
  gather_blocks(s);
}

}  // namespace xg

namespace xg {
namespace {

// Caller-held rows (xpcs_multitau2): rows stay as given; a pixel takes the
// integer path only if its frames are strictly increasing within [0, F), its
// values are integers and sum |v| < 4096.
__global__ void k_classify_rows(int32_t P, int32_t F, int32_t tcap, const int64_t *__restrict__ row_ptr,
                                const int32_t *__restrict__ fr, const float *__restrict__ val,
                                int32_t *__restrict__ row_len, uint8_t *__restrict__ pclass,
                                ClassLists cl, DevStats *__restrict__ stats) {
  const int32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p - (int32_t)(threadIdx.x & 31) >= P) return;  // whole warp past the end
  const bool has = p < P;
  const int64_t b = has ? row_ptr[p] : 0;
  const int32_t n = has ? (int32_t)(row_ptr[p + 1] - b) : 0;
  if (has) row_len[p] = n;
  bool ok = n <= MT_LONG_CAP;
  long long total = 0;
  int32_t prev = -1;
  for (int32_t i = 0; i < n && ok; i++) {
    int32_t f = fr[b + i];
    float x = val[b + i];
    ok = f > prev && f < F && x == truncf(x) && fabsf(x) < 16777216.f;
    if (ok) total += llabs((long long)x);
    prev = f;
  }
  const uint8_t c = n == 0 ? (uint8_t)PCLASS_EMPTY : pixel_class(n, ok, total, F, tcap);
  record_class_warp(has, p, c, n, pclass, cl, stats);
}

}  // namespace

void multitau_rows_upload(Series &s, const int64_t *row_ptr, const int32_t *frame,
                          const float *value, int64_t events) {
  cudaStream_t st = s.stream;
  const int32_t P = s.P;
  size_t ne = events > 0 ? (size_t)events : 1;
  s.row_ptr.reserve((size_t)P + 1, st);
  s.row_len.reserve(P, st);
  s.pclass.reserve(P, st);
  s.flist.reserve(P, st);
  s.wlist.reserve(P, st);
  s.llist.reserve(P, st);
  s.stats.reserve(1, st);
  s.ev_frame.reserve(ne, st);
  s.ev_val.reserve(ne, st);
  s.raw_events = events;
  XG_CUDA(cudaMemsetAsync(s.stats.p, 0, sizeof(DevStats), st));
  XG_CUDA(cudaMemcpyAsync(s.row_ptr.p, row_ptr, sizeof(int64_t) * ((size_t)P + 1),
                          cudaMemcpyHostToDevice, st));
  if (events > 0) {
    XG_CUDA(cudaMemcpyAsync(s.ev_frame.p, frame, sizeof(int32_t) * events, cudaMemcpyHostToDevice, st));
    XG_CUDA(cudaMemcpyAsync(s.ev_val.p, value, sizeof(float) * events, cudaMemcpyHostToDevice, st));
  }
  default_knobs(s, true);
  const int bs = 256;
  k_classify_rows<<<(P + bs - 1) / bs, bs, 0, st>>>(P, s.F, s.class_cap, s.row_ptr.p, s.ev_frame.p,
                                                     s.ev_val.p, s.row_len.p, s.pclass.p,
                                                     ClassLists{s.wlist.p, s.llist.p, s.flist.p},
                                                     s.stats.p);
  XG_CHECK_LAUNCH();
}

}  // namespace xg
