// Matrix tile emission on the device: the four UInt32 columns of a matrix
// RecordBatch (source_idx, target_idx, duration_ms, distance_m) from a
// row-major block of durations, as build_matrix_batch and
// build_matrix_tile_batch build them on the host
// (route/src/server/flight.rs:432-500, :509-589):
//   * cells in row-major order; a cell is pruned when the source's sorted
//     radius list (indexed by the source's original index) lacks the
//     destination's original index (:452-456, :528-532);
//   * a pruned cell reads u32::MAX, any other the matrix value, u32::MAX
//     above the time bound (:459, :534-539);
//   * sparse output drops cells whose duration is u32::MAX (:465, :542);
//   * duration_ms = d.saturating_mul(1000); distance_m = the lat matrix's
//     cell or u32::MAX; both u32::MAX on a sentinel cell (:470-483, :548-566).
// The columns come out as plain u32 arrays: Arrow's layout of a UInt32 array
// without nulls, so the caller wraps them without a copy.
//
// Dense: four consecutive cells of the block per thread whatever the row
// width, 16-byte reads and column writes (a thread per cell where an array is
// not 16-byte aligned). Sparse: an order-preserving compaction - a count and
// the kept-cell ballots per block (a row segment of up to 16384 cells for
// rows of 2048 cells or more, its radius list read once and set into a bitmap
// in shared memory; else 2048 consecutive cells), a scan of the counts, then
// an ordered write of the kept cells.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "engine.cuh"
#include "scan.cuh"

using namespace bf;

namespace {

constexpr uint32_t MAXV = 0xFFFFFFFFu;
constexpr uint32_t TPB = 256, ITEMS = 8, CELLS = TPB * ITEMS;
constexpr uint64_t FEW_CELLS = 1u << 20;  // 152 SMs x 2048 threads, 3.4 cells each
constexpr uint32_t ERR_NO_LIST = 1u, ERR_BAD_LIST = 2u;

struct TileIn {
  const uint32_t* m;
  const uint32_t* lat;  // may be null
  uint32_t n_src, n_dst;
  const uint32_t* src_orig;
  const uint32_t* dst_orig;
  uint32_t threshold;
  const uint64_t* mask_off;  // null: no radius mask
  const uint32_t* mask;
  uint32_t n_mask_src;
  uint64_t n_mask;
  uint32_t sparse;
};

struct TileOut {
  uint32_t *s, *t, *du, *di;
};

// (row, column) of a flat cell index; 32-bit division when the block allows.
__device__ __forceinline__ void split(uint64_t i, uint32_t n_dst, bool narrow, uint32_t* si,
                                      uint32_t* di) {
  if (narrow) {
    const uint32_t q = (uint32_t)i / n_dst;
    *si = q;
    *di = (uint32_t)i - q * n_dst;
  } else {
    *si = (uint32_t)(i / n_dst);
    *di = (uint32_t)(i % n_dst);
  }
}

// binary_search's answer (present or not) on a sorted list: halving steps on
// 32-bit offsets, one comparison at the end.
__device__ __forceinline__ bool in_list(const uint32_t* __restrict__ v, uint32_t len, uint32_t x) {
  if (len == 0) return false;
  while (len > 1) {
    const uint32_t half = len >> 1;
    if (v[half] <= x) v += half;
    len -= half;
  }
  return *v == x;
}

// The cell's duration d (already loaded) after pruning and the time bound
// (both give u32::MAX, so the bound is tested first and only cells within
// it search the radius list); os, od: the original indices.
__device__ __forceinline__ uint32_t decide(const TileIn& a, uint32_t d, uint32_t os, uint32_t od,
                                           uint32_t* err) {
  if (a.mask_off && os >= a.n_mask_src) {  // the reference indexes every row's list
    atomicOr(err, ERR_NO_LIST);
    return MAXV;
  }
  if (d > a.threshold) return MAXV;
  if (a.mask_off) {
    const uint64_t lo = a.mask_off[os], hi = a.mask_off[os + 1];
    if (hi < lo || hi > a.n_mask || hi - lo > 0xFFFFFFFFull) {
      atomicOr(err, ERR_BAD_LIST);
      return MAXV;
    }
    if (!in_list(a.mask + lo, (uint32_t)(hi - lo), od)) return MAXV;
  }
  return d;
}

__device__ __forceinline__ uint32_t cell_value(const TileIn& a, uint32_t si, uint32_t di,
                                               uint64_t cell, uint32_t* os, uint32_t* od,
                                               uint32_t* err) {
  *os = a.src_orig[si];
  *od = a.dst_orig[di];
  return decide(a, a.m[cell], *os, *od, err);
}

__device__ __forceinline__ void put(const TileIn& a, const TileOut& o, uint64_t k, uint64_t cell,
                                    uint32_t os, uint32_t od, uint32_t d) {
  o.s[k] = os;
  o.t[k] = od;
  if (d == MAXV) {
    o.du[k] = MAXV;
    o.di[k] = MAXV;
  } else {
    const uint64_t ms = (uint64_t)d * 1000u;
    o.du[k] = ms > MAXV ? MAXV : (uint32_t)ms;
    o.di[k] = a.lat ? a.lat[cell] : MAXV;
  }
}


__global__ void __launch_bounds__(TPB) k_tile_dense(TileIn a, TileOut o, uint32_t* err) {
  for (uint32_t si = blockIdx.y; si < a.n_src; si += gridDim.y)
    for (uint32_t di = blockIdx.x * TPB + threadIdx.x; di < a.n_dst; di += gridDim.x * TPB) {
      const uint64_t cell = (uint64_t)si * a.n_dst + di;
      uint32_t os, od;
      const uint32_t d = cell_value(a, si, di, cell, &os, &od, err);
      put(a, o, cell, cell, os, od, d);
    }
}

// Dense with four consecutive cells of the block per thread (arrays 16-byte
// aligned, any row width: cell 4 q lies on a 16-byte boundary whichever row it
// falls in): one 16-byte load of durations (and lengths), one 16-byte store
// per column. Bound by HBM: 8 bytes in and 16 out per cell.
// 5003 x 4001 cells with lengths: 69 us (7.0 TB/s) against 114 us of a thread
// per cell, which rows not a multiple of four cells took.
__global__ void __launch_bounds__(TPB)
    k_tile_dense4(TileIn a, TileOut o, uint64_t n, bool narrow, bool skip_sentinels, uint32_t* err) {
  const uint64_t q4 = (n + 3) >> 2;
  for (uint64_t q = (uint64_t)blockIdx.x * TPB + threadIdx.x; q < q4;
       q += (uint64_t)gridDim.x * TPB) {
    const uint64_t cell = 4 * q;
    const bool whole = cell + 4 <= n;
    uint32_t dv[4], lv[4];
    if (whole) {
      const uint4 m4 = __ldcs(reinterpret_cast<const uint4*>(a.m + cell));
      const uint4 l4 = a.lat ? __ldcs(reinterpret_cast<const uint4*>(a.lat + cell))
                             : make_uint4(MAXV, MAXV, MAXV, MAXV);
      dv[0] = m4.x, dv[1] = m4.y, dv[2] = m4.z, dv[3] = m4.w;
      lv[0] = l4.x, lv[1] = l4.y, lv[2] = l4.z, lv[3] = l4.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        dv[k] = cell + k < n ? a.m[cell + k] : MAXV;
        lv[k] = a.lat && cell + k < n ? a.lat[cell + k] : MAXV;
      }
    }
    uint32_t si, di;
    split(cell, a.n_dst, narrow, &si, &di);
    uint32_t os = a.src_orig[si];
    uint32_t s4[4], t4[4], du[4], ln[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (cell + k >= n) break;
      if (di == a.n_dst) {  // the quad goes on in the next row
        di = 0;
        os = a.src_orig[++si];
      }
      s4[k] = os;
      t4[k] = a.dst_orig[di++];
      // the sentinel's list is not looked at where it never was
      const bool skip = skip_sentinels && dv[k] == MAXV && !(a.mask_off && os >= a.n_mask_src);
      const uint32_t d = skip ? MAXV : decide(a, dv[k], os, t4[k], err);
      const uint64_t ms = (uint64_t)d * 1000u;
      du[k] = d == MAXV || ms > MAXV ? MAXV : (uint32_t)ms;
      ln[k] = d == MAXV ? MAXV : lv[k];
    }
    if (whole) {
      __stcs(reinterpret_cast<uint4*>(o.s + cell), make_uint4(s4[0], s4[1], s4[2], s4[3]));
      __stcs(reinterpret_cast<uint4*>(o.t + cell), make_uint4(t4[0], t4[1], t4[2], t4[3]));
      __stcs(reinterpret_cast<uint4*>(o.du + cell), make_uint4(du[0], du[1], du[2], du[3]));
      __stcs(reinterpret_cast<uint4*>(o.di + cell), make_uint4(ln[0], ln[1], ln[2], ln[3]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (cell + k >= n) break;
        o.s[cell + k] = s4[k];
        o.t[cell + k] = t4[k];
        o.du[cell + k] = du[k];
        o.di[cell + k] = ln[k];
      }
    }
  }
}

// Sparse pass 1: per block the kept cells, per (step, warp) the ballot of
// kept cells (bit lane of word (cell / 32)); rows and columns advance by
// TPB cells a step instead of a division per cell.
__global__ void __launch_bounds__(TPB)
    k_tile_count(TileIn a, uint64_t n, bool narrow, unsigned long long* __restrict__ cnt,
                 uint32_t* __restrict__ keep_bits, uint32_t* err) {
  __shared__ uint32_t red[TPB / 32];
  const uint64_t base = (uint64_t)blockIdx.x * CELLS;
  uint32_t c = 0, si = 0, di = 0;
  split(base + threadIdx.x, a.n_dst, narrow, &si, &di);
  uint32_t dur[ITEMS];  // the block's durations, all loads in flight before any decision
#pragma unroll
  for (uint32_t j = 0; j < ITEMS; ++j) {
    const uint64_t i = base + (uint64_t)j * TPB + threadIdx.x;
    dur[j] = i < n ? a.m[i] : MAXV;
  }
#pragma unroll
  for (uint32_t j = 0; j < ITEMS; ++j) {
    const uint64_t i = base + (uint64_t)j * TPB + threadIdx.x;
    if (base + (uint64_t)j * TPB >= n) break;  // uniform across the block
    if (j) {
      if (a.n_dst >= TPB) {
        di += TPB;
        if (di >= a.n_dst) {
          di -= a.n_dst;
          ++si;
        }
      } else {
        split(i, a.n_dst, narrow, &si, &di);
      }
    }
    bool keep = false;
    if (i < n) keep = decide(a, dur[j], a.src_orig[si], a.dst_orig[di], err) != MAXV;
    const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep);
    if ((threadIdx.x & 31) == 0) keep_bits[(base + (uint64_t)j * TPB) / 32 + (threadIdx.x >> 5)] = bal;
    c += keep;
  }
  for (int s = 16; s > 0; s >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (uint32_t w = 0; w < TPB / 32; ++w) t += red[w];
    cnt[blockIdx.x] = t;
  }
}

// Wide rows (n_dst >= ROW_MIN): a block per row segment of up to SEG cells,
// so a row's radius list is read once per segment: staged in shared memory
// when it holds at most LIST_STAGE entries, else searched in place. Ballot
// words are per row (wpr = ceil(n_dst / 32) words each), counts per
// segment, in cell order.
constexpr uint32_t ROW_MIN = 2048, SEG = 16384, SEG_WORDS = SEG / 32, LIST_STAGE = 4096;
enum : uint32_t { RL_NONE = 0, RL_SMEM = 1, RL_GLOBAL = 2, RL_BAD = 3, RL_MISSING = 4 };
// A staged list is set into a bitmap of original indices below BITMAP_BITS,
// so a destination id below it is one shared-memory word test; where ids at or
// above it exist, the list itself is staged too and searched for those.
constexpr uint32_t BITMAP_BITS = 1u << 17, BITMAP_WORDS = BITMAP_BITS / 32;
constexpr uint32_t STAGE_STEP = 8;  // list entries a thread has in flight

struct RowList {
  uint32_t v[LIST_STAGE];
  uint32_t bmp[BITMAP_WORDS];
};

// Stages len list entries (block-uniform call): the bitmap's first nbw words
// (ids below 32 nbw: the destination ids' range, capped), and the entries
// themselves unless the bitmap answers for every id.
__device__ __forceinline__ void stage_row_list(RowList& rl, const uint32_t* __restrict__ src,
                                               uint32_t len, uint32_t nbw, bool bitmap_only) {
  uint32_t x[STAGE_STEP];
#pragma unroll
  for (uint32_t u = 0; u < STAGE_STEP; ++u) {
    const uint32_t k = u * TPB + threadIdx.x;
    x[u] = k < len ? src[k] : MAXV;
  }
  for (uint32_t k = threadIdx.x; k < nbw; k += TPB) rl.bmp[k] = 0;
  __syncthreads();
  for (uint32_t k0 = 0; k0 < len; k0 += STAGE_STEP * TPB) {
#pragma unroll
    for (uint32_t u = 0; u < STAGE_STEP; ++u) {
      const uint32_t k = k0 + u * TPB + threadIdx.x;
      if (k < len) {
        if (!bitmap_only) rl.v[k] = x[u];
        if (x[u] < nbw * 32) atomicOr(&rl.bmp[x[u] >> 5], 1u << (x[u] & 31));
      }
    }
    if (k0 + STAGE_STEP * TPB < len) {
#pragma unroll
      for (uint32_t u = 0; u < STAGE_STEP; ++u) {
        const uint32_t k = k0 + (STAGE_STEP + u) * TPB + threadIdx.x;
        x[u] = k < len ? src[k] : MAXV;
      }
    }
  }
  __syncthreads();
}

// A wide row's position on the 16-byte grid of the matrix: cells are counted
// from the last 16-byte boundary at or before the row, so position p of the
// row is column p - row_lead and quads of positions load as one word whatever
// the row width and the matrix's own alignment.
__device__ __forceinline__ uint32_t row_lead(const TileIn& a, uint32_t si) {
  return (uint32_t)(((uintptr_t)a.m >> 2) + (uint64_t)si * a.n_dst) & 3u;
}

// Per wide row, once per call: how its radius list is read ({mode, len, list
// offset low and high words}, decide()'s rules), and into bound[0] the
// largest destination id (the bitmap's range).
__global__ void __launch_bounds__(TPB) k_tile_rowinfo(TileIn a, uint4* __restrict__ info,
                                                      uint32_t* __restrict__ bound) {
  const uint32_t stride = gridDim.x * TPB;
  for (uint32_t si = blockIdx.x * TPB + threadIdx.x; si < a.n_src; si += stride) {
    uint32_t mode = RL_NONE, len = 0;
    uint64_t lo = 0;
    if (a.mask_off) {
      const uint32_t os = a.src_orig[si];
      if (os >= a.n_mask_src) {
        mode = RL_MISSING;
      } else {
        lo = a.mask_off[os];
        const uint64_t hi = a.mask_off[os + 1];
        if (hi < lo || hi > a.n_mask || hi - lo > 0xFFFFFFFFull) {
          mode = RL_BAD;
          lo = 0;
        } else {
          len = (uint32_t)(hi - lo);
          mode = len <= LIST_STAGE ? RL_SMEM : RL_GLOBAL;
        }
      }
    }
    info[si] = make_uint4(mode, len, (uint32_t)lo, (uint32_t)(lo >> 32));
  }
  uint32_t mx = 0;
  for (uint32_t c = blockIdx.x * TPB + threadIdx.x; c < a.n_dst; c += stride)
    mx = max(mx, a.dst_orig[c]);
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(bound, mx);
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* red) {
  for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  for (uint32_t w = 0; w < TPB / 32; ++w) t += red[w];
  return t;
}

// Sparse pass 1 for wide rows: the segment's kept cells and ballots, with
// decide()'s rules: a row without a list keeps nothing (ERR_NO_LIST), a bad
// list keeps nothing and is an error once a cell is within the bound. A thread
// takes VEC quads of positions a step, the next step's loads in flight while
// this one is decided. The floor is HBM (the durations and the radius lists,
// once); what bounds it is issue, so the work of a step is kept small: one
// 16-bit mask of a thread's cells within the bound, the list asked for its
// set bits alone (most cells of a table are beyond the bound), and one
// exchange of three shuffles that turns the masks of 8 lanes into the ballot
// words of all VEC quads.
// 10,000 x 10,000 cells, lists of 2,000, 2.1 % within the bound: 117 us
// (4.1 TB/s) against 167 us with three shuffles and four bitmap words per
// quad. Five blocks an SM: 188 us for the whole call, against 198 with four
// and 240 with six, whose registers spill.
constexpr uint32_t VEC = 4, CELLS4 = TPB * 4 * VEC;

__device__ __forceinline__ void load_step(const uint32_t* __restrict__ base, uint32_t b0,
                                          uint32_t first, uint32_t end, uint4 (&q)[VEC]) {
  const uint32_t p0 = b0 + threadIdx.x * 4;
  if (b0 >= first && end >= CELLS4 && b0 <= end - CELLS4) {  // the whole step lies in the row
#pragma unroll
    for (uint32_t u = 0; u < VEC; ++u)
      q[u] = *reinterpret_cast<const uint4*>(base + p0 + u * TPB * 4);
    return;
  }
  if (b0 >= end) return;  // the step after the last: never looked at
#pragma unroll
  for (uint32_t u = 0; u < VEC; ++u) {
    const uint32_t p = p0 + u * TPB * 4;
    if (p >= first && p + 4 <= end) {
      q[u] = *reinterpret_cast<const uint4*>(base + p);
    } else {
      uint32_t v[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) v[k] = p + k >= first && p + k < end ? base[p + k] : MAXV;
      q[u] = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
}

// The ballot word this lane stores, of the 16-bit masks (nibble u: quad u) of
// its 8-lane group: lane l of the group returns the 32 cells of quad
// word_quad(l), the same word in lanes l and l ^ 4.
__device__ __forceinline__ uint32_t word_quad(uint32_t lane) {
  return (lane & 1) * 2 + ((lane >> 1) & 1);
}
__device__ __forceinline__ uint32_t ballot_word(uint32_t m16, uint32_t lane) {
  static_assert(VEC == 4, "three halvings of four quads");
  // lanes l, l ^ 1: the even one keeps quads 0 and 1, the odd one 2 and 3
  const bool o1 = lane & 1, o2 = lane & 2, o4 = lane & 4;
  uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, m16, 1);
  uint32_t mine = o1 ? m16 >> 8 : m16 & 0xFFu;
  other = o1 ? other >> 8 : other & 0xFFu;
  // {even lane's nibble, odd lane's nibble} of the first quad, then the second
  const uint32_t ev = o1 ? other : mine, od = o1 ? mine : other;
  const uint32_t two = (ev & 0xFu) | ((od & 0xFu) << 4) | ((ev & 0xF0u) << 4) | ((od & 0xF0u) << 8);
  other = __shfl_xor_sync(0xFFFFFFFFu, two, 2);
  mine = o2 ? two >> 8 : two & 0xFFu;
  other = o2 ? other >> 8 : other & 0xFFu;
  const uint32_t four = o2 ? other | (mine << 8) : mine | (other << 8);
  other = __shfl_xor_sync(0xFFFFFFFFu, four, 4);
  return o4 ? other | (four << 16) : four | (other << 16);
}

__global__ void __launch_bounds__(TPB, 5)
    k_tile_count_rows(TileIn a, uint32_t segs, uint32_t wpr, const uint4* __restrict__ info,
                      const uint32_t* __restrict__ bound, unsigned long long* __restrict__ cnt,
                      uint32_t* __restrict__ keep_bits, uint32_t* err) {
  __shared__ RowList rl;
  __shared__ uint32_t red[TPB / 32];
  const uint32_t si = blockIdx.x / segs, sg = blockIdx.x % segs;
  const uint32_t lead = row_lead(a, si), row_end = lead + a.n_dst;
  const uint32_t p_begin = sg * SEG, p_end = min(p_begin + SEG, row_end);  // may be empty
  const uint32_t lane = threadIdx.x & 31;
  // the row's 16-byte boundary; positions before `lead` are not read
  const uint32_t* base = a.m + ((int64_t)si * a.n_dst - lead);
  // the first step's durations load while the row's list is looked up
  uint4 dur[VEC];
  load_step(base, p_begin, lead, p_end, dur);
  const uint4 ri = info[si];  // {mode, len, list offset (lo, hi words)}
  const uint32_t nbw = min(BITMAP_WORDS, (*bound >> 5) + 1);
  const bool bitmap_only = (*bound >> 5) < BITMAP_WORDS;  // every destination id has a bit
  const uint32_t mode = ri.x, len = ri.y;
  const uint64_t lo = ri.z | ((uint64_t)ri.w << 32);
  if (mode == RL_MISSING && threadIdx.x == 0) atomicOr(err, ERR_NO_LIST);
  // uniform: every thread read the same row record
  if (mode == RL_SMEM) stage_row_list(rl, a.mask + lo, len, nbw, bitmap_only);
  const uint32_t* lg = a.mask + lo;
  uint32_t* bits = keep_bits + (uint64_t)si * wpr;
  // a cell is within the bound iff d <= thr1 (the u32::MAX sentinel never
  // is); positions outside the row read as the sentinel, so no column test
  const uint32_t thr1 = min(a.threshold, MAXV - 1);
  const uint32_t lim = nbw * 32;
  uint32_t c = 0;
  bool bad_hit = false;
  for (uint32_t b0 = p_begin; b0 < p_end; b0 += CELLS4) {
    uint4 nxt[VEC];
    load_step(base, b0 + CELLS4, lead, p_end, nxt);
    uint32_t in16 = 0;
#pragma unroll
    for (uint32_t u = 0; u < VEC; ++u) {
      const uint4 d = dur[u];
      in16 |= (d.x <= thr1 ? 1u << (4 * u) : 0u) | (d.y <= thr1 ? 2u << (4 * u) : 0u) |
              (d.z <= thr1 ? 4u << (4 * u) : 0u) | (d.w <= thr1 ? 8u << (4 * u) : 0u);
      dur[u] = nxt[u];
    }
    uint32_t keep = in16;
    if (mode != RL_NONE && in16) {
      if (mode == RL_SMEM || mode == RL_GLOBAL) {
        // the thread's position of bit 0 of quad 0, as a column
        const uint32_t* od = a.dst_orig + (int64_t)b0 + threadIdx.x * 4 - lead;
        for (uint32_t left = in16; left; left &= left - 1) {
          const uint32_t k = __ffs(left) - 1;
          const uint32_t x = od[(k >> 2) * (TPB * 4) + (k & 3)];
          bool in;
          if (mode == RL_GLOBAL) in = in_list(lg, len, x);
          else if (x < lim) in = (rl.bmp[x >> 5] >> (x & 31)) & 1u;
          else in = in_list(rl.v, len, x);
          if (!in) keep ^= 1u << k;
        }
      } else {
        bad_hit |= mode == RL_BAD;
        keep = 0;
      }
    }
    c += __popc(keep);
    const uint32_t word = ballot_word(keep, lane);
    const uint32_t wcell = b0 + (word_quad(lane) * TPB + (threadIdx.x & ~31u)) * 4 + (lane >> 3) * 32;
    if (!(lane & 4) && wcell < p_end) bits[wcell / 32] = word;
  }
  if (bad_hit) atomicOr(err, ERR_BAD_LIST);
  const uint32_t t = block_sum(c, red);
  if (threadIdx.x == 0) cnt[blockIdx.x] = t;
}

// Dense for wide rows with radius lists (ROW_MIN cells or more, arrays 16-byte
// aligned): a block per row segment, its list staged as in the count pass, so
// a cell asks one bitmap word instead of searching the list in memory.
// 5000 x 4000 cells with lists of 800, 2.1 % of the cells within the bound:
// 118 us a call against 181 with a search in memory; lists of 2,000 and every
// cell within the bound: 133 us against 268.
__global__ void __launch_bounds__(TPB)
    k_tile_dense_rows(TileIn a, TileOut o, uint32_t segs, const uint4* __restrict__ info,
                      const uint32_t* __restrict__ bound, bool skip_sentinels, uint32_t* err) {
  __shared__ RowList rl;
  const uint32_t si = blockIdx.x / segs, sg = blockIdx.x % segs;
  const uint32_t lead = row_lead(a, si), row_end = lead + a.n_dst;
  const uint32_t p_begin = sg * SEG, p_end = min(p_begin + SEG, row_end);
  const int64_t cell0 = (int64_t)si * a.n_dst - lead;  // of position 0, a multiple of 4
  uint4 dur[VEC];
  load_step(a.m + cell0, p_begin, lead, p_end, dur);
  const uint4 ri = info[si];
  const uint32_t nbw = min(BITMAP_WORDS, (*bound >> 5) + 1), lim = nbw * 32;
  const bool bitmap_only = (*bound >> 5) < BITMAP_WORDS;
  const uint32_t mode = ri.x, len = ri.y;
  const uint64_t lo = ri.z | ((uint64_t)ri.w << 32);
  if (mode == RL_MISSING && threadIdx.x == 0) atomicOr(err, ERR_NO_LIST);
  if (mode == RL_SMEM) stage_row_list(rl, a.mask + lo, len, nbw, bitmap_only);
  const uint32_t* lg = a.mask + lo;
  const uint32_t os = a.src_orig[si];
  bool bad_hit = false;
  for (uint32_t b0 = p_begin; b0 < p_end; b0 += CELLS4) {
    uint4 lat[VEC];
    if (a.lat) load_step(a.lat + cell0, b0, lead, p_end, lat);
#pragma unroll
    for (uint32_t u = 0; u < VEC; ++u) {
      const uint32_t p = b0 + (u * TPB + threadIdx.x) * 4;
      if (p >= p_end) break;  // later quads lie further on
      const uint32_t dv[4] = {dur[u].x, dur[u].y, dur[u].z, dur[u].w};
      const uint32_t lv[4] = {a.lat ? lat[u].x : MAXV, a.lat ? lat[u].y : MAXV,
                              a.lat ? lat[u].z : MAXV, a.lat ? lat[u].w : MAXV};
      const bool whole = p >= lead && p + 4 <= p_end;
      uint32_t t4[4], du[4], ln[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const bool real = whole || (p + k >= lead && p + k < p_end);
        const uint32_t x = real ? a.dst_orig[p + k - lead] : 0u, d = dv[k];
        t4[k] = x;
        bool in = real && d <= a.threshold && d != MAXV;
        if (in) {
          if (mode == RL_SMEM && x < lim) in = (rl.bmp[x >> 5] >> (x & 31)) & 1u;
          else if (mode == RL_SMEM) in = in_list(rl.v, len, x);
          else if (mode == RL_GLOBAL) in = in_list(lg, len, x);
          else in = false;
        }
        bad_hit |= mode == RL_BAD && real && d <= a.threshold && !(skip_sentinels && d == MAXV);
        const uint64_t ms = (uint64_t)d * 1000u;
        du[k] = !in || ms > MAXV ? MAXV : (uint32_t)ms;
        ln[k] = in ? lv[k] : MAXV;
      }
      const int64_t c = cell0 + p;
      if (whole) {
        __stcs(reinterpret_cast<uint4*>(o.s + c), make_uint4(os, os, os, os));
        __stcs(reinterpret_cast<uint4*>(o.t + c), make_uint4(t4[0], t4[1], t4[2], t4[3]));
        __stcs(reinterpret_cast<uint4*>(o.du + c), make_uint4(du[0], du[1], du[2], du[3]));
        __stcs(reinterpret_cast<uint4*>(o.di + c), make_uint4(ln[0], ln[1], ln[2], ln[3]));
      } else {
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          if (p + k < lead || p + k >= p_end) continue;
          o.s[c + k] = os;
          o.t[c + k] = t4[k];
          o.du[c + k] = du[k];
          o.di[c + k] = ln[k];
        }
      }
    }
    load_step(a.m + cell0, b0 + CELLS4, lead, p_end, dur);
  }
  if (bad_hit) atomicOr(err, ERR_BAD_LIST);
}

// Sparse pass 2 for wide rows: the segment's kept cells in order, a warp per
// row segment (no block barrier). 32 ballot words at a time (the next 32
// loading meanwhile) are expanded, a word a lane, into a list of kept
// positions in shared memory at the offsets of a shuffle scan of their
// popcounts; a full or final list is written out with a lane per cell. Bound
// by the latency of a segment's chain: the kept cells of a row are read side
// by side; walked word by word, each waited for its own duration.
// The same block's 420,000 kept cells: 24 us against 63.
constexpr uint32_t WLIST = 2048;  // positions a warp lists before it writes

__device__ __forceinline__ void write_list(const TileIn& a, const TileOut& o,
                                           const uint16_t* __restrict__ list, uint32_t fill,
                                           uint64_t k0, uint64_t cell0, uint32_t p0, uint32_t lead,
                                           uint32_t os) {
  for (uint32_t k = threadIdx.x & 31; k < fill; k += 32) {
    const uint32_t col = p0 + list[k] - lead;
    const uint64_t cell = cell0 + col;
    put(a, o, k0 + k, cell, os, a.dst_orig[col], a.m[cell]);
  }
}

__global__ void __launch_bounds__(TPB)
    k_tile_write_rows(TileIn a, TileOut o, uint64_t nseg, uint32_t segs, uint32_t wpr,
                      const unsigned long long* __restrict__ pre,
                      const uint32_t* __restrict__ keep_bits) {
  static_assert(SEG <= 65536, "list entries are positions of a segment in 16 bits");
  __shared__ uint16_t lists[TPB / 32][WLIST];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t seg = (uint64_t)blockIdx.x * (TPB / 32) + wid;
  if (seg >= nseg) return;
  unsigned long long k0 = pre[seg];
  if (pre[seg + 1] == k0) return;  // nothing kept in this segment (uniform per warp)
  uint16_t* list = lists[wid];
  const uint32_t si = (uint32_t)(seg / segs), sg = (uint32_t)(seg % segs);
  const uint32_t lead = row_lead(a, si);
  const uint32_t w_begin = sg * SEG_WORDS;
  const uint32_t w_end = min(w_begin + SEG_WORDS, (lead + a.n_dst + 31) / 32);
  const uint32_t* bits_row = keep_bits + (uint64_t)si * wpr;
  const uint32_t os = a.src_orig[si];
  const uint64_t row0 = (uint64_t)si * a.n_dst;
  uint32_t fill = 0;
  uint32_t bits = w_begin + lane < w_end ? bits_row[w_begin + lane] : 0u;
  for (uint32_t w0 = w_begin; w0 < w_end; w0 += 32) {
    const uint32_t wn = w0 + 32 + lane;
    const uint32_t nbits = wn < w_end ? bits_row[wn] : 0u;
    const uint32_t cn = __popc(bits);
    uint32_t inc = cn;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 31);  // at most 1024
    if (fill + total > WLIST) {  // uniform per warp
      __syncwarp();
      write_list(a, o, list, fill, k0, row0, w_begin * 32, lead, os);
      k0 += fill;
      fill = 0;
      __syncwarp();
    }
    uint32_t at = fill + inc - cn;
    const uint32_t p = (w0 - w_begin + lane) * 32;
    for (uint32_t b = bits; b; b &= b - 1) list[at++] = (uint16_t)(p + __ffs(b) - 1);
    fill += total;
    bits = nbits;
  }
  __syncwarp();
  write_list(a, o, list, fill, k0, row0, w_begin * 32, lead, os);
}

// Exclusive scan of up to SCAN_ONE counts in one block (out[n] = total): a
// warp scans a contiguous run of them, all its loads at once. One launch
// instead of the three of a scan over many blocks, which at this size are all
// gap: 12 us and two gaps for 10,000 counts against 7.
constexpr uint32_t SCAN_RUN = 16, SCAN_ONE = SCAN_TPB * SCAN_RUN;

__global__ void __launch_bounds__(SCAN_TPB)
    k_tile_scan(const unsigned long long* __restrict__ cnt, uint32_t n,
                unsigned long long* __restrict__ out) {
  static_assert((uint64_t)SCAN_ONE * SEG <= 0xFFFFFFFFull, "sums fit 32 bits");
  __shared__ uint32_t sums[SCAN_TPB / 32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t b0 = wid * 32 * SCAN_RUN + lane;
  uint32_t v[SCAN_RUN], carry = 0;  // inclusive within the warp's run
#pragma unroll
  for (uint32_t j = 0; j < SCAN_RUN; ++j) v[j] = b0 + 32 * j < n ? (uint32_t)cnt[b0 + 32 * j] : 0u;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1)
#pragma unroll
    for (uint32_t j = 0; j < SCAN_RUN; ++j) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v[j], d);
      if (lane >= d) v[j] += y;
    }
#pragma unroll
  for (uint32_t j = 0; j < SCAN_RUN; ++j) {
    const uint32_t t = __shfl_sync(0xFFFFFFFFu, v[j], 31);
    v[j] += carry;
    carry += t;
  }
  if (lane == 0) sums[wid] = carry;
  __syncthreads();
  uint32_t before = lane < wid ? sums[lane] : 0u;
#pragma unroll
  for (uint32_t d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, d);
  if (threadIdx.x == 0) out[0] = 0;
#pragma unroll
  for (uint32_t j = 0; j < SCAN_RUN; ++j)
    if (b0 + 32 * j < n) out[b0 + 32 * j + 1] = before + v[j];
}

// Sparse pass 2: the block's kept cells, in order, from pass 1's ballots:
// a thread's output slot is the block's offset plus the kept cells of the
// earlier words of the block (a two-warp shuffle scan of the word counts)
// and the lower lanes of its own word. A kept cell passed the bound and its
// radius list in pass 1, so its duration is written as read.
__global__ void __launch_bounds__(TPB)
    k_tile_write(TileIn a, TileOut o, uint64_t n, bool narrow,
                 const unsigned long long* __restrict__ pre,
                 const uint32_t* __restrict__ keep_bits) {
  constexpr uint32_t WORDS = CELLS / 32;
  static_assert(WORDS == 64 && TPB >= 64, "two warps scan the block's 64 ballot words");
  __shared__ uint32_t wpre[WORDS];
  __shared__ uint32_t half;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned long long k0 = pre[blockIdx.x];
  if (pre[blockIdx.x + 1] == k0) return;  // nothing kept in this block (uniform)
  const uint64_t base = (uint64_t)blockIdx.x * CELLS;
  const uint64_t w0 = base / 32, nw = (n + 31) / 32;
  if (wid < 2) {
    const uint32_t w = wid * 32 + lane;
    const uint32_t c = w0 + w < nw ? __popc(keep_bits[w0 + w]) : 0;
    uint32_t inc = c;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, d);
      if (lane >= d) inc += y;
    }
    wpre[w] = inc - c;
    if (wid == 0 && lane == 31) half = inc;
  }
  __syncthreads();
  for (uint32_t w = wid; w < WORDS; w += TPB / 32) {
    if (w0 + w >= nw) break;
    const uint32_t bits = keep_bits[w0 + w];
    if (!((bits >> lane) & 1u)) continue;
    const uint64_t i = (w0 + w) * 32 + lane;
    uint32_t si, di;
    split(i, a.n_dst, narrow, &si, &di);
    const uint32_t slot = wpre[w] + (w >= 32 ? half : 0u) + __popc(bits & ((1u << lane) - 1u));
    put(a, o, k0 + slot, i, a.src_orig[si], a.dst_orig[di], a.m[i]);
  }
}

// Scratch of the device variant and the host variant's copies, per device.
struct TileWs {
  std::mutex mu;
  cudaStream_t st = nullptr;
  void* buf[12] = {};
  size_t cap[12] = {};
  void* pin = nullptr;  // 16 bytes of pinned host memory: rows and error bits of a call
};
TileWs& tile_ws(int device) {
  static TileWs ws[64];
  return ws[device];
}

template <class T>
cudaError_t ws_get(TileWs& ws, int i, size_t bytes, T** p) {
  bytes = std::max<size_t>(bytes, 16);
  if (ws.cap[i] < bytes) {
    if (ws.buf[i]) cudaFree(ws.buf[i]);
    ws.buf[i] = nullptr;
    ws.cap[i] = 0;
    const cudaError_t e = cudaMalloc(&ws.buf[i], bytes);
    if (e != cudaSuccess) return e;
    ws.cap[i] = bytes;
  }
  *p = reinterpret_cast<T*>(ws.buf[i]);
  return cudaSuccess;
}

bf_status check_args(uint32_t n_src, uint32_t n_dst, const void* m, const void* so,
                     const void* dor, const bf_tile_columns* out, uint64_t* n_rows,
                     const void* mask_off, const void* mask, uint64_t n_mask) {
  const bool cells = (uint64_t)n_src * n_dst != 0;
  if (!out || !n_rows || (cells && (!m || !so || !dor)) ||
      (cells && (!out->source_idx || !out->target_idx || !out->duration_ms || !out->distance_m)) ||
      (mask_off && n_mask && !mask)) {
    set_error("bf_tile_emit: null argument");
    return BF_ERR_INVALID;
  }
  return BF_OK;
}

// Emission from device inputs into device columns on `st`; *n_rows after a
// synchronisation of the stream.
bf_status emit_device(TileWs& ws, const TileIn& a, const TileOut& o, cudaStream_t st,
                      uint64_t* n_rows) {
  const uint64_t n = (uint64_t)a.n_src * a.n_dst;
  uint32_t* d_err = nullptr;  // {error bits, largest destination id}
  BF_CUDA(ws_get(ws, 0, 8, &d_err));
  BF_CUDA(cudaMemsetAsync(d_err, 0, 8, st));
  if (!ws.pin) BF_CUDA(cudaMallocHost(&ws.pin, 16));
  uint64_t* const h_rows = reinterpret_cast<uint64_t*>(ws.pin);
  uint32_t* const h_err = reinterpret_cast<uint32_t*>(ws.pin) + 2;
  *h_rows = 0;
  const bool narrow = n <= 0xFFFFFFFFull;
  auto scan_counts = [&](unsigned long long* cnt, uint64_t nb) -> bf_status {
    if (nb <= SCAN_ONE) {
      k_tile_scan<<<1, SCAN_TPB, 0, st>>>(cnt, (uint32_t)nb, cnt + nb);
      return BF_OK;
    }
    uint64_t* d_bsum = nullptr;
    BF_CUDA(ws_get(ws, 10, ((nb + SCAN_BLOCK - 1) / SCAN_BLOCK + 2) * 8, &d_bsum));
    scan_launch<uint64_t>(U64Val{reinterpret_cast<const uint64_t*>(cnt)}, nb, d_bsum,
                          reinterpret_cast<uint64_t*>(cnt + nb), st);
    return BF_OK;
  };
  bf_status rc;
  // wide rows: a block per row segment (a row's 16-byte boundary lies up to 3
  // cells before its first), list records and the destination ids' range (from
  // which the blocks size their bitmaps) of all rows first
  const bool wide = a.n_dst >= ROW_MIN && a.n_dst <= 0xFFFFFFFFu - 2 * SEG &&
                    (uint64_t)a.n_src * ((a.n_dst + 3 + SEG - 1) / SEG) <= 0x7FFFFFFFull;
  const uint32_t segs = wide ? (a.n_dst + 3 + SEG - 1) / SEG : 0;
  uint4* d_info = nullptr;
  uint32_t* const d_bound = d_err + 1;
  auto row_lists = [&]() -> bf_status {
    BF_CUDA(ws_get(ws, 11, (uint64_t)a.n_src * 16, &d_info));
    const unsigned gi = (unsigned)std::min<uint64_t>(
        (std::max(a.n_src, a.n_dst) + TPB - 1) / TPB, 152 * 8);
    k_tile_rowinfo<<<gi, TPB, 0, st>>>(a, d_info, d_bound);
    return BF_OK;
  };
  if (n && !a.sparse) {
    auto al = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
    // which sentinel cells meet a bad list (an error) follows the row width
    const bool skip = a.n_dst % 4 == 0 && al(a.dst_orig);
    // four searches in a row per thread only pay once their threads fill the
    // chip: 300 x 130 cells with lists take 35 us a cell a thread, 40 us four
    const bool few = a.mask_off && !skip && n < FEW_CELLS;
    if (!few && al(a.m) && (!a.lat || al(a.lat)) && al(o.s) && al(o.t) && al(o.du) && al(o.di)) {
      if (wide && a.mask_off) {
        if ((rc = row_lists())) return rc;
        k_tile_dense_rows<<<(unsigned)(a.n_src * segs), TPB, 0, st>>>(a, o, segs, d_info, d_bound,
                                                                     skip, d_err);
      } else {
        const uint64_t nb = ((n + 3) / 4 + TPB - 1) / TPB;
        k_tile_dense4<<<(unsigned)std::min<uint64_t>(nb, 0x7FFFFFFF), TPB, 0, st>>>(
            a, o, n, narrow, skip, d_err);
      }
    } else {
      const unsigned gx =
          (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((a.n_dst + TPB - 1) / TPB, 64));
      const unsigned gy = (unsigned)std::min<uint64_t>(a.n_src, 65535);
      k_tile_dense<<<dim3(gx, gy), TPB, 0, st>>>(a, o, d_err);
    }
    BF_CUDA(cudaGetLastError());
    *h_rows = n;
  } else if (n && wide) {
    const uint32_t wpr = (a.n_dst + 3 + 31) / 32;
    const uint64_t nb = (uint64_t)a.n_src * segs;
    unsigned long long* d_cnt = nullptr;
    uint32_t* d_bits = nullptr;
    BF_CUDA(ws_get(ws, 1, (2 * nb + 1) * 8, &d_cnt));
    BF_CUDA(ws_get(ws, 9, (uint64_t)a.n_src * wpr * 4, &d_bits));
    if ((rc = row_lists())) return rc;
    k_tile_count_rows<<<(unsigned)nb, TPB, 0, st>>>(a, segs, wpr, d_info, d_bound, d_cnt, d_bits,
                                                    d_err);
    if ((rc = scan_counts(d_cnt, nb))) return rc;
    k_tile_write_rows<<<(unsigned)((nb + TPB / 32 - 1) / (TPB / 32)), TPB, 0, st>>>(
        a, o, nb, segs, wpr, d_cnt + nb, d_bits);
    BF_CUDA(cudaGetLastError());
    BF_CUDA(cudaMemcpyAsync(h_rows, d_cnt + 2 * nb, 8, cudaMemcpyDeviceToHost, st));
  } else if (n) {
    const uint64_t nb = (n + CELLS - 1) / CELLS;
    if (nb > 0x7FFFFFFFull) {
      set_error("bf_tile_emit: block too large");
      return BF_ERR_INVALID;
    }
    unsigned long long* d_cnt = nullptr;
    uint32_t* d_bits = nullptr;
    BF_CUDA(ws_get(ws, 1, (2 * nb + 1) * 8, &d_cnt));
    BF_CUDA(ws_get(ws, 9, nb * (CELLS / 32) * 4, &d_bits));
    k_tile_count<<<(unsigned)nb, TPB, 0, st>>>(a, n, narrow, d_cnt, d_bits, d_err);
    if ((rc = scan_counts(d_cnt, nb))) return rc;
    k_tile_write<<<(unsigned)nb, TPB, 0, st>>>(a, o, n, narrow, d_cnt + nb, d_bits);
    BF_CUDA(cudaGetLastError());
    BF_CUDA(cudaMemcpyAsync(h_rows, d_cnt + 2 * nb, 8, cudaMemcpyDeviceToHost, st));
  }
  BF_CUDA(cudaMemcpyAsync(h_err, d_err, 4, cudaMemcpyDeviceToHost, st));
  BF_CUDA(cudaStreamSynchronize(st));
  const uint32_t err = *h_err;
  if (err & ERR_NO_LIST) {
    set_error("bf_tile_emit: a source's original index has no radius list");
    return BF_ERR_INVALID;
  }
  if (err & ERR_BAD_LIST) {
    set_error("bf_tile_emit: a radius list's offsets decrease or run past the list array");
    return BF_ERR_INVALID;
  }
  *n_rows = *h_rows;
  return BF_OK;
}

bf_status set_device(int device) {
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev || device >= 64) {
    cudaGetLastError();
    set_error("bf_tile_emit: no such device");
    return BF_ERR_INVALID;
  }
  if (cudaSetDevice(device) != cudaSuccess) return cuda_status(cudaGetLastError(), "cudaSetDevice");
  return BF_OK;
}

}  // namespace

extern "C" {

bf_status bf_tile_emit_device(const uint32_t* d_matrix, const uint32_t* d_lat, uint32_t n_src,
                              uint32_t n_dst, const uint32_t* d_src_orig,
                              const uint32_t* d_dst_orig, uint32_t threshold,
                              const uint64_t* d_mask_off, const uint32_t* d_mask,
                              uint32_t n_mask_src, uint64_t n_mask, uint32_t sparse, int device,
                              void* stream, const bf_tile_columns* d_out, uint64_t* n_rows) {
  bf_status rc;
  if ((rc = check_args(n_src, n_dst, d_matrix, d_src_orig, d_dst_orig, d_out, n_rows, d_mask_off,
                       d_mask, n_mask)))
    return rc;
  if ((rc = set_device(device))) return rc;
  TileWs& ws = tile_ws(device);
  std::lock_guard<std::mutex> lk(ws.mu);
  if (!ws.st) BF_CUDA(cudaStreamCreateWithFlags(&ws.st, cudaStreamNonBlocking));
  cudaStream_t st = stream ? (cudaStream_t)stream : ws.st;
  const TileIn a{d_matrix, d_lat, n_src, n_dst, d_src_orig, d_dst_orig, threshold,
                 d_mask_off, d_mask, n_mask_src, n_mask, sparse};
  const TileOut o{d_out->source_idx, d_out->target_idx, d_out->duration_ms, d_out->distance_m};
  return emit_device(ws, a, o, st, n_rows);
}

bf_status bf_tile_emit(const uint32_t* matrix, const uint32_t* lat, uint32_t n_src,
                       uint32_t n_dst, const uint32_t* src_orig, const uint32_t* dst_orig,
                       uint32_t threshold, const uint64_t* mask_off, const uint32_t* mask,
                       uint32_t n_mask_src, uint32_t sparse, int device,
                       const bf_tile_columns* out, uint64_t* n_rows) {
  const uint64_t n_mask = mask_off ? mask_off[n_mask_src] : 0;
  bf_status rc;
  if ((rc = check_args(n_src, n_dst, matrix, src_orig, dst_orig, out, n_rows, mask_off, mask,
                       n_mask)))
    return rc;
  if (mask_off)
    for (uint32_t s = 0; s < n_mask_src; ++s)
      if (mask_off[s + 1] < mask_off[s]) {
        set_error("bf_tile_emit: radius list offsets must be non-decreasing");
        return BF_ERR_INVALID;
      }
  if ((rc = set_device(device))) return rc;
  TileWs& ws = tile_ws(device);
  std::lock_guard<std::mutex> lk(ws.mu);
  if (!ws.st) BF_CUDA(cudaStreamCreateWithFlags(&ws.st, cudaStreamNonBlocking));
  cudaStream_t st = ws.st;
  const uint64_t n = (uint64_t)n_src * n_dst;
  uint32_t *dm = nullptr, *dl = nullptr, *ds = nullptr, *dd = nullptr, *dmask = nullptr;
  uint64_t* dmoff = nullptr;
  uint32_t* dcol = nullptr;
  cudaError_t e = ws_get(ws, 2, n * 4, &dm);
  if (e == cudaSuccess && lat) e = ws_get(ws, 3, n * 4, &dl);
  if (e == cudaSuccess) e = ws_get(ws, 4, (uint64_t)n_src * 4, &ds);
  if (e == cudaSuccess) e = ws_get(ws, 5, (uint64_t)n_dst * 4, &dd);
  if (e == cudaSuccess && mask_off) e = ws_get(ws, 6, ((uint64_t)n_mask_src + 1) * 8, &dmoff);
  if (e == cudaSuccess && mask_off) e = ws_get(ws, 7, n_mask * 4, &dmask);
  if (e == cudaSuccess) e = ws_get(ws, 8, n * 16, &dcol);
  if (e != cudaSuccess) return cuda_status(e, "bf_tile_emit: device memory");
  auto up = [&](void* d, const void* h, uint64_t bytes) {
    if (e == cudaSuccess && bytes) e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st);
  };
  up(dm, matrix, n * 4);
  if (lat) up(dl, lat, n * 4);
  up(ds, src_orig, (uint64_t)n_src * 4);
  up(dd, dst_orig, (uint64_t)n_dst * 4);
  if (mask_off) {
    up(dmoff, mask_off, ((uint64_t)n_mask_src + 1) * 8);
    up(dmask, mask, n_mask * 4);
  }
  if (e != cudaSuccess) return cuda_status(e, "bf_tile_emit: upload");
  const TileIn a{dm, lat ? dl : nullptr, n_src, n_dst, ds, dd, threshold,
                 mask_off ? dmoff : nullptr, dmask, n_mask_src, n_mask, sparse};
  const TileOut o{dcol, dcol + n, dcol + 2 * n, dcol + 3 * n};
  uint64_t rows = 0;
  if ((rc = emit_device(ws, a, o, st, &rows))) return rc;
  uint32_t* dst_cols[4] = {out->source_idx, out->target_idx, out->duration_ms, out->distance_m};
  for (int c = 0; c < 4 && rows; ++c)
    BF_CUDA(cudaMemcpyAsync(dst_cols[c], dcol + (uint64_t)c * n, rows * 4, cudaMemcpyDeviceToHost,
                            st));
  BF_CUDA(cudaStreamSynchronize(st));
  *n_rows = rows;
  return BF_OK;
}

void bf_tile_release(int device) {
  if (device < 0 || device >= 64) return;
  TileWs& ws = tile_ws(device);
  std::lock_guard<std::mutex> lk(ws.mu);
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (ws.st) cudaStreamSynchronize(ws.st);
  for (int i = 0; i < 12; ++i) {
    if (ws.buf[i]) cudaFree(ws.buf[i]);
    ws.buf[i] = nullptr;
    ws.cap[i] = 0;
  }
  if (ws.pin) cudaFreeHost(ws.pin);
  ws.pin = nullptr;
  if (ws.st) cudaStreamDestroy(ws.st);
  ws.st = nullptr;
}

}  // extern "C"
