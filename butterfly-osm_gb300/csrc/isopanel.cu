// isopanel.cu — isochrone waves over panels.
//
// A wave's lanes (origins in (threshold, rank) order) are cut into tiles of 64
// lanes, each with its own 16-bit slab [row][64] (a row of a tile is one
// 128-byte line; rows are ranks). Neighbouring lanes share a threshold and a
// neighbourhood, so a tile reaches a small part of the graph although the wave
// reaches all of it: every row carries a word with a bit per tile that holds a
// label within its lane's threshold there. A unit of work is a panel (panel.cu)
// in one tile: it is skipped when none of the panel's sources and seeded rows is
// active in the tile, only active sources are gathered, and only rows that
// become active are written (nothing reads the others). Labels above a lane's
// threshold are not cut: they only lead to labels above it, and whoever reads a
// label compares it with the threshold.
//
// Panels of more than four rows take a warp each, a thread holding two lanes (one
// packed word per row); smaller ones, most of a road graph, eight threads of
// eight lanes. Levels of few panels take a block per unit, whose warps share the
// sources.
//
// Bound by latency in the upper levels and by the records and activity of
// inactive panels in the lower ones. 1500 origins of 5 to 60 minutes on the
// country graph: the wave-wide item sweep gathered and wrote 200 GB in 60 ms,
// the tiles 17 GB in 16 ms; five origins on the 1000 x 1250 region 3.0 -> 1.0
// ms. On the way: a warp per unit also for small panels 50 ms, tiles walked one
// after the other also in levels of few panels 21 ms.

#include <algorithm>

#include "engine.cuh"

namespace bf {

namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;

struct IsoArgs {
  const uint4* pan;        // panels (Panels::d_a, d_b)
  const uint2* panb;
  const uint32_t* src;     // source ranks
  const uint32_t* w;       // weight tiles, both halfwords alike
  uint32_t n;
  uint32_t* slab;          // [tiles][n][32] two lanes a word
  uint32_t* act;           // [n] tiles in which the row holds a label within its threshold
  const uint32_t* seeded;  // [n] tiles in which the row was reset and may hold seeds
  const uint32_t* thr;     // [tiles][32] thresholds, two lanes a word
  unsigned long long* cnt;  // bytes gathered and written, rows written (or null)
};

// min(acc, d + w) on both halfwords. SAT: any thresholds below 0xFFFF; sums
// saturate at 0xFFFF. Otherwise thresholds are below 0x7FFF, labels at most
// 0x8000 and weights at most 0x7FFF, so no sum wraps.
template <bool SAT>
__device__ __forceinline__ uint32_t relax2(uint32_t d, uint32_t w, uint32_t acc) {
  return SAT ? __viaddmin_u16x2(__vminu2(d, ~w), w, acc) : __viaddmin_u16x2(d, w, acc);
}
template <bool SAT>
constexpr uint32_t far2 = SAT ? 0xFFFFFFFFu : 0x80008000u;

struct IsoPanel {
  uint32_t hi, live, stride, nu, u0, w0;
};
__device__ __forceinline__ IsoPanel iso_panel(const uint4 a, const uint2 b) {
  return IsoPanel{a.x, a.y & 0xFF, (a.y >> 8) & 0xFF, a.z, b.x, b.y};
}

template <uint32_t K, bool SAT>
__device__ __forceinline__ void relax_source(uint32_t v, const uint32_t* w, uint32_t (&acc)[K]) {
  if constexpr (K >= 4) {
#pragma unroll
    for (uint32_t j = 0; j < K; j += 4) {
      const uint4 x = *reinterpret_cast<const uint4*>(w + j);
      acc[j] = relax2<SAT>(v, x.x, acc[j]);
      acc[j + 1] = relax2<SAT>(v, x.y, acc[j + 1]);
      acc[j + 2] = relax2<SAT>(v, x.z, acc[j + 2]);
      acc[j + 3] = relax2<SAT>(v, x.w, acc[j + 3]);
    }
  } else if constexpr (K == 2) {
    const uint2 x = *reinterpret_cast<const uint2*>(w);
    acc[0] = relax2<SAT>(v, x.x, acc[0]);
    acc[1] = relax2<SAT>(v, x.y, acc[1]);
  } else {
    acc[0] = relax2<SAT>(v, *w, acc[0]);
  }
}

// The sources base + (set bits of bm) of a unit, F rows in flight. s: the
// source rank of base + lane.
template <uint32_t K, bool SAT, uint32_t F = 4>
__device__ __forceinline__ void relax_active(uint32_t bm, uint32_t s, const uint32_t* w,
                                             uint32_t stride, const uint32_t* slab, uint32_t lane,
                                             uint32_t (&acc)[K]) {
  while (bm) {
    uint32_t i[F], v[F];
#pragma unroll
    for (uint32_t q = 0; q < F; ++q) {
      i[q] = bm ? __ffs(bm) - 1 : 32u;
      bm &= bm - 1;
      if (i[q] < 32) {
        const uint32_t r = __shfl_sync(FULL, s, i[q]);
        v[q] = __ldcg(slab + (size_t)r * 32 + lane);
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < F; ++q)
      if (i[q] < 32) relax_source<K, SAT>(v[q], w + (size_t)i[q] * stride, acc);
  }
}

// Seeds, triangle, activity and rows of a unit. sd: bit j set when row j was
// reset. Returns the number of rows written.
template <uint32_t K, bool SAT>
__device__ __forceinline__ uint32_t finish_unit(const IsoArgs& g, const IsoPanel& p, uint32_t t,
                                                uint32_t sd, const uint32_t* tri, uint32_t* slab,
                                                uint32_t lane, uint32_t (&acc)[K]) {
  if (sd) {
#pragma unroll
    for (uint32_t j = 0; j < K; ++j)
      if ((sd >> j) & 1u) acc[j] = __vminu2(acc[j], __ldcg(slab + (size_t)(p.hi - j) * 32 + lane));
  }
#pragma unroll
  for (uint32_t i = 0; i + 1 < K; ++i) {
    if constexpr (K >= 4) {
#pragma unroll
      for (uint32_t v = (i + 1) / 4; v < K / 4; ++v) {
        const uint4 x = *reinterpret_cast<const uint4*>(tri + i * p.stride + 4 * v);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          if (4 * v + q > i) acc[4 * v + q] = relax2<SAT>(acc[i], w[q], acc[4 * v + q]);
      }
    } else {
#pragma unroll
      for (uint32_t j = i + 1; j < K; ++j)
        acc[j] = relax2<SAT>(acc[i], tri[i * p.stride + j], acc[j]);
    }
  }
  const uint32_t thr = g.thr[t * 32 + lane];
  uint32_t rows = 0;  // rows with a label within its threshold
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) {
    if (j >= p.live) break;
    // a halfword of x is zero where the label is within the threshold
    const uint32_t x = __vminu2(acc[j], thr) ^ acc[j];
    if (__any_sync(FULL, ((x - 0x00010001u) & ~x & 0x80008000u) != 0)) {
      rows |= 1u << j;
      slab[(size_t)(p.hi - j) * 32 + lane] = acc[j];
    }
  }
  if ((rows >> lane) & 1u) atomicOr(&g.act[p.hi - lane], 1u << t);
  return __popc(rows);
}

// One unit by a warp. s, am: ranks and activity of the first 32 sources.
template <uint32_t K, bool SAT>
__device__ __forceinline__ void iso_unit(const IsoArgs& g, const IsoPanel& p, uint32_t t,
                                         uint32_t s, uint32_t am, uint32_t seeds, uint32_t lane,
                                         uint32_t& gathered, uint32_t& written) {
  uint32_t acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = far2<SAT>;
  uint32_t* slab = g.slab + (size_t)t * g.n * 32;
  const uint32_t sd = __ballot_sync(FULL, (seeds >> t) & 1u);
  for (uint32_t base = 0;;) {
    const uint32_t bm = __ballot_sync(FULL, (am >> t) & 1u);
    gathered += __popc(bm);
    relax_active<K, SAT>(bm, s, g.w + p.w0 + (size_t)base * p.stride, p.stride, slab, lane, acc);
    base += 32;
    if (base >= p.nu) break;
    s = base + lane < p.nu ? g.src[p.u0 + base + lane] : 0u;
    am = base + lane < p.nu ? __ldcg(g.act + s) : 0u;
  }
  written += finish_unit<K, SAT>(g, p, t, sd, g.w + p.w0 + (size_t)p.nu * p.stride, slab, lane,
                                 acc);
}

template <bool SAT>
__device__ __forceinline__ void iso_units(const IsoArgs& g, const IsoPanel& p, uint32_t mask,
                                          uint32_t s, uint32_t am, uint32_t seeds, uint32_t lane,
                                          uint32_t& gathered, uint32_t& written) {
  while (mask) {
    const uint32_t t = __ffs(mask) - 1;
    mask &= mask - 1;
#define BF_ISO(K) iso_unit<K, SAT>(g, p, t, s, am, seeds, lane, gathered, written)
    if (p.live > 8) BF_ISO(16);
    else BF_ISO(8);
#undef BF_ISO
  }
}

__device__ __forceinline__ void iso_count(const IsoArgs& g, uint32_t lane, uint64_t gathered,
                                          uint64_t written) {
  if (g.cnt && lane == 0 && (gathered | written)) {
    atomicAdd(&g.cnt[0], (gathered + written) * 128ull);
    atomicAdd(&g.cnt[1], (unsigned long long)written);
  }
}

// Panels of at most four rows: eight threads of eight lanes (four words) each.
// All groups of the warp walk together: `t` is the group's tile where on.
template <bool SAT>
__device__ __forceinline__ void small_unit(const IsoArgs& g, const IsoPanel& p, bool on, uint32_t t,
                                           uint32_t s, uint32_t am, uint32_t seeds, uint32_t most,
                                           uint32_t lane, uint32_t& gathered, uint32_t& written) {
  const uint32_t gl = lane & 7, g0 = lane & 24;
  uint32_t* slab = g.slab + (size_t)t * g.n * 32 + gl * 4;
  const uint32_t* w = g.w + p.w0;
  uint32_t acc[4][4];
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
    for (uint32_t l = 0; l < 4; ++l) acc[j][l] = far2<SAT>;
  auto relax_row = [&](const uint4& v, const uint4& x) {
    const uint32_t d[4] = {v.x, v.y, v.z, v.w}, wj[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
      for (uint32_t l = 0; l < 4; ++l) acc[j][l] = relax2<SAT>(d[l], wj[j], acc[j][l]);
  };
  for (uint32_t q0 = 0; q0 < most; q0 += 2) {  // two sources in flight
    uint4 v[2], x[2];
    bool use[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t q = q0 + h;
      uint32_t sq, aq;
      if (q0 < 8) {
        sq = __shfl_sync(FULL, s, g0 + q);
        aq = __shfl_sync(FULL, am, g0 + q);
      } else {
        sq = q < p.nu ? g.src[p.u0 + q] : 0u;
        aq = q < p.nu ? __ldcg(g.act + sq) : 0u;
      }
      use[h] = on && q < p.nu && ((aq >> t) & 1u);
      if (use[h]) {
        v[h] = __ldcg(reinterpret_cast<const uint4*>(slab + (size_t)sq * 32));
        x[h] = *reinterpret_cast<const uint4*>(w + q * 4);
        ++gathered;
      }
    }
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h)
      if (use[h]) relax_row(v[h], x[h]);
  }
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    const uint32_t sj = __shfl_sync(FULL, seeds, g0 + j);
    if (on && j < p.live && ((sj >> t) & 1u)) {
      const uint4 v = __ldcg(reinterpret_cast<const uint4*>(slab + (size_t)(p.hi - j) * 32));
      acc[j][0] = __vminu2(acc[j][0], v.x), acc[j][1] = __vminu2(acc[j][1], v.y);
      acc[j][2] = __vminu2(acc[j][2], v.z), acc[j][3] = __vminu2(acc[j][3], v.w);
    }
  }
  if (on && p.live > 1) {
    const uint4* tri = reinterpret_cast<const uint4*>(w + (size_t)p.nu * 4);
    const uint4 r0 = tri[0], r1 = tri[1], r2 = tri[2];
#pragma unroll
    for (uint32_t l = 0; l < 4; ++l) {
      acc[1][l] = relax2<SAT>(acc[0][l], r0.y, acc[1][l]);
      acc[2][l] = relax2<SAT>(acc[0][l], r0.z, acc[2][l]);
      acc[3][l] = relax2<SAT>(acc[0][l], r0.w, acc[3][l]);
      acc[2][l] = relax2<SAT>(acc[1][l], r1.z, acc[2][l]);
      acc[3][l] = relax2<SAT>(acc[1][l], r1.w, acc[3][l]);
      acc[3][l] = relax2<SAT>(acc[2][l], r2.w, acc[3][l]);
    }
  }
  const uint4 th = *reinterpret_cast<const uint4*>(g.thr + (on ? t : 0u) * 32 + gl * 4);
  const uint32_t thr[4] = {th.x, th.y, th.z, th.w};
  uint32_t rows = 0;
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    uint32_t in = 0;
#pragma unroll
    for (uint32_t l = 0; l < 4; ++l) {
      const uint32_t x = __vminu2(acc[j][l], thr[l]) ^ acc[j][l];
      in |= (x - 0x00010001u) & ~x & 0x80008000u;
    }
    const uint32_t b = __ballot_sync(FULL, on && j < p.live && in != 0);
    if ((b >> g0) & 0xFFu) {
      rows |= 1u << j;
      *reinterpret_cast<uint4*>(slab + (size_t)(p.hi - j) * 32) =
          make_uint4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
    }
  }
  if ((rows >> gl) & 1u) atomicOr(&g.act[p.hi - gl], 1u << t);
  written += __popc(rows);
}

// A level: blocks [0, big_blocks) take the panels [p0, pb) of more than four
// rows, a warp each, the others the panels [pb, p1), eight threads each, and
// blockIdx.y every gridDim.y-th tile. What does not depend on the level before
// (records, source ranks, reset flags) is loaded while that level drains.
// Four blocks an SM leave a thread 64 registers, so the three bodies in it spill
// some 200 bytes. Wide levels are bound by issue and load latency, not by memory:
// two of them, 1024 origins on the 1000 x 1250 region, take 581 and 687 us at 1.5
// TB/s of DRAM, the schedulers issuing in 53 % of the cycles with 24 warps an SM.
template <bool SAT>
__global__ void __launch_bounds__(256, 4)
    k_iso_panels(const IsoArgs g, uint32_t p0, uint32_t pb, uint32_t p1, uint32_t big_blocks) {
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t lane = threadIdx.x & 31;
  uint32_t tiles = 0;  // this block's
  for (uint32_t t = blockIdx.y; t < 32; t += gridDim.y) tiles |= 1u << t;
  uint32_t gathered = 0, written = 0;
  if (blockIdx.x < big_blocks) {
    const uint32_t at = p0 + blockIdx.x * 8 + (threadIdx.x >> 5);
    if (at >= pb) return;
    const IsoPanel p = iso_panel(g.pan[at], g.panb[at]);
    const uint32_t s = lane < p.nu ? g.src[p.u0 + lane] : 0u;
    const uint32_t seeds = lane < p.live ? g.seeded[p.hi - lane] : 0u;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t am = lane < p.nu ? __ldcg(g.act + s) : 0u;
    uint32_t m = am | seeds;
    for (uint32_t q = 32 + lane; q < p.nu; q += 32) m |= __ldcg(g.act + g.src[p.u0 + q]);
    m = __reduce_or_sync(FULL, m) & tiles;
    if (m) iso_units<SAT>(g, p, m, s, am, seeds, lane, gathered, written);
  } else {
    const uint32_t gl = lane & 7;
    const uint32_t at = pb + (blockIdx.x - big_blocks) * 32 + (threadIdx.x >> 3);
    IsoPanel p{0, 0, 4, 0, 0, 0};
    if (at < p1) p = iso_panel(g.pan[at], g.panb[at]);
    const uint32_t s = gl < p.nu ? g.src[p.u0 + gl] : 0u;
    const uint32_t seeds = gl < p.live ? g.seeded[p.hi - gl] : 0u;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t am = gl < p.nu ? __ldcg(g.act + s) : 0u;
    uint32_t m = am | seeds;
    for (uint32_t q = 8 + gl; q < p.nu; q += 8) m |= __ldcg(g.act + g.src[p.u0 + q]);
    m |= __shfl_xor_sync(FULL, m, 1);
    m |= __shfl_xor_sync(FULL, m, 2);
    m |= __shfl_xor_sync(FULL, m, 4);
    m &= tiles;
    while (__any_sync(FULL, m != 0)) {
      const uint32_t most = __reduce_max_sync(FULL, m ? p.nu : 0u);
      const uint32_t t = m ? __ffs(m) - 1 : 0u;
      small_unit<SAT>(g, p, m != 0, t, s, am, seeds, most, lane, gathered, written);
      m &= m - 1;
    }
    gathered = gl == 0 ? gathered : 0u;
    written = gl == 0 ? written : 0u;
    gathered = __reduce_add_sync(FULL, gathered);
    written = __reduce_add_sync(FULL, written);
  }
  iso_count(g, lane, gathered, written);
}

// A level of few panels: a block per unit (panel p0 + blockIdx.x, tile
// blockIdx.y), each warp an eighth of up to 256 sources, whose weights are staged
// while the level before drains, as are the seeds. Five origins on the 1000 x 1250
// region, whole call: 1.31 ms against 1.44 with four rows in flight, groups of 32
// sources a warp and the seeds read at the end.
constexpr uint32_t ISO_WARPS = 8, ISO_CH = 256;
struct IsoSplitSmem {
  uint32_t w[ISO_CH * PANEL_ROWS];
  uint32_t tri[PANEL_ROWS * PANEL_ROWS];
  uint32_t src[ISO_CH];
  uint32_t red[ISO_WARPS][PANEL_ROWS][32];
  uint32_t seed[PANEL_ROWS][32];
};

template <uint32_t K, bool SAT>
__device__ __forceinline__ void iso_block_unit(const IsoArgs& g, const IsoPanel& p, uint32_t t,
                                               IsoSplitSmem& sm) {
  constexpr uint32_t TPB = 32 * ISO_WARPS;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t* w = g.w + p.w0;
  auto stage = [&](uint32_t c0, uint32_t m) {
    for (uint32_t i = tid; i < m; i += TPB) sm.src[i] = g.src[p.u0 + c0 + i];
    const uint4* s4 = reinterpret_cast<const uint4*>(w + (size_t)c0 * p.stride);
    for (uint32_t i = tid; i < m * p.stride / 4; i += TPB)
      reinterpret_cast<uint4*>(sm.w)[i] = s4[i];
  };
  stage(0, min(p.nu, ISO_CH));
  for (uint32_t i = tid; i < p.stride * p.stride; i += TPB) sm.tri[i] = w[(size_t)p.nu * p.stride + i];
  const uint32_t seeds = lane < p.live ? g.seeded[p.hi - lane] : 0u;
  const uint32_t sd = __ballot_sync(FULL, (seeds >> t) & 1u);
  uint32_t* slab = g.slab + (size_t)t * g.n * 32;
  // (seeds are written before the first level is launched)
  for (uint32_t j = warp; j < K; j += ISO_WARPS)
    sm.seed[j][lane] =
        (sd >> j) & 1u ? __ldcg(slab + (size_t)(p.hi - j) * 32 + lane) : far2<SAT>;
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = far2<SAT>;
  uint32_t gathered = 0;
  for (uint32_t c0 = 0; c0 < p.nu; c0 += ISO_CH) {
    const uint32_t m = min(p.nu - c0, ISO_CH);
    if (c0) {
      __syncthreads();
      stage(c0, m);
      __syncthreads();
    }
    const uint32_t each = (m + ISO_WARPS - 1) / ISO_WARPS, base = warp * each;  // (at most 32)
    if (base < m) {
      const bool in = lane < each && base + lane < m;
      const uint32_t s = in ? sm.src[base + lane] : 0u;
      const uint32_t am = in ? __ldcg(g.act + s) : 0u;
      const uint32_t bm = __ballot_sync(FULL, (am >> t) & 1u);
      gathered += __popc(bm);
      relax_active<K, SAT, 8>(bm, s, sm.w + base * p.stride, p.stride, slab, lane, acc);
    }
  }
  if (!__syncthreads_or(gathered | sd)) return;
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) sm.red[warp][j][lane] = acc[j];
  __syncthreads();
  for (uint32_t j = warp; j < K; j += ISO_WARPS) {
    uint32_t v = sm.seed[j][lane];
#pragma unroll
    for (uint32_t q = 0; q < ISO_WARPS; ++q) v = __vminu2(v, sm.red[q][j][lane]);
    sm.red[0][j][lane] = v;
  }
  __syncthreads();
  uint32_t written = 0;
  if (warp == 0) {
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) acc[j] = sm.red[0][j][lane];
    written = finish_unit<K, SAT>(g, p, t, 0, sm.tri, slab, lane, acc);  // (seeds are in)
  }
  iso_count(g, lane, gathered, written);
}

template <bool SAT>
__global__ void __launch_bounds__(32 * ISO_WARPS) k_iso_split(const IsoArgs g, uint32_t p0) {
  __shared__ __align__(16) IsoSplitSmem sm;
  asm volatile("griddepcontrol.launch_dependents;");
  const IsoPanel p = iso_panel(g.pan[p0 + blockIdx.x], g.panb[p0 + blockIdx.x]);
  const uint32_t t = blockIdx.y;
  if (p.live > 8) iso_block_unit<16, SAT>(g, p, t, sm);
  else if (p.live > 4) iso_block_unit<8, SAT>(g, p, t, sm);
  else iso_block_unit<4, SAT>(g, p, t, sm);
}

// Rows of the origins' root paths, in their lanes' tiles: a warp per origin,
// stopping where another warp of its tile has been.
__global__ void __launch_bounds__(128)
    k_iso_mark(const uint32_t* __restrict__ orig, uint32_t k, const uint32_t* __restrict__ parent,
               const uint32_t* __restrict__ run_end, uint32_t* __restrict__ seeded) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= k) return;
  const uint32_t bit = 1u << (w >> 6);
  uint32_t x = orig[w];
  for (uint32_t guard = 0; x != NONE && guard < (1u << 30); ++guard) {
    if (*(volatile uint32_t*)&seeded[x] & bit) break;
    const uint32_t e = run_end[x];
    for (uint32_t r = x + lane; r <= e; r += 32) atomicOr(&seeded[r], bit);
    __syncwarp();
    x = parent[e];
  }
}

// Reset the seeded rows: a warp per 32 rows, one 128-byte line a store.
__global__ void __launch_bounds__(256)
    k_iso_reset(const uint32_t* __restrict__ seeded, uint32_t n, uint32_t* __restrict__ slab,
                uint32_t fill) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * blockDim.x / 32;
  for (uint64_t r0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; r0 < n;
       r0 += (uint64_t)warps * 32) {
    const uint32_t m = r0 + lane < n ? seeded[r0 + lane] : 0u;
    uint32_t any = __ballot_sync(FULL, m != 0);
    while (any) {
      const uint32_t i = __ffs(any) - 1;
      any &= any - 1;
      uint32_t mm = __shfl_sync(FULL, m, i);
      while (mm) {
        const uint32_t t = __ffs(mm) - 1;
        mm &= mm - 1;
        slab[((size_t)t * n + r0 + i) * 32 + lane] = fill;
      }
    }
  }
}

// Bitset rows of a wave (out_row[l] for lane l, w32 words each) and counts: a
// block owns 2048 ranks of one tile; a warp turns 32 ranks x 64 lanes into a
// word per lane by ballots, staged in shared memory so that a lane's 64 words
// are written as one 256-byte run. Bound by the latency of the active rows' loads
// and of the staging: 1024 origins on the 1000 x 1250 region, 915 us for 2.6 GB
// read and 0.37 GB written (3.3 TB/s).
constexpr uint32_t IB_RANKS = 2048;
__global__ void __launch_bounds__(256)
    k_iso_bits(const uint32_t* __restrict__ slab, uint32_t n, const uint32_t* __restrict__ act,
               const uint32_t* __restrict__ lane_thr, uint32_t kw, uint32_t* __restrict__ bits,
               uint64_t w32, unsigned long long* __restrict__ counts,
               const uint32_t* __restrict__ out_row) {
  __shared__ uint32_t sw[64][IB_RANKS / 32 + 1];
  __shared__ uint32_t sthr[64];
  const uint32_t r0 = blockIdx.x * IB_RANKS, t = blockIdx.y, l0 = t * 64;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < 64) sthr[threadIdx.x] = l0 + threadIdx.x < kw ? lane_thr[l0 + threadIdx.x] : 0u;
  __syncthreads();
  const uint32_t* tile = slab + (size_t)t * n * 32;
  for (uint32_t gi = warp; gi < IB_RANKS / 32; gi += 8) {
    const uint32_t rank = r0 + gi * 32 + lane;
    const bool on = rank < n && ((act[rank] >> t) & 1u);
    if (!__any_sync(FULL, on)) {
      sw[lane][gi] = 0;
      sw[lane + 32][gi] = 0;
      continue;
    }
    uint4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      v[q] = on ? *reinterpret_cast<const uint4*>(tile + (size_t)rank * 32 + 4 * q)
                : make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t w4[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const uint32_t j = 8 * q + h;  // lane within the tile
        const uint32_t d = (w4[h >> 1] >> ((h & 1) * 16)) & 0xFFFFu;
        const uint32_t word = __ballot_sync(FULL, d <= sthr[j] && on);
        if (lane == (j & 31)) sw[j][gi] = word;
      }
    }
  }
  __syncthreads();
  const uint32_t nl = kw > l0 ? min(64u, kw - l0) : 0u;
  const uint64_t wbase = r0 >> 5;
  for (uint32_t j = warp; j < nl; j += 8) {
    const uint64_t orow = out_row[l0 + j];
    uint32_t pc = 0;
    for (uint32_t k = lane; k < IB_RANKS / 32; k += 32) {
      const uint64_t wi = wbase + k;
      if (wi < w32) {
        const uint32_t word = sw[j][k];
        bits[orow * w32 + wi] = word;
        pc += __popc(word);
      }
    }
    pc = __reduce_add_sync(FULL, pc);
    if (lane == 0 && pc) atomicAdd(&counts[orow], (unsigned long long)pc);
  }
}

__global__ void k_iso_thr(const uint32_t* __restrict__ lane_thr, uint32_t kw, uint32_t lanes,
                          uint32_t* __restrict__ thr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (2 * i >= lanes) return;
  const uint32_t lo = 2 * i < kw ? lane_thr[2 * i] : 0u, hi = 2 * i + 1 < kw ? lane_thr[2 * i + 1] : 0u;
  thr[i] = lo | hi << 16;
}

}  // namespace

// One wave of kw <= 2048 lanes with thresholds of at most tmax < 0xFFFF: slab of
// ceil(kw / 64) tiles, words[n] activity and words[n] reset flags (zeroed here),
// then, 16-byte aligned like words, the packed thresholds. Leaves the labels in the slab; ev (or null) is
// recorded between the upward pass and the sweep.
bf_status iso_wave_panels(Graph* g, const uint32_t* d_orig, const uint32_t* d_thr, uint32_t kw,
                          uint32_t tmax, uint32_t* slab, uint32_t* words, uint64_t* cnt,
                          cudaStream_t st, cudaEvent_t ev, uint64_t* launches) {
  const Panels& P = g->panels;
  const uint32_t n = g->n, tiles = (kw + 63) / 64;
  const bool sat = tmax >= 0x7FFFu;
  bool pdl = false;  // (every level may read the seeds early, as in sweep_panels)
  uint32_t *act = words, *seeded = words + n, *thr = words + ((2 * (size_t)n + 3) & ~(size_t)3);
  BF_CUDA(cudaMemsetAsync(words, 0, 2 * (size_t)n * 4, st));
  k_iso_thr<<<(tiles * 32 + 127) / 128, 128, 0, st>>>(d_thr, kw, tiles * 64, thr);
  k_iso_mark<<<(kw + 3) / 4, 128, 0, st>>>(d_orig, kw, g->d_parent, g->d_run_end, seeded);
  k_iso_reset<<<std::min<uint32_t>((n + 255) / 256, 152 * 16), 256, 0, st>>>(
      seeded, n, slab, sat ? far2<true> : far2<false>);
  BF_CUDA(cudaGetLastError());
  bf_status s;
  if ((s = launch_upward(g, d_orig, kw, INF, nullptr, slab, n, act, st, d_thr, nullptr, nullptr,
                         UPWARD_OUT_TILES16)))
    return s;
  *launches += 4;
  if (ev) BF_CUDA(cudaEventRecord(ev, st));
  IsoArgs a{P.d_a, P.d_b, P.d_src, sat ? P.d_w16s : P.d_w16, n, slab, act, seeded, thr,
            reinterpret_cast<unsigned long long*>(cnt)};
  for (uint32_t l = 0; l < P.n_levels; ++l) {
    const uint32_t p0 = P.lvl_first[l], p1 = P.lvl_first[l + 1], m = p1 - p0;
    // a block per unit where a warp per unit would leave most of the GPU idle
    // behind one warp's walk over up to a few hundred sources
    if (m <= 2 * g->sm_count || (m <= 2048 && m * tiles <= 16384)) {
      BF_CUDA(sat ? launch_level(k_iso_split<true>, dim3(m, tiles), 32 * ISO_WARPS, pdl, st, a, p0)
                  : launch_level(k_iso_split<false>, dim3(m, tiles), 32 * ISO_WARPS, pdl, st, a,
                                 p0));
    } else {
      const uint32_t pb = P.lvl_small[l], big = (pb - p0 + 7) / 8, small = (p1 - pb + 31) / 32;
      // a level of few blocks spreads its tiles over more of them
      const uint32_t y = std::min(tiles, std::max(1u, 16 * g->sm_count / (big + small)));
      BF_CUDA(launch_level(sat ? k_iso_panels<true> : k_iso_panels<false>, dim3(big + small, y),
                           256, pdl, st, a, p0, pb, p1, big));
    }
    pdl = g->tune.pdl != 0;
    ++*launches;
  }
  return BF_OK;
}

// The wave's bitsets (rows out_row[lane] of bits) and counts from its slab.
bf_status iso_bits_panels(Graph* g, const uint32_t* slab, const uint32_t* words,
                          const uint32_t* d_thr, uint32_t kw, uint32_t* bits, uint64_t w32,
                          uint64_t* counts, const uint32_t* out_row, cudaStream_t st) {
  k_iso_bits<<<dim3((g->n + IB_RANKS - 1) / IB_RANKS, (kw + 63) / 64), 256, 0, st>>>(
      slab, g->n, words, d_thr, kw, bits, w32, reinterpret_cast<unsigned long long*>(counts),
      out_row);
  BF_CUDA(cudaGetLastError());
  return BF_OK;
}

}  // namespace bf
