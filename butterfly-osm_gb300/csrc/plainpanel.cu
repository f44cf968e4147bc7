// plainpanel.cu — the plain engine's sweep over panels: every node of the graph,
// K = 32 sources, in one cooperative launch.
//
// Slab rows are ranks (row j of a panel is rank hi - j), a lane a source. The
// blocks walk the levels of the panel DAG with a grid barrier between them; each
// row is written once, by its panel, so the slab needs no initial values: seeds
// lie in a second slab, with a bit per seeded row.

#include <algorithm>

#include "engine.cuh"

namespace bf {

namespace {

constexpr uint32_t PP_WARPS = 8;
constexpr uint32_t PP_CH = 16;  // sources of a chunk: their rows are in flight together

struct PlainArgs {
  const uint4* a;       // Panels::d_a, d_b, d_lvl
  const uint2* b;
  const uint32_t *lvl, *lvl_small;
  uint32_t n_levels;
  const uint32_t *src, *w;
  uint32_t absent;
  uint32_t *dist, *seed, *flag;
  uint32_t threshold;
};

struct PlainSmem {
  uint32_t w[PP_WARPS][PP_CH * PANEL_ROWS];         // a chunk's tile per warp
  uint32_t tri[PP_WARPS][PANEL_ROWS * PANEL_ROWS];  // a panel's triangle per warp
  uint32_t red[PP_WARPS][PANEL_ROWS][32];           // minima of a shared panel's warps
  uint32_t seed[PANEL_ROWS][32];                    // and its seeds
};

__device__ __forceinline__ uint32_t min_plus(uint32_t d, uint32_t w, uint32_t acc) {
  return __viaddmin_u32(min(d, ~w), w, acc);  // min(acc, d + w), the sum saturating at INF
}

__device__ __forceinline__ uint32_t stride_of(const uint4& a) { return (a.y >> 8) & 0xFF; }

// Sources per warp of a chunk.
template <bool SHARED>
__device__ __forceinline__ uint32_t chunk_of(uint32_t nu) {
  return SHARED ? min(PP_CH, (nu + PP_WARPS - 1) / PP_WARPS) : PP_CH;
}

// A chunk's source ids (a lane each) and tile, into registers.
template <uint32_t K>
__device__ __forceinline__ void load_chunk(const PlainArgs& g, const uint2 b, uint32_t c0,
                                           uint32_t m, uint32_t lane, uint32_t* id,
                                           uint32_t (&wv)[K / 2]) {
  *id = lane < m ? __ldg(g.src + b.x + c0 + lane) : 0u;
  const uint32_t* tile = g.w + b.y + (size_t)c0 * K;
#pragma unroll
  for (uint32_t i = 0; i < K / 2; ++i)
    wv[i] = i * 32 + lane < m * K ? __ldg(tile + i * 32 + lane) : INF;
}

template <uint32_t K>
__device__ __forceinline__ void store_chunk(const PlainArgs& g, uint32_t* ws, uint32_t lane,
                                            const uint32_t (&wv)[K / 2]) {
#pragma unroll
  for (uint32_t i = 0; i < K / 2; ++i) ws[i * 32 + lane] = wv[i] == g.absent ? INF : wv[i];
}

template <uint32_t K>
__device__ __forceinline__ void load_triangle(const PlainArgs& g, const uint4 a, const uint2 b,
                                              uint32_t lane, uint32_t* tri) {
  const uint32_t* t = g.w + b.y + (size_t)a.z * K;
#pragma unroll
  for (uint32_t i = 0; i < K * K; i += 32)
    if (i + lane < K * K) {
      const uint32_t v = __ldg(t + i + lane);
      tri[i + lane] = v == g.absent ? INF : v;
    }
}

// Row r's seeds, read and given back (its bit f is set).
__device__ __forceinline__ uint32_t take_seed(const PlainArgs& g, uint32_t r, uint32_t lane) {
  uint32_t* at = g.seed + (size_t)r * PLAIN_K + lane;
  const uint32_t v = *at;
  *at = INF;
  __syncwarp();
  if (lane == 0) atomicAnd(g.flag + (r >> 5), ~(1u << (r & 31)));
  return v;
}

// The minimum over the four groups of eight lanes.
__device__ __forceinline__ uint32_t across(uint32_t v) {
  v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 8));
  return min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 16));
}

// What a shared panel needs that no earlier level writes: each warp's first
// chunk, the triangle and the seeds. Returns the warp's source ids.
template <uint32_t K>
__device__ __forceinline__ uint32_t stage_shared(const PlainArgs& g, const uint4 a, const uint2 b,
                                                 PlainSmem& sm) {
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t ch = chunk_of<true>(a.z), c0 = wib * ch;
  uint32_t id = 0, wv[K / 2];
  if (c0 < a.z) load_chunk<K>(g, b, c0, min(ch, a.z - c0), lane, &id, wv);
  if (wib == PP_WARPS - 1) load_triangle<K>(g, a, b, lane, sm.tri[0]);
  for (uint32_t j = wib; j < (a.y & 0xFF); j += PP_WARPS) {
    const uint32_t r = a.x - j;
    sm.seed[j][lane] =
        (__ldcg(g.flag + (r >> 5)) >> (r & 31)) & 1u ? take_seed(g, r, lane) : INF;
  }
  if (c0 < a.z) store_chunk<K>(g, sm.w[wib], lane, wv);
  return id;
}

// A panel (stride K) by one warp, or with SHARED by all warps of the block, a
// chunk of the sources each, staged before (id: its first chunk's ids). NARROW
// (at most 8 lanes hold sources): four of the panel's sources side by side, eight
// lanes each, their minima combined at the end.
template <uint32_t K, bool SHARED, bool NARROW>
__device__ __forceinline__ void plain_panel(const PlainArgs& g, const uint4 a, const uint2 b,
                                            uint32_t id, PlainSmem& sm) {
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  constexpr uint32_t SIDE = NARROW ? 4 : 1;  // sources side by side
  const uint32_t at = NARROW ? lane & 7 : lane, side = NARROW ? lane >> 3 : 0;
  const uint32_t rows = a.y & 0xFF, nu = a.z;
  uint32_t* ws = sm.w[wib];
  uint32_t* tri = sm.tri[SHARED ? 0 : wib];
  const uint32_t ch = chunk_of<SHARED>(nu), step = SHARED ? PP_WARPS * ch : ch;
  uint32_t c0 = SHARED ? wib * ch : 0;
  uint32_t wv[K / 2];
  if (!SHARED) {
    if (nu) load_chunk<K>(g, b, 0, min(ch, nu), lane, &id, wv);
    load_triangle<K>(g, a, b, lane, tri);
    if (nu) store_chunk<K>(g, ws, lane, wv);
  }
  __syncwarp();
  uint32_t acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = INF;
  while (c0 < nu) {
    const uint32_t m = min(ch, nu - c0), next = c0 + step;
    uint32_t d[PP_CH / SIDE];
#pragma unroll
    for (uint32_t q = 0; q < PP_CH / SIDE; ++q) {
      const uint32_t s = q * SIDE + side, r = __shfl_sync(0xFFFFFFFFu, id, s);
      d[q] = s < m ? __ldcg(g.dist + (size_t)r * PLAIN_K + at) : INF;
    }
    if (next < nu) load_chunk<K>(g, b, next, min(ch, nu - next), lane, &id, wv);
#pragma unroll
    for (uint32_t q = 0; q < PP_CH / SIDE; ++q) {
      if (q * SIDE >= m) break;
#pragma unroll
      for (uint32_t j = 0; j < K; j += 4) {
        const uint4 x = *reinterpret_cast<const uint4*>(ws + (q * SIDE + side) * K + j);
        acc[j] = min_plus(d[q], x.x, acc[j]);
        acc[j + 1] = min_plus(d[q], x.y, acc[j + 1]);
        acc[j + 2] = min_plus(d[q], x.z, acc[j + 2]);
        acc[j + 3] = min_plus(d[q], x.w, acc[j + 3]);
      }
    }
    __syncwarp();
    if (next < nu) store_chunk<K>(g, ws, lane, wv);
    __syncwarp();
    c0 = next;
  }
  if (SHARED) {
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) sm.red[wib][j][lane] = acc[j];
    __syncthreads();
    for (uint32_t j = wib; j < rows; j += PP_WARPS) {
      uint32_t v = sm.seed[j][lane];
#pragma unroll
      for (uint32_t q = 0; q < PP_WARPS; ++q) v = min(v, sm.red[q][j][lane]);
      if (NARROW) v = across(v);
      sm.red[0][j][lane] = v;
    }
    __syncthreads();
  }
  if (!SHARED || wib == 0) {
    if (SHARED) {
#pragma unroll
      for (uint32_t j = 0; j < K; ++j) acc[j] = sm.red[0][j][lane];
    } else {
      if (NARROW)
#pragma unroll
        for (uint32_t j = 0; j < K; ++j) acc[j] = across(acc[j]);
      const uint32_t w0 = (a.x + 1 - rows) >> 5, w1 = a.x >> 5;
      const uint32_t f0 = __ldcg(g.flag + w0), f1 = w1 == w0 ? f0 : __ldcg(g.flag + w1);
#pragma unroll
      for (uint32_t j = 0; j < K; ++j) {
        const uint32_t r = a.x - j;
        if (j < rows && (((r >> 5) == w0 ? f0 : f1) >> (r & 31)) & 1u)
          acc[j] = min(acc[j], take_seed(g, r, lane));
      }
    }
#pragma unroll
    for (uint32_t i = 0; i + 1 < K; ++i)
#pragma unroll
      for (uint32_t v = (i + 1) / 4; v < K / 4; ++v) {
        const uint4 x = *reinterpret_cast<const uint4*>(tri + i * K + 4 * v);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          if (4 * v + q > i) acc[4 * v + q] = min_plus(acc[i], w[q], acc[4 * v + q]);
      }
#pragma unroll
    for (uint32_t j = 0; j < K; ++j)
      if (j < rows && side == 0)
        g.dist[(size_t)(a.x - j) * PLAIN_K + at] = acc[j] > g.threshold ? INF : acc[j];
    __syncwarp();  // (the warp's next panel writes the shared tile and triangle)
  }
  if (SHARED) __syncthreads();
}

// A panel of up to four rows by G threads, four lanes each (eight, or two where
// at most 8 lanes hold sources; mg: their bits of the warp): several panels of a
// warp at a time, and rows, weights and seeds move 16 bytes a load.
__device__ __forceinline__ uint4 min_plus4(const uint4 d, uint32_t w, const uint4 acc) {
  return make_uint4(min_plus(d.x, w, acc.x), min_plus(d.y, w, acc.y), min_plus(d.z, w, acc.z),
                    min_plus(d.w, w, acc.w));
}

template <uint32_t G>
__device__ __forceinline__ void plain_small(const PlainArgs& g, uint32_t p) {
  const unsigned mg = ((1u << G) - 1) << (threadIdx.x & 31 & ~(G - 1));
  constexpr uint32_t K = 4, U = 4;  // source rows in flight
  const uint4 a = g.a[p];
  const uint2 b = g.b[p];
  const uint32_t rows = a.y & 0xFF, nu = a.z, l4 = (threadIdx.x & (G - 1)) * 4;
  const uint32_t* tile = g.w + b.y;
  const uint32_t w0 = (a.x + 1 - rows) >> 5, w1 = a.x >> 5;
  const uint32_t f0 = __ldcg(g.flag + w0), f1 = w1 == w0 ? f0 : __ldcg(g.flag + w1);
  __syncwarp(mg);  // (all have read the bits before one clears them)
  uint4 acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) {
    const uint32_t r = a.x - j;
    acc[j] = make_uint4(INF, INF, INF, INF);
    if (j < rows && (((r >> 5) == w0 ? f0 : f1) >> (r & 31)) & 1u) {
      uint4* at = reinterpret_cast<uint4*>(g.seed + (size_t)r * PLAIN_K + l4);
      acc[j] = *at;
      *at = make_uint4(INF, INF, INF, INF);
      if (l4 == 0) atomicAnd(g.flag + (r >> 5), ~(1u << (r & 31)));
    }
  }
  auto weights = [&](uint32_t at) {
    uint4 w = __ldg(reinterpret_cast<const uint4*>(tile + (size_t)at * K));
    w.x = w.x == g.absent ? INF : w.x;
    w.y = w.y == g.absent ? INF : w.y;
    w.z = w.z == g.absent ? INF : w.z;
    w.w = w.w == g.absent ? INF : w.w;
    return w;
  };
  for (uint32_t s = 0; s < nu; s += U) {
    uint4 d[U];
#pragma unroll
    for (uint32_t q = 0; q < U; ++q)
      if (s + q < nu)
        d[q] = __ldcg(reinterpret_cast<const uint4*>(
            g.dist + (size_t)__ldg(g.src + b.x + s + q) * PLAIN_K + l4));
#pragma unroll
    for (uint32_t q = 0; q < U; ++q) {
      if (s + q >= nu) break;
      const uint4 w = weights(s + q);
      acc[0] = min_plus4(d[q], w.x, acc[0]);
      acc[1] = min_plus4(d[q], w.y, acc[1]);
      acc[2] = min_plus4(d[q], w.z, acc[2]);
      acc[3] = min_plus4(d[q], w.w, acc[3]);
    }
  }
#pragma unroll
  for (uint32_t i = 0; i + 1 < K; ++i) {
    const uint4 w = weights(nu + i);
    if (i < 1) acc[1] = min_plus4(acc[i], w.y, acc[1]);
    if (i < 2) acc[2] = min_plus4(acc[i], w.z, acc[2]);
    acc[3] = min_plus4(acc[i], w.w, acc[3]);
  }
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) {
    if (j >= rows) break;
    uint4 v = acc[j];
    v.x = v.x > g.threshold ? INF : v.x;
    v.y = v.y > g.threshold ? INF : v.y;
    v.z = v.z > g.threshold ? INF : v.z;
    v.w = v.w > g.threshold ? INF : v.w;
    *reinterpret_cast<uint4*>(g.dist + (size_t)(a.x - j) * PLAIN_K + l4) = v;
  }
}

#define BF_BY_STRIDE(a, CALL)      \
  switch (stride_of(a)) {          \
    case 4: CALL(4); break;        \
    case 8: CALL(8); break;        \
    case 12: CALL(12); break;      \
    default: CALL(16);             \
  }

// Bound by the chain of levels: a grid barrier and the dependent reads of
// each. A level with few panels has a block share each one, what no earlier
// level writes staged between its arrival at the barrier and its wait; else
// every warp takes panels of its own: once a block's turn comes round more than
// four times, its warps do better apart (twice or once: within 3 %). `withhold`
// (a test hook, NONE otherwise) names a block that leaves before its first
// barrier arrival.
//
// 29 sources to all of the town's 119,249 nodes: sweep 615 -> 220 us, whole call
// 849 -> 335 (348 with the staging before the arrival). A batch's sweep on the
// 1000 x 1250 region 2.99 -> 1.36 ms, on the country graph 6.73 -> 4.58 (9.1 with
// a warp for panels of up to four rows too). NARROW, eight sources: 0.93 and 2.73
// ms there; one source on grid100, whole call: 546 -> 452 us (2250 by rows). On
// the region the schedulers issue in a fifth of the cycles: the warps wait at the
// barriers and for rows.
template <int PER_SM, bool NARROW>
__global__ void __launch_bounds__(32 * PP_WARPS, PER_SM)
    k_plain_panels(const PlainArgs g, uint32_t* __restrict__ bar, long long timeout,
                   uint32_t withhold, uint32_t* __restrict__ err) {
  __shared__ __align__(16) PlainSmem sm;
  if (blockIdx.x == withhold) return;
  const uint32_t share = 4 * gridDim.x;
  uint4 a = make_uint4(0, 0, 0, 0);
  uint2 b = make_uint2(0, 0);
  uint32_t id = 0;
  auto stage = [&](uint32_t p) {
    a = g.a[p];
    b = g.b[p];
#define BF_STAGE(K) id = stage_shared<K>(g, a, b, sm)
    BF_BY_STRIDE(a, BF_STAGE)
#undef BF_STAGE
  };
  uint32_t p0 = g.lvl[0], p1 = g.lvl[1];
  bool staged = false;
  for (uint32_t l = 0; l < g.n_levels; ++l) {
    const uint32_t p2 = l + 1 < g.n_levels ? g.lvl[l + 2] : p1;
    if (p1 - p0 <= share) {
      for (uint32_t p = p0 + blockIdx.x; p < p1; p += gridDim.x) {
        if (!staged) stage(p);
        staged = false;
#define BF_SOLVE(K) plain_panel<K, true, NARROW>(g, a, b, id, sm)
        BF_BY_STRIDE(a, BF_SOLVE)
#undef BF_SOLVE
      }
    } else {
      const uint32_t ps = g.lvl_small[l];  // panels of up to four rows, last in a level
      for (uint32_t p = p0 + blockIdx.x * PP_WARPS + (threadIdx.x >> 5); p < ps;
           p += gridDim.x * PP_WARPS) {
        const uint4 wa = g.a[p];
        const uint2 wb = g.b[p];
#define BF_SOLVE(K) plain_panel<K, false, NARROW>(g, wa, wb, 0, sm)
        BF_BY_STRIDE(wa, BF_SOLVE)
#undef BF_SOLVE
      }
      constexpr uint32_t G = NARROW ? 2 : 8;
      for (uint32_t p = ps + (blockIdx.x * PP_WARPS * 32 + threadIdx.x) / G; p < p1;
           p += gridDim.x * PP_WARPS * 32 / G)
        plain_small<G>(g, p);
      __syncthreads();
    }
    if (l + 1 == g.n_levels) break;
    grid_arrive(bar);
    if (p2 - p1 <= share && p1 + blockIdx.x < p2) {
      stage(p1 + blockIdx.x);
      staged = true;
    }
    if (!grid_wait(bar, l, timeout, err)) return;
    p0 = p1;
    p1 = p2;
  }
}
#undef BF_BY_STRIDE

}  // namespace

bf_status plain_sweep_panels(Graph* g, uint32_t k, uint32_t threshold, cudaStream_t st,
                             uint64_t* launches) {
  bf_status s;
  if ((s = ensure_barrier(g))) return s;
  const Panels& P = g->panels;
  const PlainArgs a{P.d_a,    P.d_b,     P.d_lvl,   P.d_lvl_small, P.n_levels, P.d_src, P.d_w,
                    P.absent, g->d_dist, g->d_seed, g->d_flag,  threshold};
  const bool hook = test_withhold_arrival();
  // a slab beyond L2: rows come from HBM, and more blocks hide that although
  // their kernel spills more (630 bytes a thread against 160; country graph 4.7 ms
  // a batch against 5.45 with two an SM, the town 400 us a call against 361)
  const bool wide = (uint64_t)g->n * PLAIN_K * 4 > g->l2_bytes;
  const bool narrow = k <= 8;
  const auto kern = wide ? narrow ? k_plain_panels<4, true> : k_plain_panels<4, false>
                         : narrow ? k_plain_panels<2, true> : k_plain_panels<2, false>;
  const unsigned blocks = persistent_blocks(g, (const void*)kern, 32 * PP_WARPS,
                                            (wide ? 4 : 2) * g->sm_count);
  BF_CUDA(cudaMemsetAsync(g->d_bar, 0, 8, st));
  BF_CUDA(launch_persistent(kern, blocks, 32 * PP_WARPS, st, a, g->d_bar,
                            hook ? 2000000ll : BARRIER_TIMEOUT_CYCLES, hook ? 1u : NONE,
                            g->d_err));
  ++*launches;
  return BF_OK;
}

}  // namespace bf
