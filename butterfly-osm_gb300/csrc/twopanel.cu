// twopanel.cu — two-channel sweeps and upward passes over panels.
//
// The one-channel forms (panel.cu, upward.cu) with u64 labels, time in the high
// word and length in the low one, ordered as one number: both channels add with
// saturation and a minimum of labels is the lexicographic one (twochannel.cu). A
// panel's length tile lies beside its time tile, INF where there is no edge.

#include <algorithm>

#include "engine.cuh"

namespace bf {

namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr uint64_t LINF = ~0ull;
constexpr uint32_t TP_WARPS = 8, TP_CH = 128;
constexpr uint32_t TP_FLIGHT = 8;  // source rows in flight per thread of a shared panel

__device__ __forceinline__ uint64_t lab_relax(uint64_t a, uint32_t wt, uint32_t wl, uint64_t acc) {
  const uint32_t t = sat_add((uint32_t)(a >> 32), wt), l = sat_add((uint32_t)a, wl);
  return min(acc, (uint64_t)t << 32 | l);
}

// A source's label into all K rows of a panel: its weights 16 bytes a load
// (strides are multiples of four).
template <uint32_t K>
__device__ __forceinline__ void relax_source(uint64_t d, const uint32_t* wt, const uint32_t* wl,
                                             uint64_t (&acc)[K]) {
#pragma unroll
  for (uint32_t j = 0; j < K; j += 4) {
    const uint4 t = *reinterpret_cast<const uint4*>(wt + j);
    const uint4 l = *reinterpret_cast<const uint4*>(wl + j);
    acc[j] = lab_relax(d, t.x, l.x, acc[j]);
    if (j + 1 < K) acc[j + 1] = lab_relax(d, t.y, l.y, acc[j + 1]);
    if (j + 2 < K) acc[j + 2] = lab_relax(d, t.z, l.z, acc[j + 2]);
    if (j + 3 < K) acc[j + 3] = lab_relax(d, t.w, l.w, acc[j + 3]);
  }
}

struct TwoArgs {
  const uint4* item;       // panel items (Sched::d_pitem)
  const uint32_t* prow;    // slab rows of their sources
  const uint32_t *wt, *wl;  // tiles
  uint64_t* slab;
  uint32_t Kp2;
  const uint32_t* seeded;
};

__device__ __forceinline__ uint32_t time_of(uint32_t wt, uint32_t wl) {
  return wl == INF ? INF : wt;  // (absent edges may weigh less in the time tile)
}

// Row j's seed in lane x (LINF where it has none).
__device__ __forceinline__ uint64_t seed_of(const TwoArgs& g, uint4 it, uint32_t j, uint32_t x) {
  const uint32_t r = it.x - j;
  if (j >= (it.y & 31u) || !((g.seeded[r >> 5] >> (r & 31)) & 1u)) return LINF;
  return __ldcg((const unsigned long long*)g.slab + (size_t)r * g.Kp2 + x);
}

// Rows i < j of the panel into row j, then all live rows of one lane.
template <uint32_t K>
__device__ __forceinline__ void finish_rows(const TwoArgs& g, uint4 it, uint32_t x,
                                            const uint32_t* tt, const uint32_t* tl,
                                            uint64_t (&v)[K]) {
  const uint32_t live = it.y & 31u, stride = (it.y >> 5) & 31u;
#pragma unroll
  for (uint32_t i = 0; i + 1 < K; ++i)
#pragma unroll
    for (uint32_t j4 = (i + 1) / 4 * 4; j4 < K; j4 += 4) {
      const uint4 t = *reinterpret_cast<const uint4*>(tt + i * stride + j4);
      const uint4 l = *reinterpret_cast<const uint4*>(tl + i * stride + j4);
      const uint32_t wt[4] = {t.x, t.y, t.z, t.w}, wl[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        if (j4 + q > i && j4 + q < K)
          v[j4 + q] = lab_relax(v[i], time_of(wt[q], wl[q]), wl[q], v[j4 + q]);
    }
#pragma unroll
  for (uint32_t j = 0; j < K; ++j)
    if (j < live) g.slab[(size_t)(it.x - j) * g.Kp2 + x] = v[j];
}

// A block per (panel, 32 lanes): its warps share the sources, whose weights are
// staged while the level before drains, and combine through shared memory.
struct TwoSmem {
  uint32_t wt[TP_CH * PANEL_ROWS], wl[TP_CH * PANEL_ROWS];
  uint32_t tt[PANEL_ROWS * PANEL_ROWS], tl[PANEL_ROWS * PANEL_ROWS];
  uint32_t row[TP_CH];
  uint64_t seed[PANEL_ROWS][32];
};

template <uint32_t K>
__device__ __forceinline__ void block_item(const TwoArgs& g, uint4 it, TwoSmem& sm,
                                           uint64_t (*red)[PANEL_ROWS][32]) {
  constexpr uint32_t TPB = 32 * TP_WARPS;
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t stride = (it.y >> 5) & 31u, nu = it.y >> 10;
  const uint32_t x = blockIdx.y * 32 + lane;
  const bool on = x < g.Kp2;
  auto stage = [&](uint32_t c0, uint32_t m) {
    for (uint32_t i = t; i < m; i += TPB) sm.row[i] = g.prow[it.w + c0 + i];
    for (uint32_t i = t; i < m * stride; i += TPB) {
      const size_t at = it.z + (size_t)c0 * stride + i;
      const uint32_t wl = g.wl[at];
      sm.wl[i] = wl;
      sm.wt[i] = time_of(g.wt[at], wl);
    }
  };
  stage(0, min(nu, TP_CH));
  for (uint32_t i = t; i < stride * stride; i += TPB) {
    sm.tl[i] = g.wl[it.z + (size_t)nu * stride + i];
    sm.tt[i] = g.wt[it.z + (size_t)nu * stride + i];
  }
  // (seeds are written before the first level is launched)
  for (uint32_t j = warp; j < K; j += TP_WARPS) sm.seed[j][lane] = on ? seed_of(g, it, j, x) : LINF;
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint64_t acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = LINF;
  for (uint32_t c0 = 0; c0 < nu; c0 += TP_CH) {
    const uint32_t m = min(nu - c0, TP_CH);
    if (c0) {
      __syncthreads();
      stage(c0, m);
      __syncthreads();
    }
    if (on)
      for (uint32_t s0 = warp; s0 < m; s0 += TP_FLIGHT * TP_WARPS) {
        const unsigned long long* slab = (const unsigned long long*)g.slab + x;
        uint64_t d[TP_FLIGHT];
#pragma unroll
        for (uint32_t q = 0; q < TP_FLIGHT; ++q) {
          const uint32_t s = s0 + q * TP_WARPS;
          d[q] = s < m ? __ldcg(slab + (size_t)sm.row[s] * g.Kp2) : LINF;
        }
#pragma unroll
        for (uint32_t q = 0; q < TP_FLIGHT; ++q) {
          const uint32_t s = s0 + q * TP_WARPS;
          if (s >= m) break;
          relax_source<K>(d[q], sm.wt + s * stride, sm.wl + s * stride, acc);
        }
      }
  }
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) red[warp][j][lane] = acc[j];
  __syncthreads();
  for (uint32_t j = warp; j < K; j += TP_WARPS) {
    uint64_t v = sm.seed[j][lane];
#pragma unroll
    for (uint32_t q = 0; q < TP_WARPS; ++q) v = min(v, red[q][j][lane]);
    red[0][j][lane] = v;
  }
  __syncthreads();
  if (warp || !on) return;
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = red[0][j][lane];
  finish_rows<K>(g, it, x, sm.tt, sm.tl, acc);
}

// Bound by the chain of levels, and with u64 labels by a level's arithmetic (ten
// instructions a weight). 60 x 90 ends of one to three seeds on the 1000 x 1250
// region, whole call: 4.85 ms with a launch per level of rows, 0.94 ms by panels
// (1.08 with two rows in flight and the seeds read at the end, 0.96 with a load
// per weight instead of one per four).
__global__ void __launch_bounds__(32 * TP_WARPS) k_two_split(const TwoArgs g, uint32_t i0) {
  extern __shared__ __align__(16) unsigned char two_smem[];
  TwoSmem& sm = *reinterpret_cast<TwoSmem*>(two_smem);
  uint64_t(*red)[PANEL_ROWS][32] =
      reinterpret_cast<uint64_t(*)[PANEL_ROWS][32]>(two_smem + sizeof(TwoSmem));
  asm volatile("griddepcontrol.launch_dependents;");
  const uint4 it = g.item[i0 + blockIdx.x];
  const uint32_t live = it.y & 31u;
  if (live > 8) block_item<16>(g, it, sm, red);
  else if (live > 4) block_item<8>(g, it, sm, red);
  else if (live > 2) block_item<4>(g, it, sm, red);
  else block_item<2>(g, it, sm, red);
}
constexpr size_t TWO_SMEM = sizeof(TwoSmem) + (size_t)TP_WARPS * PANEL_ROWS * 32 * 8;

// Levels with more units than the GPU holds blocks: a warp per (panel, 32
// lanes), weights from global memory.
template <uint32_t K>
__device__ __forceinline__ void warp_item(const TwoArgs& g, uint4 it, uint32_t x) {
  const uint32_t stride = (it.y >> 5) & 31u, nu = it.y >> 10;
  const uint32_t *wt = g.wt + it.z, *wl = g.wl + it.z;
  uint64_t acc[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = LINF;
  const unsigned long long* slab = (const unsigned long long*)g.slab + x;
#pragma unroll 2
  for (uint32_t s = 0; s < nu; ++s) {
    const uint64_t d = __ldcg(slab + (size_t)g.prow[it.w + s] * g.Kp2);
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) {
      const uint32_t l = wl[(size_t)s * stride + j];
      acc[j] = lab_relax(d, time_of(wt[(size_t)s * stride + j], l), l, acc[j]);
    }
  }
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) acc[j] = min(acc[j], seed_of(g, it, j, x));
  finish_rows<K>(g, it, x, wt + (size_t)nu * stride, wl + (size_t)nu * stride, acc);
}

__global__ void __launch_bounds__(256) k_two_warps(const TwoArgs g, uint32_t i0, uint32_t m,
                                                   uint32_t tiles) {
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const bool in = u < m * tiles;
  const uint4 it = in ? g.item[i0 + u / tiles] : make_uint4(0, 0, 0, 0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t x = (u % tiles) * 32 + (threadIdx.x & 31);
  if (!in || x >= g.Kp2) return;
  const uint32_t live = it.y & 31u;
  if (live > 8) warp_item<16>(g, it, x);
  else if (live > 4) warp_item<8>(g, it, x);
  else if (live > 2) warp_item<4>(g, it, x);
  else warp_item<2>(g, it, x);
}

// ---- upward -------------------------------------------------------------------

template <uint32_t K>
__device__ __forceinline__ uint64_t panel_up2(uint64_t d, uint32_t jm, uint32_t threshold,
                                              const uint32_t* __restrict__ wt,
                                              const uint32_t* __restrict__ wl,
                                              const uint32_t* __restrict__ ends, uint32_t nt,
                                              volatile uint64_t* pd, uint32_t last, uint32_t lane,
                                              volatile uint64_t* srow) {
  auto pushes = [&](uint64_t lab) {
    const uint32_t t = (uint32_t)(lab >> 32);
    return t != INF && t <= threshold;
  };
  const uint32_t *tt = wt + (size_t)nt * K, *tl = wl + (size_t)nt * K;
  uint32_t at[K], al[K];  // this lane's column of the triangle
#pragma unroll
  for (uint32_t j = 1; j < K; ++j) {
    at[j] = lane < j ? __ldg(tt + j * K + lane) : INF;
    al[j] = lane < j ? __ldg(tl + j * K + lane) : INF;
  }
#pragma unroll
  for (uint32_t j = K - 1; j > 0; --j)
    if (j <= jm) {
      const uint64_t dj = __shfl_sync(FULL, d, j);
      if (pushes(dj)) d = lab_relax(dj, at[j], al[j], d);
    }
  if (lane < K) srow[lane] = pushes(d) ? d : LINF;
  __syncwarp();
  uint64_t dj[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) dj[j] = srow[j];
  for (uint32_t q = lane; q < nt; q += 32) {
    uint64_t v = LINF;
#pragma unroll
    for (uint32_t j = 0; j < K; j += 4) {
      const uint4 a = __ldg(reinterpret_cast<const uint4*>(wt + (size_t)q * K + j));
      const uint4 b = __ldg(reinterpret_cast<const uint4*>(wl + (size_t)q * K + j));
      v = lab_relax(dj[j], a.x, b.x, v);
      v = lab_relax(dj[j + 1], a.y, b.y, v);
      v = lab_relax(dj[j + 2], a.z, b.z, v);
      v = lab_relax(dj[j + 3], a.w, b.w, v);
    }
    const uint32_t t = last - __ldg(ends + q);
    if (v < pd[t]) pd[t] = v;
  }
  __syncwarp();
  return d;
}

// k_upward_panels with u64 labels; unit w starts at (u_cost, u_len) and writes
// (min) every label within the threshold into lane u_lane[w].
__global__ void __launch_bounds__(UPWARD_WARPS * 32)
    k_upward_two(uint32_t k, const uint32_t* __restrict__ u_rank,
                 const uint32_t* __restrict__ u_cost, const uint32_t* __restrict__ u_len,
                 const uint32_t* __restrict__ u_lane, uint32_t threshold, uint32_t n,
                 const uint32_t* __restrict__ of, const uint4* __restrict__ up,
                 const uint32_t* __restrict__ up_end, const uint32_t* __restrict__ up_w,
                 const uint32_t* __restrict__ up_l, const uint32_t* __restrict__ cidx,
                 uint64_t* __restrict__ slab, uint32_t stride, uint32_t* __restrict__ flag,
                 uint32_t dcap, uint32_t* __restrict__ err) {
  extern __shared__ __align__(16) uint64_t smem[];
  const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t w = blockIdx.x * UPWARD_WARPS + wib;
  if (w >= k) return;
  const uint32_t s = u_rank[w];
  if (s >= n) {
    if (lane == 0) atomicOr(err, DEVERR_PATH);
    return;
  }
  uint64_t* pd = smem + (size_t)wib * (dcap + PANEL_ROWS);
  uint64_t* srow = pd + dcap;
  const uint32_t p0 = of[s];
  uint4 a = up[2 * (size_t)p0], b = up[2 * (size_t)p0 + 1];
  uint32_t jm = b.x - s;
  const uint32_t D = a.x + jm + 1;
  if (D > dcap || jm >= PANEL_ROWS) {
    if (lane == 0) atomicOr(err, DEVERR_PATH);
    return;
  }
  const uint64_t seed = (uint64_t)u_cost[w] << 32 | u_len[w];
  const uint32_t out_lane = u_lane[w];
  for (uint32_t l = lane; l < D; l += 32) pd[l] = l == 0 ? seed : LINF;
  __syncwarp();
  for (;;) {
    const bool more = a.w != NONE;
    uint4 na = a, nb = b;
    if (more) {
      na = up[2 * (size_t)a.w];
      nb = up[2 * (size_t)a.w + 1];
    }
    const uint32_t idx = D - 1 - a.x;
    if (a.x > D - 1 || jm > idx || jm >= PANEL_ROWS) {
      if (lane == 0) atomicOr(err, DEVERR_PATH);
      return;
    }
    uint64_t d = lane <= jm ? pd[idx - lane] : LINF;
    const uint32_t ks = (a.y >> 8) & 0xFF;
    const uint32_t *wt = up_w + b.z, *wl = up_l + b.z, *ends = up_end + b.y;
    if (ks == 4) d = panel_up2<4>(d, jm, threshold, wt, wl, ends, a.z, pd, D - 1, lane, srow);
    else if (ks == 8) d = panel_up2<8>(d, jm, threshold, wt, wl, ends, a.z, pd, D - 1, lane, srow);
    else if (ks == 12) d = panel_up2<12>(d, jm, threshold, wt, wl, ends, a.z, pd, D - 1, lane, srow);
    else d = panel_up2<16>(d, jm, threshold, wt, wl, ends, a.z, pd, D - 1, lane, srow);
    const uint32_t t = (uint32_t)(d >> 32);
    if (lane <= jm && t != INF && t <= threshold) {
      const uint32_t row = cidx[b.x - lane];
      if (row != NONE) {
        atomicMin((unsigned long long*)&slab[(size_t)row * stride + out_lane],
                  (unsigned long long)d);
        if (flag) atomicOr(&flag[row >> 5], 1u << (row & 31));
      }
    }
    if (!more) break;
    jm = b.w;
    a = na;
    b = nb;
  }
}

size_t upward_two_smem(const Graph* g) {
  const uint32_t dcap = ((g->max_depth + 1) + 31) & ~31u;
  return (size_t)UPWARD_WARPS * (dcap + PANEL_ROWS) * 8;
}

}  // namespace

cudaError_t sweep_panels_2ch(Graph* g, Sched& sc, uint64_t* slab, uint32_t Kp2, cudaStream_t st,
                             uint64_t* launches, const uint32_t* seeded) {
  const Panels& P = g->panels;
  bool pdl = false;  // (every level may read the seeds early, as in sweep_panels)
  const TwoArgs a{sc.d_pitem, sc.d_prow, P.d_w, P.d_len, slab, Kp2, seeded};
  const uint32_t tiles = (Kp2 + 31) / 32;
  for (uint32_t l = 0; l + 1 < sc.lvl_pan.size(); ++l) {
    const uint32_t i0 = sc.lvl_pan[l], m = sc.lvl_pan[l + 1] - i0;
    if (!m) continue;
    // a block per unit while a level's units are few: a warp of the other form
    // walks all sources of its panel alone
    const uint64_t units = (uint64_t)m * tiles;
    const cudaError_t e =
        units <= 8ull * g->sm_count || units >= 0x80000000ull
            ? launch_level_smem(k_two_split, dim3(m, tiles), 32 * TP_WARPS, TWO_SMEM, pdl, st, a,
                                i0)
            : launch_level(k_two_warps, dim3((unsigned)((units + 7) / 8)), 256, pdl, st, a, i0, m,
                           tiles);
    if (e != cudaSuccess) return e;
    pdl = g->tune.pdl != 0;
    ++*launches;
  }
  return cudaSuccess;
}

bool upward_2ch_by_panels(const Graph* g) {
  return g->panels.n && g->panels.d_up_len && upward_two_smem(g) <= 200 * 1024;
}

bf_status upward_2ch_kernel_init() {
  BF_CUDA(cudaFuncSetAttribute(k_upward_two, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               200 * 1024));
  BF_CUDA(cudaFuncSetAttribute(k_two_split, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)TWO_SMEM));
  return BF_OK;
}

bf_status launch_upward_2ch_panels(Graph* g, const uint32_t* d_units, uint64_t nu,
                                   uint32_t threshold, const uint32_t* cidx, uint64_t* slab,
                                   uint32_t stride, uint32_t* flag, cudaStream_t st) {
  const Panels& P = g->panels;
  k_upward_two<<<(unsigned)((nu + UPWARD_WARPS - 1) / UPWARD_WARPS), UPWARD_WARPS * 32,
                 upward_two_smem(g), st>>>((uint32_t)nu, d_units, d_units + nu, d_units + 2 * nu,
                                           d_units + 3 * nu, threshold, g->n, P.d_of, P.d_up,
                                           P.d_up_end, P.d_up_w, P.d_up_len, cidx, slab, stride,
                                           flag, ((g->max_depth + 1) + 31) & ~31u, g->d_err);
  BF_CUDA(cudaGetLastError());
  return BF_OK;
}

}  // namespace bf
