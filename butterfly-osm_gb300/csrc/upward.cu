// upward.cu — the upward pass over panels.
//
// One warp per source (or seed unit) walks the panels of its root path. In a
// panel, lane j holds the label of row j (j ranks below the panel's highest);
// the path meets the panel in rows jm .. 0, lowest rank first. The rows relax
// each other through the panel's triangle, one shuffle a row, and are final;
// then 32 targets a step, lane q takes the minimum over the rows for its
// target (a row of the dense tile) and lowers the target's path label: targets
// are distinct, so a plain read and write do. Against a walk of single ranks
// (an atomic minimum per UP edge), a panel costs one chain of loads instead of
// sixteen, and a target's label is touched once per panel instead of once per
// edge. Path labels lie in shared memory by path index; a rank's index is its
// depth below the source's, so neither ranks nor runs are kept. Few sources are
// bound by the chain of panels, many by the L2 reads of the tiles (64 bytes a
// target and panel). Against the walk of single ranks: the wait for the pass of
// 37 sources on the 1000 x 1250 region 0.16 -> 0.03 ms (it runs beside the
// schedule's build), 10 000 sources on the country graph 2.07 -> 1.46 ms (the
// kernel alone, cold).

#include "engine.cuh"

namespace bf {

namespace {

// Minimum over rows of d[j] + w[j] (saturating), for one target.
template <uint32_t K>
__device__ __forceinline__ uint32_t target_min(const uint32_t (&d)[K], const uint32_t* w) {
  uint32_t v = INF;
#pragma unroll
  for (uint32_t j = 0; j < K; j += 4) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(w + j));
    v = __viaddmin_u32(min(d[j], ~x.x), x.x, v);
    v = __viaddmin_u32(min(d[j + 1], ~x.y), x.y, v);
    v = __viaddmin_u32(min(d[j + 2], ~x.z), x.z, v);
    v = __viaddmin_u32(min(d[j + 3], ~x.w), x.w, v);
  }
  return v;
}

// Rows jm .. 0 of one panel: solve the triangle, push to the targets. d: this
// lane's row's label (INF past jm); returns it final. pd: path labels; a target
// of depth x has index last - x.
template <uint32_t K>
__device__ __forceinline__ uint32_t panel_up(uint32_t d, uint32_t jm, uint32_t thr1,
                                             const uint32_t* __restrict__ w,
                                             const uint32_t* __restrict__ ends, uint32_t nt,
                                             volatile uint32_t* pd, uint32_t last, uint32_t lane,
                                             volatile uint32_t* srow) {
  constexpr unsigned FULL = 0xFFFFFFFFu;
  uint32_t tri[K];  // this lane's column of the triangle
  const uint32_t* tr = w + (size_t)nt * K;
#pragma unroll
  for (uint32_t j = 1; j < K; ++j) tri[j] = lane < j ? __ldg(tr + j * K + lane) : INF;
#pragma unroll
  for (uint32_t j = K - 1; j > 0; --j)
    if (j <= jm) {
      const uint32_t dj = __shfl_sync(FULL, d, j);
      if (dj <= thr1) d = min(d, sat_add(dj, tri[j]));
    }
  // labels above the threshold push nothing
  if (lane < K) srow[lane] = d <= thr1 ? d : INF;
  __syncwarp();
  uint32_t dj[K];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) dj[j] = srow[j];
#pragma unroll 2
  for (uint32_t q = lane; q < nt; q += 32) {
    const uint32_t v = target_min<K>(dj, w + (size_t)q * K);
    const uint32_t t = last - __ldg(ends + q);
    if (v < pd[t]) pd[t] = v;
  }
  __syncwarp();
  return d;
}

// Dynamic shared memory: UPWARD_WARPS x (dcap path labels + 16 words).
__global__ void __launch_bounds__(UPWARD_WARPS * 32, 6)
    k_upward_panels(const uint32_t* __restrict__ src, uint32_t k, uint32_t threshold, uint32_t n,
                    const uint32_t* __restrict__ of, const uint4* __restrict__ up,
                    const uint32_t* __restrict__ up_end, const uint32_t* __restrict__ up_w,
                    const uint32_t* __restrict__ pos_of,
                    uint32_t* __restrict__ seed, uint32_t seed_stride, uint32_t* __restrict__ flag,
                    uint32_t dcap, uint32_t* __restrict__ err,
                    const uint32_t* __restrict__ lane_thr, const uint32_t* __restrict__ unit_cost,
                    const uint32_t* __restrict__ unit_lane, uint32_t mode) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t w = blockIdx.x * UPWARD_WARPS + wib;
  if (w >= k) return;
  const uint32_t s = src[w];
  if (s >= n) {
    if (lane == 0) atomicOr(err, DEVERR_PATH);
    return;
  }
  uint32_t* pd = smem + wib * (dcap + PANEL_ROWS);
  uint32_t* srow = pd + dcap;
  const uint32_t p0 = of[s];
  uint4 a = up[2 * (size_t)p0], b = up[2 * (size_t)p0 + 1];
  uint32_t jm = b.x - s;
  const uint32_t D = a.x + jm + 1;  // path entries; the last has index D - 1 and depth 0
  if (D > dcap || jm >= PANEL_ROWS) {
    if (lane == 0) atomicOr(err, DEVERR_PATH);
    return;
  }
  // a seeded unit starts at its seed cost and writes (min) into its source's lane
  const uint32_t c0 = unit_cost ? unit_cost[w] : 0u;
  const uint32_t out_lane = unit_lane ? unit_lane[w] : w;
  // a per-lane threshold also bounds the relaxations: values above it can
  // never lead to a distance within it
  if (lane_thr) threshold = min(threshold, lane_thr[out_lane]);
  const uint32_t thr1 = min(threshold, INF - 1);  // d must also be finite
  const uint32_t lt = lane_thr ? lane_thr[out_lane] : threshold;
  for (uint32_t l = lane; l < D; l += 32) pd[l] = l == 0 ? c0 : INF;
  __syncwarp();
  for (;;) {
    const bool more = a.w != NONE;
    uint4 na = a, nb = b;
    if (more) {  // the next panel's record, while this one is relaxed
      na = up[2 * (size_t)a.w];
      nb = up[2 * (size_t)a.w + 1];
    }
    const uint32_t idx = D - 1 - a.x;  // path index of row 0
    if (a.x > D - 1 || jm > idx || jm >= PANEL_ROWS) {
      if (lane == 0) atomicOr(err, DEVERR_PATH);
      return;
    }
    uint32_t d = lane <= jm ? pd[idx - lane] : INF;
    const uint32_t stride = (a.y >> 8) & 0xFF;
    const uint32_t* wt = up_w + b.z;
    const uint32_t* ends = up_end + b.y;
    if (stride == 4) d = panel_up<4>(d, jm, thr1, wt, ends, a.z, pd, D - 1, lane, srow);
    else if (stride == 8) d = panel_up<8>(d, jm, thr1, wt, ends, a.z, pd, D - 1, lane, srow);
    else if (stride == 12) d = panel_up<12>(d, jm, thr1, wt, ends, a.z, pd, D - 1, lane, srow);
    else d = panel_up<16>(d, jm, thr1, wt, ends, a.z, pd, D - 1, lane, srow);
    if (lane <= jm) {  // the rows are final: write them
      const uint32_t x = b.x - lane;
      const bool in = d != INF && d <= threshold;
      if (mode == UPWARD_OUT_COMPACT) {
        // entry depth * seed_stride + w: indexed from the root, so entries of
        // different sources at one index mostly name the same top-of-tree row
        const uint32_t p = !in ? NONE : pos_of ? pos_of[x] : x;
        reinterpret_cast<uint2*>(seed)[(size_t)(a.x + lane) * seed_stride + w] = make_uint2(p, d);
      } else if (mode == UPWARD_OUT_TILES16) {
        if (in) {  // (within its lane threshold, < 0xFFFF)
          reinterpret_cast<uint16_t*>(seed)[((size_t)(w >> 6) * seed_stride + x) * 64 + (w & 63)] =
              (uint16_t)d;
          atomicOr(&flag[x], 1u << (w >> 6));
        }
      } else if (in) {
        const uint32_t p = pos_of ? pos_of[x] : x;
        if (p != NONE) {
          if (unit_lane) atomicMin(&seed[(size_t)p * seed_stride + out_lane], d);
          else if (mode == UPWARD_OUT_SLAB16)  // (d is within its lane threshold, < 0xFFFF)
            reinterpret_cast<uint16_t*>(seed)[(size_t)p * seed_stride + w] = (uint16_t)d;
          else seed[(size_t)p * seed_stride + w] = d;
          // with lane_thr, a seed above this lane's own threshold can never
          // reach a node within it: it does not mark its row active
          if (flag && d <= lt) atomicOr(&flag[p >> 5], 1u << (p & 31));
        }
      }
    }
    if (!more) break;
    jm = b.w;
    a = na;
    b = nb;
  }
}

}  // namespace

// Path labels fit the shared memory of k_upward_panels' blocks.
static size_t upward_smem(const Graph* g) {
  const uint32_t dcap = ((g->max_depth + 1) + 31) & ~31u;
  return (size_t)UPWARD_WARPS * (dcap + PANEL_ROWS) * 4;
}

bool upward_by_panels(const Graph* g) { return g->panels.n && upward_smem(g) <= 100 * 1024; }

bf_status upward_kernel_init() {
  BF_CUDA(cudaFuncSetAttribute(k_upward_panels, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               100 * 1024));
  return BF_OK;
}

bf_status launch_upward_panels(Graph* g, const uint32_t* d_src, uint64_t k, uint32_t threshold,
                               const uint32_t* pos_map, uint32_t* seed, uint32_t stride,
                               uint32_t* flag, cudaStream_t st, const uint32_t* lane_thr,
                               const uint32_t* unit_cost, const uint32_t* unit_lane,
                               uint32_t mode) {
  const Panels& P = g->panels;
  k_upward_panels<<<(unsigned)((k + UPWARD_WARPS - 1) / UPWARD_WARPS), UPWARD_WARPS * 32,
                    upward_smem(g), st>>>(d_src, (uint32_t)k, threshold, g->n, P.d_of, P.d_up,
                                          P.d_up_end, P.d_up_w, pos_map, seed, stride, flag,
                                          ((g->max_depth + 1) + 31) & ~31u, g->d_err, lane_thr,
                                          unit_cost, unit_lane, mode);
  BF_CUDA(cudaGetLastError());
  return BF_OK;
}

}  // namespace bf
