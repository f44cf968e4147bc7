// cchpanel.cu — triangle relaxation over panels of apexes.
//
// Near the top of the hierarchy a level of single apexes is small work behind
// its own launch, and hundreds of levels follow each other, while the apexes of
// one run share nearly all their upper neighbours: every pair of those is read
// and lowered again by each of them. Up to 16 consecutive ranks of a run (each
// the lowest upper neighbour of the one before) form a panel, relaxed whole in
// two launches per level of panels:
//   solve  the panel's own pairs, then per column (an upper neighbour y outside
//          the panel) the pairs {row, y}, apex after apex: row i final, its
//          candidates into rows j > i;
//   push   every pair of columns {x, y}: the minimum over the panel's apexes, in
//          registers, and one read and at most one atomicMin of the target slot.
// An apex's candidates use its own pairs only once every lower neighbour has
// pushed into them, as in the form by levels, so values, middles, tie-breaks and
// saturating sums are the same. Neither step needs the topology to be closed:
// pairs and directions it lacks hold u32::MAX, pass nothing on and are not
// written.
//
// The 1000 x 1250 region: 650 launches become 63, 45 and 44; a whole
// customization 5.45 -> 4.85 ms, of which 2.6 ms are the copies and 1.3 ms the
// 63 levels below.
#include <algorithm>

#include "customize.cuh"

namespace bf {

namespace {

constexpr uint32_t CP_ROWS = 16;
constexpr uint32_t SOLVE_TPB = 256, SOLVE_Q = 4;             // columns of a warp, side by side
constexpr uint32_t CP_COLS = SOLVE_TPB / 32 * SOLVE_Q;       // columns of a solve unit
constexpr uint32_t CP_TILE = 16;                             // columns on a side of a push unit
constexpr uint32_t PUSH_TPB = 64;

// Entries of a column: its rows, padded to 4, 8 or 16.
__host__ __device__ constexpr uint32_t log_stride(uint32_t k) { return k > 8 ? 4 : k > 4 ? 3 : 2; }
// A level and all above it go by panels once its apexes have this many pair
// candidates in the mean (rows of about 32): below, levels are wide enough to
// fill the GPU by apexes, and a panel has few rows and columns for its two
// launches. Device time on the 1000 x 1250 region (all by apexes: 2.85 ms) at
// 64 / 90 / 200 / 500 / 2000: 2.63 / 2.41 / 2.29 / 2.25 / 2.24 ms; on the town
// (119,249 rows) 0.33 / 0.32 / 0.25 / 0.25 / 0.32 ms.
constexpr uint64_t CP_MIN = 500;

// min(acc, leg1 + leg2) through apex m; legs of weight u32::MAX give ~0, which
// lowers nothing (branch-free: the legs' values differ from lane to lane).
template <bool LEX>
__device__ __forceinline__ uint64_t lower(uint64_t leg1, uint64_t leg2, uint32_t m, uint64_t acc) {
  const uint32_t a = (uint32_t)(leg1 >> 32), b = (uint32_t)(leg2 >> 32);
  const bool skip = a == INF || b == INF;
  const uint32_t hi = skip ? INF : sat_add(a, b);
  const uint32_t lo = skip ? INF : LEX ? sat_add((uint32_t)leg1, (uint32_t)leg2) : m;
  return min(acc, (uint64_t)hi << 32 | lo);
}

// One level of panels, first launch: a block per panel and 32 columns.
// Own pairs: a thread per pair {row j, row m} and direction, lowered through the
// rows i < j one after the other; row j's are final, and published, after step
// j - 1. Each of the panel's blocks does this; the first one writes them back.
// Another may still read them: what it reads lies between the old value and the
// final one, and solves to the final one too.
// Columns: a warp holds four, lane = (row, direction); step i passes row i's
// value to the rows above it by shuffle.
// Bound by its chain of 15 short steps twice over. The steps of a column as one
// lane's straight code (120 relaxations) took 25 us of instruction fetches for
// one launch.
template <bool LEX>
__global__ void __launch_bounds__(SOLVE_TPB)
    k_cp_solve(const uint4* __restrict__ pan, const uint64_t* __restrict__ e0,
               const uint32_t* __restrict__ ent, const uint2* __restrict__ unit, uint64_t u0,
               ulonglong2* __restrict__ sl) {
  __shared__ uint64_t in[CP_ROWS][CP_ROWS][2];
  pdl_launch();
  const uint2 u = unit[u0 + blockIdx.x];
  const uint4 p = pan[u.x];
  const uint32_t* e = ent + e0[u.x];
  const uint32_t lo = p.x, k = p.y, c = p.z, t = threadIdx.x, lane = t & 31;
  unsigned long long* half = reinterpret_cast<unsigned long long*>(sl);
  // this thread's own pair; the plan's arrays do not depend on the launch before
  uint32_t j = 0, m = (t >> 1) + 1;
  const uint32_t d = t & 1;
  while (j + 1 < k && m >= k) {  // row j has pairs m = j + 1 .. k - 1
    m -= k - 1 - j;
    ++j;
    m += 1;
  }
  const bool item = m < k && j < m;
  uint32_t own = item ? e[j * k + m] : 0u;
  const bool own_on = own & (d ? T_DOWN : T_UP);
  // and its lane of the warp's columns
  const uint32_t row = lane >> 1, c0 = u.y * CP_COLS + (t >> 5) * SOLVE_Q, ls = log_stride(k);
  uint32_t ce[SOLVE_Q];
#pragma unroll
  for (uint32_t q = 0; q < SOLVE_Q; ++q) {
    ce[q] = row < k && c0 + q < c ? e[k * k + ((size_t)(c0 + q) << ls) + row] : 0u;
    ce[q] = ce[q] & (d ? T_DOWN : T_UP) ? ce[q] & T_PAIR : NONE;
  }
  own = 2 * (own & T_PAIR) + d;
  pdl_wait();
  const uint64_t own_old = own_on ? __ldcg(half + own) : ~0ull;
  uint64_t v[SOLVE_Q], v_old[SOLVE_Q];
#pragma unroll
  for (uint32_t q = 0; q < SOLVE_Q; ++q)
    v[q] = v_old[q] = ce[q] != NONE ? __ldcg(half + 2 * (size_t)ce[q] + d) : ~0ull;
  uint64_t acc = own_old;
  if (item) in[j][m][d] = acc;
  __syncthreads();
  for (uint32_t i = 0; i + 2 < k; ++i) {
    if (own_on && j > i) {
      // j -> m from (j -> i) + (i -> m); m -> j from (m -> i) + (i -> j)
      acc = lower<LEX>(in[i][j][1 - d], in[i][m][d], lo + i, acc);
      if (j == i + 1) in[j][m][d] = acc;
    }
    __syncthreads();
  }
  if (u.y == 0 && acc != own_old) atomicMin(half + own, (unsigned long long)acc);
  if (c0 >= c) return;
#pragma unroll 5
  for (uint32_t i = 0; i + 1 < CP_ROWS; ++i) {
    if (i + 1 >= k) break;
    const uint64_t leg = i < row && row < k ? in[i][row][1 - d] : ~0ull;
#pragma unroll
    for (uint32_t q = 0; q < SOLVE_Q; ++q) {
      const uint64_t x = __shfl_sync(0xFFFFFFFFu, v[q], 2 * i + d);
      if (ce[q] != NONE) v[q] = lower<LEX>(leg, x, lo + i, v[q]);
    }
  }
#pragma unroll
  for (uint32_t q = 0; q < SOLVE_Q; ++q)
    if (v[q] != v_old[q]) half[2 * (size_t)ce[q] + d] = v[q];
}

// Second launch: 16 x 16 pairs of columns a block, four a thread. The legs of
// all the panel's apexes are staged in shared memory; each target slot is read
// once and lowered at most once per direction for the whole panel.
template <bool LEX>
__global__ void __launch_bounds__(PUSH_TPB)
    k_cp_push(const uint4* __restrict__ pan, const uint64_t* __restrict__ e0,
              const uint32_t* __restrict__ ent, const uint2* __restrict__ unit, uint64_t u0,
              const uint32_t* __restrict__ tgt, ulonglong2* __restrict__ sl) {
  constexpr uint32_t RL = CP_ROWS * CP_TILE / PUSH_TPB;  // legs of a side per thread
  __shared__ ulonglong2 legs[2][CP_ROWS][CP_TILE];
  pdl_launch();
  const uint64_t ui = u0 + blockIdx.x;
  const uint2 u = unit[ui];
  const uint4 p = pan[u.x];
  const uint32_t k = p.y, c = p.z, bx = u.y & 0xFFFF, by = u.y >> 16, t = threadIdx.x;
  const uint32_t* e = ent + e0[u.x] + (size_t)k * k;
  // legs of a side: 16 columns of a stride's rows, in order
  const uint32_t ls = log_stride(k), rm = (1u << ls) - 1, nl = CP_TILE << ls;
  uint32_t le[2 * RL];
#pragma unroll
  for (uint32_t q = 0; q < 2 * RL; ++q) {
    const uint32_t x = t + PUSH_TPB * (q % RL), c0 = (q / RL ? by : bx) * CP_TILE;
    le[q] = x < nl && c0 + (x >> ls) < c ? e[((size_t)c0 << ls) + x] : 0u;
  }
  const uint4 t4 = __ldcs(reinterpret_cast<const uint4*>(tgt + ui * CP_TILE * CP_TILE) + t);
  const uint32_t tg[4] = {t4.x, t4.y, t4.z, t4.w};
  const uint32_t a = t / 4, b = (t % 4) * 4;  // pairs (a, b .. b + 3)
  pdl_wait();
  ulonglong2 old[4], best[4];
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    old[q] = make_ulonglong2(~0ull, ~0ull);
    if (tg[q]) old[q] = __ldcg(sl + (tg[q] & T_PAIR));
  }
#pragma unroll
  for (uint32_t q = 0; q < 2 * RL; ++q) {
    const uint32_t x = t + PUSH_TPB * (q % RL);
    if (x >= nl) continue;
    ulonglong2 s = make_ulonglong2(~0ull, ~0ull);
    if (le[q]) s = __ldcg(sl + (le[q] & T_PAIR));
    legs[q / RL][x & rm][x >> ls] = s;
  }
  __syncthreads();
  if (!(tg[0] | tg[1] | tg[2] | tg[3])) return;
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) best[q] = old[q];
  for (uint32_t i = 0; i < k; ++i) {
    const ulonglong2 x = legs[0][i][a];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const ulonglong2 y = legs[1][i][b + q];
      best[q].x = lower<LEX>(x.y, y.x, p.x + i, best[q].x);  // x -> y
      best[q].y = lower<LEX>(y.y, x.x, p.x + i, best[q].y);  // y -> x
    }
  }
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    if (!tg[q]) continue;
    ulonglong2* at = sl + (tg[q] & T_PAIR);
    if ((tg[q] & T_UP) && best[q].x < old[q].x) atomicMin(&at->x, (unsigned long long)best[q].x);
    if ((tg[q] & T_DOWN) && best[q].y < old[q].y) atomicMin(&at->y, (unsigned long long)best[q].y);
  }
}

// The targets of the push units' pairs, once per plan: {x, y} searched in x's row.
__global__ void __launch_bounds__(CP_TILE * CP_TILE)
    k_cp_targets(const uint4* __restrict__ pan, const uint32_t* __restrict__ cols,
                 const uint2* __restrict__ unit, const uint64_t* __restrict__ qo,
                 const uint32_t* __restrict__ qt, const uint8_t* __restrict__ pf,
                 uint32_t* __restrict__ tgt) {
  const uint2 u = unit[blockIdx.x];
  const uint4 p = pan[u.x];
  const uint32_t i = threadIdx.x;
  const uint32_t a = (u.y & 0xFFFF) * CP_TILE + i / CP_TILE, b = (u.y >> 16) * CP_TILE + i % CP_TILE;
  uint32_t r = 0;
  if (a < b && b < p.z) {
    const uint32_t x = cols[p.w + a], y = cols[p.w + b];
    uint64_t lo = qo[x], hi = qo[x + 1];
    const uint64_t end = hi;
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (qt[mid] < y) lo = mid + 1;
      else hi = mid;
    }
    if (lo < end && qt[lo] == y)
      r = (uint32_t)lo | (pf[lo] & P_UP ? T_UP : 0u) | (pf[lo] & P_DOWN ? T_DOWN : 0u);
  }
  tgt[(size_t)blockIdx.x * CP_TILE * CP_TILE + i] = r;
}

template <class T>
bf_status room_for(T** d, size_t m) {
  if (test_fail_alloc("cch_panels") ||
      cudaMalloc((void**)d, std::max<size_t>(m, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    *d = nullptr;
    return BF_ERR_OOM;
  }
  return BF_OK;
}
template <class T>
bf_status put(T** d, const std::vector<T>& h) {
  const bf_status rc = room_for(d, h.size());
  if (rc) return rc;
  BF_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  return BF_OK;
}

}  // namespace

void free_cch_panels(CchPanels& P) {
  void* p[] = {P.d_pan, P.d_e0, P.d_col, P.d_ent, P.d_solve, P.d_push, P.d_tgt};
  for (void* q : p)
    if (q) cudaFree(q);
  P = CchPanels();
}

static bf_status make_cch_panels(CchPanels& P, uint32_t n, const std::vector<uint64_t>& qo,
                                 const std::vector<uint32_t>& qt, const std::vector<uint8_t>& pf,
                                 const std::vector<uint32_t>& lev, uint32_t n_levels,
                                 const uint64_t* d_qo, const uint32_t* d_qt, const uint8_t* d_pf,
                                 uint64_t room, cudaStream_t s) {
  // the first level whose apexes have CP_MIN candidates in the mean
  std::vector<uint64_t> cand(n_levels, 0), apexes(n_levels, 0);
  for (uint32_t m = 0; m < n; ++m) {
    const uint64_t d = qo[m + 1] - qo[m];
    if (d < 2) continue;
    cand[lev[m]] += d * (d - 1) / 2;
    ++apexes[lev[m]];
  }
  uint32_t first = 0;
  while (first < n_levels && cand[first] < std::max<uint64_t>(CP_MIN * apexes[first], 1)) ++first;
  if (first >= n_levels) return BF_OK;

  std::vector<uint32_t> of(n, NONE);  // row -> panel
  std::vector<uint4> pan;
  for (uint32_t x = 0; x < n;) {
    if (lev[x] < first) {
      ++x;
      continue;
    }
    uint32_t e = x;
    while (e - x + 1 < CP_ROWS && qo[e + 1] > qo[e] && qt[qo[e]] == e + 1) ++e;
    for (uint32_t y = x; y <= e; ++y) of[y] = (uint32_t)pan.size();
    pan.push_back(make_uint4(x, e - x + 1, 0, 0));
    x = e + 1;
  }
  std::vector<uint32_t> plev(pan.size(), 0), cols, ent;
  std::vector<uint64_t> e0(pan.size());
  uint32_t levels = 1;
  uint64_t push_units = 0;
  std::vector<uint32_t> uni, tmp;
  for (uint32_t p = 0; p < pan.size(); ++p) {
    const uint32_t lo = pan[p].x, k = pan[p].y, hi = lo + k - 1;
    uni.clear();
    for (uint32_t j = lo; j <= hi; ++j) {
      auto b = std::upper_bound(qt.begin() + qo[j], qt.begin() + qo[j + 1], hi);
      tmp.clear();
      std::set_union(uni.begin(), uni.end(), b, qt.begin() + qo[j + 1], std::back_inserter(tmp));
      uni.swap(tmp);
    }
    const uint32_t c = (uint32_t)uni.size();
    const uint64_t nb = (c + CP_TILE - 1) / CP_TILE;
    push_units += nb * (nb + 1) / 2;
    if (nb > 0xFFFF || cols.size() + c > 0xFFFFFFFFull || push_units > 0x7FFFFFFFull ||
        (push_units * CP_TILE * CP_TILE + ent.size() + k * k + ((uint64_t)c << log_stride(k))) * 4 >
            room)
      return BF_OK;  // left to the levels of apexes
    pan[p].z = c;
    pan[p].w = (uint32_t)cols.size();
    e0[p] = ent.size();
    ent.resize(ent.size() + k * k + ((size_t)c << log_stride(k)), 0u);
    uint32_t* en = ent.data() + e0[p];
    for (uint32_t j = lo; j <= hi; ++j) {
      uint32_t at = 0;
      for (uint64_t i = qo[j]; i < qo[j + 1]; ++i) {
        const uint32_t w =
            (uint32_t)i | (pf[i] & P_UP ? T_UP : 0u) | (pf[i] & P_DOWN ? T_DOWN : 0u);
        if (qt[i] <= hi) {
          en[(j - lo) * k + (qt[i] - lo)] = w;
        } else {
          while (uni[at] != qt[i]) ++at;
          en[k * k + ((size_t)at << log_stride(k)) + (j - lo)] = w;
        }
      }
    }
    cols.insert(cols.end(), uni.begin(), uni.end());
    // (every column lies in a panel: levels rise along every edge)
    for (uint32_t y : uni) plev[of[y]] = std::max(plev[of[y]], plev[p] + 1);
    levels = std::max(levels, plev[p] + 1);
  }
  // work units by level; a row alone has nothing to solve, one column nothing to push
  std::vector<std::vector<uint32_t>> by(levels);
  for (uint32_t p = 0; p < pan.size(); ++p) by[plev[p]].push_back(p);
  std::vector<uint2> solve, push;
  P.lvl_solve.assign(1, 0);
  P.lvl_push.assign(1, 0);
  for (uint32_t l = 0; l < levels; ++l) {
    for (uint32_t p : by[l]) {
      const uint32_t k = pan[p].y, c = pan[p].z;
      if (k > 2 || (k == 2 && c))
        for (uint32_t b = 0; b < std::max(1u, (c + CP_COLS - 1) / CP_COLS); ++b)
          solve.push_back(make_uint2(p, b));
      if (c < 2) continue;
      const uint32_t nb = (c + CP_TILE - 1) / CP_TILE;
      for (uint32_t x = 0; x < nb; ++x)
        for (uint32_t y = x; y < nb; ++y) push.push_back(make_uint2(p, x | y << 16));
    }
    P.lvl_solve.push_back(solve.size());
    P.lvl_push.push_back(push.size());
  }
  bf_status rc;
  if ((rc = put(&P.d_pan, pan)) || (rc = put(&P.d_e0, e0)) || (rc = put(&P.d_col, cols)) ||
      (rc = put(&P.d_ent, ent)) || (rc = put(&P.d_solve, solve)) || (rc = put(&P.d_push, push)) ||
      (rc = room_for(&P.d_tgt, push.size() * CP_TILE * CP_TILE)))
    return rc;
  BF_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // (the uploads, before `s`)
  if (!push.empty())
    k_cp_targets<<<(unsigned)push.size(), CP_TILE * CP_TILE, 0, s>>>(P.d_pan, P.d_col, P.d_push,
                                                                     d_qo, d_qt, d_pf, P.d_tgt);
  BF_CUDA(cudaGetLastError());
  BF_CUDA(cudaStreamSynchronize(s));
  P.first_level = first;
  return BF_OK;
}

bf_status build_cch_panels(CchPanels& P, uint32_t n, const std::vector<uint64_t>& qo,
                           const std::vector<uint32_t>& qt, const std::vector<uint8_t>& pf,
                           const std::vector<uint32_t>& lev, uint32_t n_levels,
                           const uint64_t* d_qo, const uint32_t* d_qt, const uint8_t* d_pf,
                           uint64_t room, cudaStream_t s) {
  bf_status rc;
  try {
    rc = make_cch_panels(P, n, qo, qt, pf, lev, n_levels, d_qo, d_qt, d_pf, room, s);
  } catch (const std::bad_alloc&) {
    rc = BF_ERR_OOM;
  }
  if (rc != BF_ERR_OOM) return rc;
  free_cch_panels(P);  // no room for them: left to the levels of apexes
  return BF_OK;
}

cudaError_t relax_cch_panels(const CchPanels& P, bool lex, bool pdl, ulonglong2* sl,
                             cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  for (size_t l = 0; l + 1 < P.lvl_solve.size() && e == cudaSuccess; ++l) {
    const uint64_t s0 = P.lvl_solve[l], s1 = P.lvl_solve[l + 1];
    const uint64_t p0 = P.lvl_push[l], p1 = P.lvl_push[l + 1];
    if (s1 > s0) {
      e = launch_level(lex ? k_cp_solve<true> : k_cp_solve<false>, dim3((unsigned)(s1 - s0)),
                       SOLVE_TPB, pdl, s, (const uint4*)P.d_pan, (const uint64_t*)P.d_e0,
                       (const uint32_t*)P.d_ent, (const uint2*)P.d_solve, s0, sl);
      pdl = true;
    }
    if (p1 > p0 && e == cudaSuccess) {
      e = launch_level(lex ? k_cp_push<true> : k_cp_push<false>, dim3((unsigned)(p1 - p0)), PUSH_TPB,
                       pdl, s, (const uint4*)P.d_pan, (const uint64_t*)P.d_e0,
                       (const uint32_t*)P.d_ent, (const uint2*)P.d_push, p0,
                       (const uint32_t*)P.d_tgt, sl);
      pdl = true;
    }
  }
  return e;
}

}  // namespace bf
