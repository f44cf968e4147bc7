// panel.cu — panels: the pull DAG blocked into small dense min-plus tiles.
//
// Every DOWN edge joins a node to one of its elimination-tree ancestors, and
// the nodes of a run (consecutive ranks r, r + 1, ... with parent(x) = x + 1,
// a separator of the nested dissection) pull from nearly the same ancestors.
// A panel is up to 16 consecutive ranks of one run. Its in-edges are kept as
//   * the list of ancestors above the panel that any of its rows pulls from,
//     with a dense weight tile [source][row] (INF where an edge is absent;
//     71 to 90 % of the entries of the rows a matrix sweeps are edges), and
//   * a triangle [row][row] of the edges inside the panel.
// Rows of a panel are counted from its highest rank down: row j pulls from
// rows i < j. So a sweep loads a source row once for up to 16 rows instead of
// once per edge (10k targets on the country graph: 0.45 M gathers of a row
// instead of 3.85 M), and the rows of a panel depend on each other only
// within a lane, so they are swept together: 91 dependent levels of panels
// instead of 1116 levels of rows.
//
// The rows a target set needs (the ancestors of the targets) meet each run in
// a top part [x, end], so a panel is needed in a top part too: its first
// k rows counted from the highest. The static tiles serve every target set;
// a restricted schedule is only a list of (panel, rows) per level.

#include <algorithm>
#include <cstring>

#include "engine.cuh"
#include "scan.cuh"

namespace bf {

namespace {

// Tile strides (rows a panel's weight tile is padded to).
constexpr uint32_t CLASSES[] = {1, 2, 4, 8, 12, 16};

uint32_t stride_of(uint32_t k) {
  for (uint32_t c : CLASSES)
    if (k <= c) return c;
  return PANEL_ROWS;
}

// Work buckets of a level's items, heaviest first, so that a level does not
// end on a long item that started last.
constexpr uint32_t BUCKETS = 4;
uint32_t bucket_of(uint64_t work) { return work >= 2048 ? 0 : work >= 512 ? 1 : work >= 64 ? 2 : 3; }

struct HostPanel {
  uint32_t hi, k, nu, chunk;
  uint64_t u0, w0;  // within the chunk
};

struct Chunk {
  std::vector<HostPanel> pan;
  std::vector<uint32_t> src, w;
};

// Panels of rows (lo .. hi] of one run, split in two where the dense tile
// would hold more than four times the edges it stands for (rows of one run
// that pull from different ancestors), so the tiles never exceed a small
// multiple of the graph.
void emit_panels(uint32_t lo, uint32_t hi, uint32_t ci, const uint64_t* off, const uint32_t* src,
                 const uint32_t* w, Chunk& out, std::vector<uint32_t>& uni) {
  const uint32_t k = hi - lo + 1, ks = stride_of(k);
  uni.clear();
  uint64_t edges = 0;
  for (uint32_t v = lo; v <= hi; ++v)
    for (uint64_t e = off[v]; e < off[v + 1]; ++e)
      if (src[e] > hi) {
        uni.push_back(src[e]);
        ++edges;
      }
  std::sort(uni.begin(), uni.end());
  uni.erase(std::unique(uni.begin(), uni.end()), uni.end());
  if (k > 1 && uni.size() * (uint64_t)k > 4 * edges + 64) {
    const uint32_t mid = lo + k / 2;  // rows mid .. hi, then lo .. mid - 1
    emit_panels(mid, hi, ci, off, src, w, out, uni);
    emit_panels(lo, mid - 1, ci, off, src, w, out, uni);
    return;
  }
  const uint32_t nu = (uint32_t)uni.size();
  HostPanel p{hi, k, nu, ci, out.src.size(), out.w.size()};
  out.src.insert(out.src.end(), uni.begin(), uni.end());
  // [source][row] tile, then the [row][row] triangle; starts are multiples
  // of four words so that rows of a tile load as 16-byte vectors
  const size_t words = ((size_t)nu * ks + (size_t)ks * ks + 3) & ~(size_t)3;
  out.w.resize(out.w.size() + words, INF);
  uint32_t* t = out.w.data() + p.w0;
  uint32_t* tri = t + (size_t)nu * ks;
  for (uint32_t j = 0; j < k; ++j) {
    const uint32_t v = hi - j;
    for (uint64_t e = off[v]; e < off[v + 1]; ++e) {
      uint32_t* at;
      if (src[e] > hi)
        at = t + (size_t)(std::lower_bound(uni.begin(), uni.end(), src[e]) - uni.begin()) * ks + j;
      else
        at = tri + (size_t)(hi - src[e]) * ks + j;
      *at = std::min(*at, w[e]);
    }
  }
  out.pan.push_back(p);
}

template <class T>
bf_status upload(T** d, const std::vector<T>& h, Panels& P) {
  const size_t bytes = std::max<size_t>(h.size(), 1) * sizeof(T);
  if (cudaMalloc((void**)d, bytes) != cudaSuccess) {
    cudaGetLastError();
    *d = nullptr;
    return BF_ERR_OOM;
  }
  P.bytes += bytes;
  if (!h.empty()) BF_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  return BF_OK;
}

}  // namespace

void free_panels(Panels& P) {
  void* q[] = {P.d_a, P.d_b, P.d_of, P.d_hibits, P.d_src, P.d_w};
  for (void* x : q)
    if (x) cudaFree(x);
  P = Panels();
}

// Panels of the pull CSR by rank (in-edges of v: off, src, w; src > v) on
// runs given by run_end. Leaves P empty (the item sweep then serves every
// call) when the tiles do not fit 32-bit offsets or the device.
bf_status build_panels(Graph* g, const std::vector<uint32_t>& run_end,
                       const std::vector<uint64_t>& off, const std::vector<uint32_t>& src,
                       const std::vector<uint32_t>& w, uint64_t max_up) {
  Panels& P = g->panels;
  const uint32_t n = g->n;
  if (!n || off[n] >= 0x20000000ull) return BF_OK;
  // chunks of whole runs
  std::vector<uint32_t> cut{0};
  const uint32_t step = std::max<uint32_t>(4096, n / 512);
  while (cut.back() < n) {
    const uint64_t at = std::min<uint64_t>((uint64_t)cut.back() + step, n);
    cut.push_back(at >= n ? n : run_end[at - 1] + 1);
  }
  const uint32_t nc = (uint32_t)cut.size() - 1;
  std::vector<Chunk> ch(nc);
  parallel_for(nc, [&](uint64_t c) {
    std::vector<uint32_t> uni;
    // runs from the highest rank down; a run's panels from its end down
    for (uint32_t v = cut[c + 1]; v > cut[c];) {
      const uint32_t e = v - 1;
      uint32_t a = e;
      while (a > cut[c] && run_end[a - 1] == e) --a;
      for (uint32_t hi = e;;) {
        const uint32_t lo = hi - a >= PANEL_ROWS ? hi - PANEL_ROWS + 1 : a;
        emit_panels(lo, hi, (uint32_t)c, off.data(), src.data(), w.data(), ch[c], uni);
        if (lo == a) break;
        hi = lo - 1;
      }
      v = a;
    }
  });
  uint64_t np = 0, ns = 0, nw = 0;
  std::vector<uint64_t> sbase(nc), wbase(nc);
  for (uint32_t c = 0; c < nc; ++c) {
    sbase[c] = ns;
    wbase[c] = nw;
    np += ch[c].pan.size();
    ns += ch[c].src.size();
    nw += ch[c].w.size();
  }
  if (nw >= 0xFFFFFFFFull || ns >= 0xFFFFFFFFull) return BF_OK;
  // levels (a panel one past its highest source panel), panels from the
  // highest rank down, and the longest path of the pull DAG
  std::vector<uint32_t> lvl_at(n, 0);  // by rank: the level of its panel
  std::vector<uint32_t> lvl;
  lvl.reserve(np);
  uint32_t L = 0;
  for (uint32_t c = nc; c-- > 0;)
    for (const HostPanel& p : ch[c].pan) {
      uint32_t l = 0;
      for (uint32_t i = 0; i < p.nu; ++i) l = std::max(l, lvl_at[ch[c].src[p.u0 + i]] + 1);
      for (uint32_t j = 0; j < p.k; ++j) lvl_at[p.hi - j] = l;
      lvl.push_back(l);
      L = std::max(L, l + 1);
    }
  std::vector<uint32_t>().swap(lvl_at);
  uint64_t max_down = 0;
  {
    std::vector<uint64_t> at(n, 0);
    for (uint32_t v = n; v-- > 0;) {
      for (uint64_t e = off[v]; e < off[v + 1]; ++e) at[v] = std::max(at[v], at[src[e]] + w[e]);
      max_down = std::max(max_down, at[v]);
    }
  }
  // every label of a sweep is the weight of an UP path and a DOWN path
  P.max_label = max_up + max_down;
  P.n_levels = L;
  P.lvl_first.assign(L + 1, 0);
  for (uint32_t l : lvl) ++P.lvl_first[l + 1];
  for (uint32_t l = 0; l < L; ++l) P.lvl_first[l + 1] += P.lvl_first[l];
  std::vector<uint4> a(np);
  std::vector<uint2> b(np);
  std::vector<uint32_t> of(n, NONE), hib((n + 31) / 32 + 1, 0);
  {
    std::vector<uint32_t> at(P.lvl_first.begin(), P.lvl_first.end() - 1);
    size_t i = 0;
    for (uint32_t c = nc; c-- > 0;)
      for (const HostPanel& p : ch[c].pan) {
        const uint32_t l = lvl[i++], id = at[l]++, ks = stride_of(p.k);
        a[id] = make_uint4(p.hi, p.k | ks << 8 | bucket_of((uint64_t)p.nu * p.k) << 16, p.nu, l);
        b[id] = make_uint2((uint32_t)(sbase[c] + p.u0), (uint32_t)(wbase[c] + p.w0));
        of[p.hi] = id;
        hib[p.hi >> 5] |= 1u << (p.hi & 31);
      }
  }
  P.n = (uint32_t)np;
  std::vector<uint32_t> s(ns), t(nw);
  parallel_for(nc, [&](uint64_t c) {
    std::copy(ch[c].src.begin(), ch[c].src.end(), s.begin() + sbase[c]);
    std::copy(ch[c].w.begin(), ch[c].w.end(), t.begin() + wbase[c]);
    Chunk().pan.swap(ch[c].pan);
    std::vector<uint32_t>().swap(ch[c].src);
    std::vector<uint32_t>().swap(ch[c].w);
  });
  bf_status rc;
  if ((rc = upload(&P.d_a, a, P)) || (rc = upload(&P.d_b, b, P)) || (rc = upload(&P.d_of, of, P)) ||
      (rc = upload(&P.d_hibits, hib, P)) || (rc = upload(&P.d_src, s, P)) ||
      (rc = upload(&P.d_w, t, P))) {
    free_panels(P);
    return rc == BF_ERR_OOM ? BF_OK : rc;
  }
  return BF_OK;
}

namespace {

// ---- restricted schedule ----------------------------------------------------

// Mark the targets' root paths (rank bitmap `rows`), a warp per target, whole
// runs at once, stopping where another warp has been: a set bit at x was set
// by a warp that marks x's run to its end and goes on at the parent. Each
// word of bits that a warp sets first names the panels it opened (their
// highest rank is in the word): they are listed and counted per level and
// work bucket.
__global__ void __launch_bounds__(128)
    k_pn_mark(const uint32_t* __restrict__ tgt, uint32_t T, const uint32_t* __restrict__ parent,
              const uint32_t* __restrict__ run_end, uint32_t n, const uint32_t* __restrict__ hib,
              const uint32_t* __restrict__ of, const uint4* __restrict__ pan,
              uint32_t* __restrict__ rows, uint32_t* __restrict__ list,
              uint32_t* __restrict__ n_list, uint32_t* __restrict__ hist,
              uint32_t* __restrict__ err) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= T) return;
  uint32_t x = tgt[w];
  if (x >= n) {
    if (lane == 0) atomicOr(err, DEVERR_PATH);
    return;
  }
  for (uint32_t guard = 0; x != NONE && guard < n; ++guard) {
    if ((*(volatile const uint32_t*)&rows[x >> 5] >> (x & 31)) & 1u) break;
    const uint32_t e = run_end[x];
    if (e < x || e >= n) {
      if (lane == 0) atomicOr(err, DEVERR_PATH);
      return;
    }
    for (uint32_t wd = (x >> 5) + lane; wd <= e >> 5; wd += 32) {
      uint32_t m = ~0u;
      if (wd == x >> 5) m &= ~0u << (x & 31);
      if (wd == e >> 5) m &= ~0u >> (31 - (e & 31));
      uint32_t f = m & ~atomicOr(&rows[wd], m) & hib[wd];
      while (f) {
        const uint32_t r = wd * 32 + __ffs(f) - 1;
        f &= f - 1;
        const uint32_t p = of[r];
        const uint4 a = pan[p];
        list[atomicAdd(n_list, 1u)] = p;
        atomicAdd(&hist[a.w * BUCKETS + (a.y >> 16)], 1u);
      }
    }
    __syncwarp();
    x = parent[e];
  }
}

// Level -> first item, and each (level, bucket)'s cursor in its place.
__global__ void __launch_bounds__(SCAN_TPB)
    k_pn_levels(uint32_t* __restrict__ hist, uint32_t L, uint32_t* __restrict__ lvl) {
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t l0 = 0; l0 < L; l0 += SCAN_TPB) {
    const uint32_t l = l0 + threadIdx.x;
    uint32_t h[BUCKETS], tot = 0;
    for (uint32_t b = 0; b < BUCKETS; ++b) {
      h[b] = l < L ? hist[l * BUCKETS + b] : 0;
      tot += h[b];
    }
    uint32_t all;
    uint32_t cur = carry + block_exscan<uint32_t>(tot, &all);
    if (l < L) {
      lvl[l] = cur;
      for (uint32_t b = 0; b < BUCKETS; ++b) {
        hist[l * BUCKETS + b] = cur;
        cur += h[b];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) lvl[L] = carry;
}

__device__ __forceinline__ uint32_t row_at(const uint32_t* __restrict__ rows,
                                           const uint32_t* __restrict__ wpre, uint32_t r) {
  return wpre[r >> 5] + __popc(rows[r >> 5] & ((1u << (r & 31)) - 1u));
}

// Items {row of the highest rank, rows | stride << 8, sources, -} and
// {first source, first weight}, placed level by level; target rows.
__global__ void __launch_bounds__(256)
    k_pn_items(const uint32_t* __restrict__ list, uint32_t m, const uint4* __restrict__ pan,
               const uint2* __restrict__ panb, const uint32_t* __restrict__ rows,
               const uint32_t* __restrict__ wpre, uint32_t* __restrict__ cursor,
               uint4* __restrict__ item, const uint32_t* __restrict__ tgt, uint64_t T,
               uint32_t* __restrict__ trow) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m || i < T;
       i += (uint64_t)gridDim.x * blockDim.x) {
    if (i < T) trow[i] = row_at(rows, wpre, tgt[i]);
    if (i >= m) continue;
    const uint32_t p = list[i];
    const uint4 a = pan[p];
    const uint2 b = panb[p];
    const uint32_t hi = a.x, k = a.y & 0xFF, lo = hi - k + 1;
    const uint32_t r1 = row_at(rows, wpre, hi), r0 = row_at(rows, wpre, lo);
    const uint32_t live = r1 - r0 + 1;  // the set ranks of [lo, hi] are its top part
    const uint32_t at = atomicAdd(&cursor[a.w * BUCKETS + (a.y >> 16)], 1u);
    item[2 * (size_t)at] = make_uint4(r1, live | (a.y & 0xFF00), a.z, 0);
    item[2 * (size_t)at + 1] = make_uint4(b.x, b.y, 0, 0);
  }
}

__global__ void __launch_bounds__(256)
    k_pn_cidx(uint32_t n, const uint32_t* __restrict__ rows, const uint32_t* __restrict__ wpre,
              uint32_t* __restrict__ cidx) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    cidx[r] = (rows[r >> 5] >> (r & 31)) & 1u ? row_at(rows, wpre, r) : NONE;
}

}  // namespace

// Scratch of the panel schedule builder (per context; sized by the graph).
struct PanelScratch {
  uint32_t* rows = nullptr;   // [W + 1] rank bitmap
  uint32_t* wpre = nullptr;   // [W + 2]
  uint32_t* bsum = nullptr;
  uint32_t* list = nullptr;   // [panels] opened panels
  uint32_t* hist = nullptr;   // [levels * BUCKETS], then the level table [levels + 1]
  uint32_t* tgt = nullptr;    // uploaded targets
  uint32_t* h_back = nullptr;  // page-locked: row count, panel count, level table
  size_t cap_tgt = 0;
};

void free_panel_scratch(PanelScratch* s) {
  if (!s) return;
  void* p[] = {s->rows, s->wpre, s->bsum, s->list, s->hist, s->tgt};
  for (void* q : p)
    if (q) cudaFree(q);
  if (s->h_back) cudaFreeHost(s->h_back);
  delete s;
}

namespace {

template <class T>
bf_status grow(T** p, size_t& cap, size_t need, Graph* g, bool slack) {
  if (need <= cap && *p) return BF_OK;
  if (*p) {
    cudaFree(*p);
    g->device_bytes -= cap * sizeof(T);
  }
  *p = nullptr;
  cap = 0;
  const size_t m = std::max<size_t>(slack ? need + need / 8 : need, 1);
  if (cudaMalloc((void**)p, m * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    set_error("cudaMalloc for the panel schedule failed");
    return BF_ERR_OOM;
  }
  cap = m;
  g->device_bytes += m * sizeof(T);
  return BF_OK;
}

}  // namespace

// The panel schedule of h_tgt (host) / d_tgt (the same targets on the device,
// or null). Rows are the targets' ancestors in rank order (a superset of the
// rows that reach a target: 1.28 times as many for 10k targets on the country
// graph, 9 % more gathers; peeling them off first costs a small call more
// than it saves).
bf_status build_schedule_panels(Graph* g, Ctx& c, Sched& sc, const uint32_t* h_tgt,
                                const uint32_t* d_tgt, uint64_t T, uint64_t key, cudaStream_t st) {
  const Panels& P = g->panels;
  const uint32_t n = g->n, W = (n + 31) / 32, L = P.n_levels;
  const unsigned nbw = (unsigned)((W + 1 + SCAN_BLOCK - 1) / SCAN_BLOCK);
  bf_status rc;
  if (!c.ps) {
    c.ps = new (std::nothrow) PanelScratch();
    if (!c.ps) {
      set_error("out of host memory");
      return BF_ERR_OOM;
    }
  }
  PanelScratch& s = *c.ps;
  size_t none = 0;
  if (!s.h_back) {
    // one list entry per panel, two counters behind the level table
    if ((rc = grow(&s.rows, none = 0, (size_t)W + 1, g, false)) ||
        (rc = grow(&s.wpre, none = 0, (size_t)W + 2, g, false)) ||
        (rc = grow(&s.bsum, none = 0, (size_t)nbw + 2, g, false)) ||
        (rc = grow(&s.list, none = 0, P.n, g, false)) ||
        (rc = grow(&s.hist, none = 0, (size_t)L * (BUCKETS + 1) + 3, g, false)))
      return rc;
    if (cudaHostAlloc((void**)&s.h_back, ((size_t)L + 4) * 4, cudaHostAllocDefault) !=
        cudaSuccess) {
      cudaGetLastError();
      s.h_back = nullptr;
      set_error("cannot allocate the schedule read-back buffer");
      return BF_ERR_OOM;
    }
  }
  if ((rc = grow(&sc.d_cidx, sc.cap_cidx, n, g, false)) ||
      (rc = grow(&sc.d_trow, sc.cap_t, T, g, true)))
    return rc;
  if (!d_tgt) {
    if ((rc = grow(&s.tgt, s.cap_tgt, T, g, true))) return rc;
    BF_CUDA(cudaMemcpyAsync(s.tgt, h_tgt, T * 4, cudaMemcpyHostToDevice, st));
    d_tgt = s.tgt;
  }
  uint32_t* lvl = s.hist + (size_t)L * BUCKETS;  // [L + 1], then the panel count
  uint32_t* n_list = lvl + L + 1;
  BF_CUDA(cudaMemsetAsync(s.rows, 0, ((size_t)W + 1) * 4, st));
  BF_CUDA(cudaMemsetAsync(s.hist, 0, ((size_t)L * (BUCKETS + 1) + 3) * 4, st));
  k_pn_mark<<<(unsigned)((T + 3) / 4), 128, 0, st>>>(d_tgt, (uint32_t)T, g->d_parent, g->d_run_end,
                                                     n, P.d_hibits, P.d_of, P.d_a, s.rows, s.list,
                                                     n_list, s.hist, g->d_err);
  scan_launch<uint32_t>(PopVal{s.rows}, (uint64_t)W, s.bsum, s.wpre, st);
  k_pn_levels<<<1, SCAN_TPB, 0, st>>>(s.hist, L, lvl);
  k_pn_cidx<<<std::min<uint32_t>((n + 255) / 256, 152 * 16), 256, 0, st>>>(n, s.rows, s.wpre,
                                                                          sc.d_cidx);
  BF_CUDA(cudaGetLastError());
  BF_CUDA(cudaMemcpyAsync(s.h_back, lvl, ((size_t)L + 2) * 4, cudaMemcpyDeviceToHost, st));
  BF_CUDA(cudaMemcpyAsync(s.h_back + L + 2, s.wpre + W, 4, cudaMemcpyDeviceToHost, st));
  BF_CUDA(cudaStreamSynchronize(st));
  const uint32_t m = s.h_back[L + 1], n_r = s.h_back[L + 2];
  if (m != s.h_back[L] || m > P.n || n_r > n) {
    set_error("panel schedule: inconsistent counts");
    return BF_ERR_DEVICE;
  }
  if ((rc = grow(&sc.d_pitem, sc.cap_pitem, 2 * (size_t)m, g, true))) return rc;
  k_pn_items<<<(unsigned)std::max<uint64_t>(1, (std::max<uint64_t>(m, T) + 255) / 256), 256, 0,
               st>>>(s.list, m, P.d_a, P.d_b, s.rows, s.wpre, s.hist, sc.d_pitem, d_tgt, T,
                     sc.d_trow);
  BF_CUDA(cudaGetLastError());
  sc.lvl_pan.assign(s.h_back, s.h_back + L + 1);
  sc.panel = true;
  sc.n_r = n_r;
  sc.counted = false;
  sc.lvl_item.clear();  // per-level tables of the item form are made on demand
  sc.lvl_row.clear();
  sc.lvl_edge.clear();
  sc.T = T;
  sc.key = key;
  sc.tgt.assign(h_tgt, h_tgt + T);
  sc.uses = 0;
  sc.dev_built = true;
  sc.lvl_erec_ready = false;
  sc.ranks.clear();
  sc.cidx_ready = true;
  sc.cidx_dirty = true;
  sc.hub_order.clear();
  sc.hub_rows = NONE;
  sc.valid = true;
  return BF_OK;
}

namespace {

// ---- sweep ------------------------------------------------------------------

// Labels at or above this stand for "unreachable" in the one-instruction form
// of the relaxation (below), which a sweep uses when no finite label reaches
// it; the slab itself always holds INF.
constexpr uint32_t FAR = 0x7FFFFFFFu;

// min(acc, d + w). SAT: any u32 labels and weights; the sum saturates at INF
// (min(d, ~w) + w is d + w, or INF where that would pass it). Otherwise labels
// are at most FAR + 1 and weights at most FAR: no sum wraps, and add and min
// are one instruction.
template <bool SAT>
__device__ __forceinline__ uint32_t relax(uint32_t d, uint32_t w, uint32_t acc) {
  return SAT ? __viaddmin_u32(min(d, ~w), w, acc) : __viaddmin_u32(d, w, acc);
}

template <uint32_t N>
__device__ __forceinline__ void load_lanes(const uint32_t* p, uint32_t (&v)[N]) {
  if constexpr (N == 4) {
    const uint4 x = __ldcg(reinterpret_cast<const uint4*>(p));
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else if constexpr (N == 2) {
    const uint2 x = __ldcg(reinterpret_cast<const uint2*>(p));
    v[0] = x.x, v[1] = x.y;
  } else {
    v[0] = __ldcg(p);
  }
}

template <uint32_t K>
__device__ __forceinline__ void load_weights(const uint32_t* p, uint32_t (&w)[K]) {
  if constexpr (K >= 4) {
#pragma unroll
    for (uint32_t j = 0; j < K; j += 4) {
      const uint4 x = *reinterpret_cast<const uint4*>(p + j);
      w[j] = x.x, w[j + 1] = x.y, w[j + 2] = x.z, w[j + 3] = x.w;
    }
  } else if constexpr (K == 2) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    w[0] = x.x, w[1] = x.y;
  } else {
    w[0] = *p;
  }
}

template <uint32_t LPT, uint32_t WL, uint32_t WS>
struct PanelShape {
  static constexpr uint32_t LANES = 32 * WL * LPT;   // lanes of a block
  static constexpr uint32_t TPB = 32 * WL * WS;
  static constexpr uint32_t CH = WS > 1 ? 256 : 64;  // sources staged at a time
};

template <uint32_t LPT, uint32_t WL, uint32_t WS>
struct PanelSmem {
  using S = PanelShape<LPT, WL, WS>;
  uint32_t w[S::CH * PANEL_ROWS];
  uint32_t tri[PANEL_ROWS * PANEL_ROWS];
  uint32_t row[S::CH];
  uint32_t red[WS > 1 ? PANEL_ROWS * S::LANES : 1];
};

template <uint32_t K, uint32_t LPT, uint32_t WL, uint32_t WS, bool SAT>
__device__ __forceinline__ void panel_item(const uint4 a, const uint4 b,
                                           const uint32_t* __restrict__ psrc,
                                           const uint32_t* __restrict__ pw,
                                           const uint32_t* __restrict__ cidx,
                                           uint32_t* __restrict__ slab, uint32_t Kp,
                                           const uint32_t* __restrict__ seeded,
                                           PanelSmem<LPT, WL, WS>& sm) {
  using S = PanelShape<LPT, WL, WS>;
  constexpr uint32_t FARV = SAT ? INF : FAR + 1;
  const uint32_t t = threadIdx.x, warp = t >> 5;
  const uint32_t live = a.y & 0xFF, stride = a.y >> 8, nu = a.z;
  const uint32_t lane0 = blockIdx.y * S::LANES;
  const uint32_t lane = lane0 + ((warp % WL) * 32 + (t & 31)) * LPT;
  const bool on = lane < Kp;
  const uint32_t* tri = pw + b.y + (size_t)nu * stride;
  auto weight = [](uint32_t w) { return SAT ? w : min(w, FAR); };
  auto stage = [&](uint32_t c0, uint32_t m) {
    for (uint32_t i = t; i < m; i += S::TPB) sm.row[i] = cidx[psrc[b.x + c0 + i]];
    if (stride == K) {
      if constexpr (K >= 4) {
        const uint4* w4 = reinterpret_cast<const uint4*>(pw + b.y + (size_t)c0 * K);
        for (uint32_t i = t; i < m * (K / 4); i += S::TPB) {
          uint4 x = w4[i];
          x.x = weight(x.x), x.y = weight(x.y), x.z = weight(x.z), x.w = weight(x.w);
          reinterpret_cast<uint4*>(sm.w)[i] = x;
        }
      } else {
        for (uint32_t i = t; i < m * K; i += S::TPB)
          sm.w[i] = weight(pw[b.y + (size_t)c0 * K + i]);
      }
    } else {
      for (uint32_t i = t; i < m * K; i += S::TPB)
        sm.w[i] = weight(pw[b.y + (size_t)(c0 + i / K) * stride + i % K]);
    }
  };
  // all of this is static: staged before the previous level is done
  stage(0, min(nu, S::CH));
  for (uint32_t i = t; i < K * K; i += S::TPB) sm.tri[i] = weight(tri[(i / K) * stride + i % K]);
  if constexpr (WS > 1)
    for (uint32_t i = t; i < K * S::LANES; i += S::TPB) sm.red[i] = FARV;
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t acc[K][LPT];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j)
#pragma unroll
    for (uint32_t l = 0; l < LPT; ++l) acc[j][l] = FARV;
  if constexpr (WS == 1) {  // seeds of the rows that have one
    if (on)
#pragma unroll
      for (uint32_t j = 0; j < K; ++j) {
        const uint32_t r = a.x - j;
        if (j < live && ((seeded[r >> 5] >> (r & 31)) & 1u)) {
          uint32_t v[LPT];
          load_lanes<LPT>(slab + (size_t)r * Kp + lane, v);
#pragma unroll
          for (uint32_t l = 0; l < LPT; ++l) acc[j][l] = min(v[l], FARV);
        }
      }
  }
  for (uint32_t c0 = 0; c0 < nu; c0 += S::CH) {
    const uint32_t m = min(nu - c0, S::CH);
    if (c0) {
      __syncthreads();
      stage(c0, m);
      __syncthreads();
    }
    if (on) {
      constexpr uint32_t U = 4;  // source rows in flight per thread
      for (uint32_t s0 = warp / WL; s0 < m; s0 += U * WS) {
        uint32_t d[U][LPT];
#pragma unroll
        for (uint32_t q = 0; q < U; ++q) {
          const uint32_t s = s0 + q * WS;
          if (s < m) {
            load_lanes<LPT>(slab + (size_t)sm.row[s] * Kp + lane, d[q]);
          } else {
#pragma unroll
            for (uint32_t l = 0; l < LPT; ++l) d[q][l] = INF;
          }
        }
#pragma unroll
        for (uint32_t q = 0; q < U; ++q) {
          const uint32_t s = s0 + q * WS;
          if (s >= m) break;
          uint32_t w[K];
          load_weights<K>(sm.w + s * K, w);
#pragma unroll
          for (uint32_t l = 0; l < LPT; ++l) {
            const uint32_t x = min(d[q][l], FARV);
#pragma unroll
            for (uint32_t j = 0; j < K; ++j) acc[j][l] = relax<SAT>(x, w[j], acc[j][l]);
          }
        }
      }
    }
  }
  if constexpr (WS == 1) {
    if (!on) return;
#pragma unroll
    for (uint32_t i = 0; i + 1 < K; ++i)
#pragma unroll
      for (uint32_t j = i + 1; j < K; ++j) {
        const uint32_t w = sm.tri[i * K + j];
#pragma unroll
        for (uint32_t l = 0; l < LPT; ++l) acc[j][l] = relax<SAT>(acc[i][l], w, acc[j][l]);
      }
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) {
      if (j >= live) break;
      uint32_t v[LPT];
#pragma unroll
      for (uint32_t l = 0; l < LPT; ++l)
        v[l] = !SAT && acc[j][l] >= FAR ? INF : acc[j][l];
      uint32_t* row = slab + (size_t)(a.x - j) * Kp + lane;
      if constexpr (LPT == 4)
        *reinterpret_cast<uint4*>(row) = make_uint4(v[0], v[1], v[2], v[3]);
      else if constexpr (LPT == 2)
        *reinterpret_cast<uint2*>(row) = make_uint2(v[0], v[1]);
      else
        *row = v[0];
    }
  } else {
    // the warps of a lane hold minima over different sources: combine them,
    // then a thread per lane solves the triangle
    if (on) {
      const uint32_t at = ((warp % WL) * 32 + (t & 31)) * LPT;
#pragma unroll
      for (uint32_t j = 0; j < K; ++j)
#pragma unroll
        for (uint32_t l = 0; l < LPT; ++l)
          if (acc[j][l] < FARV) atomicMin(&sm.red[j * S::LANES + at + l], acc[j][l]);
    }
    __syncthreads();
    const uint32_t x = lane0 + t;
    if (t >= S::LANES || x >= Kp) return;
    uint32_t v[K];
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) {
      const uint32_t r = a.x - j;
      v[j] = sm.red[j * S::LANES + t];
      if (j < live && ((seeded[r >> 5] >> (r & 31)) & 1u))
        v[j] = min(v[j], __ldcg(slab + (size_t)r * Kp + x));
    }
#pragma unroll
    for (uint32_t i = 0; i + 1 < K; ++i)
#pragma unroll
      for (uint32_t j = i + 1; j < K; ++j) v[j] = relax<SAT>(v[i], sm.tri[i * K + j], v[j]);
#pragma unroll
    for (uint32_t j = 0; j < K; ++j)
      if (j < live) slab[(size_t)(a.x - j) * Kp + x] = !SAT && v[j] >= FAR ? INF : v[j];
  }
}

// One level of panels: blockIdx.x = item, blockIdx.y = block of LANES lanes.
// WL warps lie along the lanes (LPT lanes a thread), WS warps share a lane's
// sources. Bound by the gathers of source rows where there are many lanes, by
// the chain of dependent levels where there are few. Against the item sweep
// (a level of rows, a gather per edge), sweep time: 10k x 10k on the country
// graph 27.2 -> 14.4 ms, 1000 x 1500 on the 1000 x 1250 region 2.18 -> 0.60
// ms, 37 x 421 there 1.69 -> 0.40 ms, 100 x 100 on grid100 1.59 -> 0.30 ms.
template <uint32_t LPT, uint32_t WL, uint32_t WS, bool SAT>
__global__ void __launch_bounds__(32 * WL * WS)
    k_sweep_panels(const uint4* __restrict__ item, uint32_t i0, const uint32_t* __restrict__ psrc,
                   const uint32_t* __restrict__ pw, const uint32_t* __restrict__ cidx,
                   uint32_t* __restrict__ slab, uint32_t Kp, const uint32_t* __restrict__ seeded) {
  __shared__ __align__(16) PanelSmem<LPT, WL, WS> sm;
  asm volatile("griddepcontrol.launch_dependents;");
  const uint4 a = item[2 * (size_t)(i0 + blockIdx.x)], b = item[2 * (size_t)(i0 + blockIdx.x) + 1];
  const uint32_t live = a.y & 0xFF;
#define BF_PANEL(K) \
  panel_item<K, LPT, WL, WS, SAT>(a, b, psrc, pw, cidx, slab, Kp, seeded, sm)
  if (live > 12) BF_PANEL(16);
  else if (live > 8) BF_PANEL(12);
  else if (live > 4) BF_PANEL(8);
  else if (live > 2) BF_PANEL(4);
  else if (live == 2) BF_PANEL(2);
  else BF_PANEL(1);
#undef BF_PANEL
}

template <bool SAT>
cudaError_t launch_panels(const Graph* g, const Sched& sc, uint32_t i0, uint32_t m, uint32_t* slab,
                          uint32_t Kp, const uint32_t* seeded, unsigned tpb, bool pdl,
                          cudaStream_t st) {
  const Panels& P = g->panels;
  auto go = [&](auto kern, uint32_t lanes, unsigned threads) {
    return launch_level(kern, dim3(m, (Kp + lanes - 1) / lanes), threads, pdl, st,
                        (const uint4*)sc.d_pitem, i0, (const uint32_t*)P.d_src,
                        (const uint32_t*)P.d_w, (const uint32_t*)sc.d_cidx, slab, Kp, seeded);
  };
  // A thread walks all sources of its panel (up to a few hundred at the top
  // of the tree): with few blocks in a level that chain is the level's time,
  // so eight warps share it and combine in shared memory; with enough blocks
  // to fill the GPU the combine costs more than it saves.
  const uint64_t wide = (uint64_t)m * ((Kp + 511) / 512);
  if (wide >= 2ull * g->sm_count && Kp > 128) {
    if (tpb >= 256) return go(k_sweep_panels<4, 8, 1, SAT>, 1024, 256);
    if (tpb == 128) return go(k_sweep_panels<4, 4, 1, SAT>, 512, 128);
    return go(k_sweep_panels<4, 2, 1, SAT>, 256, 64);
  }
  if (Kp <= 32) return go(k_sweep_panels<1, 1, 8, SAT>, 32, 256);
  if (Kp <= 64) return go(k_sweep_panels<2, 1, 8, SAT>, 64, 256);
  return go(k_sweep_panels<4, 1, 8, SAT>, 128, 256);
}

}  // namespace

// Whether a sweep from seed costs of at most max_seed may hold finite labels
// beyond the one-instruction relaxation's range.
bool panels_saturate(const Graph* g, uint64_t max_seed) {
  return g->panels.max_label + max_seed >= FAR;
}

// The level launches of a panel schedule on `st`. sat: labels may pass the
// range of the one-instruction relaxation (seed costs, or the graph's own
// longest paths).
cudaError_t sweep_panels(Graph* g, Sched& sc, uint32_t* slab, uint32_t Kp, unsigned tpb, bool sat,
                         cudaStream_t st, uint64_t* launches, const uint32_t* seeded) {
  const bool pdl = g->tune.pdl != 0;
  for (uint32_t l = 0; l + 1 < sc.lvl_pan.size(); ++l) {
    const uint32_t i0 = sc.lvl_pan[l], m = sc.lvl_pan[l + 1] - i0;
    if (!m) continue;
    const cudaError_t e = sat ? launch_panels<true>(g, sc, i0, m, slab, Kp, seeded, tpb, pdl, st)
                              : launch_panels<false>(g, sc, i0, m, slab, Kp, seeded, tpb, pdl, st);
    if (e != cudaSuccess) return e;
    ++*launches;
  }
  return cudaSuccess;
}

}  // namespace bf
