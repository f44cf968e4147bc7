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

bf_status panel_kernels_init();

namespace {

// Tile strides (rows a panel's weight tile is padded to): multiples of four
// words, so that a source's weights are a 16-byte aligned bulk copy.
constexpr uint32_t CLASSES[] = {4, 8, 12, 16};

uint32_t stride_of(uint32_t k) {
  for (uint32_t c : CLASSES)
    if (k <= c) return c;
  return PANEL_ROWS;
}

// A work item of a panel schedule: {slab row of the panel's highest rank (row j
// of the panel is j rows below it), rows | stride << 5 | sources << 10, first
// weight, first entry of the sources' slab rows}.
constexpr uint32_t MAX_SOURCES = 1u << 22;
__device__ __forceinline__ uint32_t item_live(const uint4& it) { return it.y & 31u; }
__device__ __forceinline__ uint32_t item_stride(const uint4& it) { return (it.y >> 5) & 31u; }
__device__ __forceinline__ uint32_t item_sources(const uint4& it) { return it.y >> 10; }

// Buckets of a level's panels by rows and work.
constexpr uint32_t BUCKETS = 5;
uint32_t bucket_of(uint32_t k, uint64_t work) {
  return k <= 4 ? 4 : work >= 2048 ? 0 : work >= 512 ? 1 : work >= 64 ? 2 : 3;
}

// Labels at or above this stand for "unreachable" in the one-instruction form
// of the relaxation (relax() below), which a sweep uses when no finite label
// reaches it; its rows then hold FAR + 1 where an item sweep's hold INF.
constexpr uint32_t FAR = 0x7FFFFFFFu;

struct HostPanel {
  uint32_t hi, k, nu, chunk;
  uint64_t u0, w0;  // within the chunk
  uint32_t up_n;    // the same of the UP tile
  uint64_t up_u0, up_w0;
};

// A direction's edges by rank: the other ends of v's edges are e in
// [off[v], off[v + 1]), given by their depth in the elimination tree (all lie on
// v's root path, so the depth names them) or by their rank.
struct Edges {
  const uint64_t* off;
  const uint32_t *end, *w, *len;  // len: null on one-channel graphs
};

struct Chunk {
  std::vector<HostPanel> pan;
  std::vector<uint32_t> src, w;
  std::vector<uint16_t> em;  // per source: the rows it has an edge into
  std::vector<uint32_t> up_end, up_w;
  std::vector<uint32_t> len, up_len;  // like w and up_w, on two-channel graphs
};

// The other ends outside the panel (`outside`), each once, ascending. False: a
// dense tile of k rows would hold more than four times the edges it stands for.
template <class F>
bool outer_ends(uint32_t lo, uint32_t hi, const Edges& g, F outside, std::vector<uint32_t>& uni) {
  uni.clear();
  uint64_t edges = 0;
  for (uint32_t v = lo; v <= hi; ++v)
    for (uint64_t e = g.off[v]; e < g.off[v + 1]; ++e)
      if (outside(g.end[e])) {
        uni.push_back(g.end[e]);
        ++edges;
      }
  std::sort(uni.begin(), uni.end());
  uni.erase(std::unique(uni.begin(), uni.end()), uni.end());
  return hi == lo || uni.size() * (uint64_t)(hi - lo + 1) <= 4 * edges + 64;
}

// Panels of rows [lo, hi] of one run, split in two where a tile would be mostly
// empty (rows of one run with edges to different ancestors), so the tiles never
// exceed a small multiple of the graph.
void emit_panels(uint32_t lo, uint32_t hi, uint32_t ci, const Edges& dn, const Edges& up,
                 const uint32_t* depth, Chunk& out, std::vector<uint32_t>* uni, uint16_t* tm) {
  const uint32_t k = hi - lo + 1, ks = stride_of(k), top = depth[hi];
  const bool dense_dn = outer_ends(lo, hi, dn, [=](uint32_t r) { return r > hi; }, uni[0]);
  const bool dense_up = outer_ends(lo, hi, up, [=](uint32_t d) { return d < top; }, uni[1]);
  if (!dense_dn || !dense_up) {
    const uint32_t mid = lo + k / 2;  // rows mid .. hi, then lo .. mid - 1
    emit_panels(mid, hi, ci, dn, up, depth, out, uni, tm);
    emit_panels(lo, mid - 1, ci, dn, up, depth, out, uni, tm);
    return;
  }
  // [other end][row] tiles, each followed by its [row][row] triangle; starts
  // are multiples of four words so that rows of a tile load as 16-byte vectors
  auto tile = [&](std::vector<uint32_t>& ends, std::vector<uint32_t>& w, const std::vector<uint32_t>& u) {
    ends.insert(ends.end(), u.begin(), u.end());
    const size_t at = w.size();
    w.resize(at + u.size() * ks + (size_t)ks * ks, INF);
    return w.data() + at;
  };
  HostPanel p{hi,           k, (uint32_t)uni[0].size(), ci, out.src.size(), out.w.size(),
              (uint32_t)uni[1].size(), out.up_end.size(), out.up_w.size()};
  uint32_t* t = tile(out.src, out.w, uni[0]);
  uint32_t* tri = t + (size_t)p.nu * ks;
  uint32_t* ut = tile(out.up_end, out.up_w, uni[1]);
  uint32_t* utri = ut + (size_t)p.up_n * ks;
  out.em.resize(out.em.size() + p.nu, 0);
  uint16_t* em = out.em.data() + p.u0;
  if (dn.len) {
    out.len.resize(out.w.size(), INF);
    out.up_len.resize(out.up_w.size(), INF);
  }
  // parallel edges: the smaller (time, length)
  auto put = [](uint32_t* at, std::vector<uint32_t>& w, std::vector<uint32_t>& len, const Edges& g,
                uint64_t e) {
    if (!g.len) {
      *at = std::min(*at, g.w[e]);
      return;
    }
    uint32_t& l = len[at - w.data()];
    if (g.w[e] < *at || (g.w[e] == *at && g.len[e] < l)) {
      *at = g.w[e];
      l = g.len[e];
    }
  };
  auto find = [](const std::vector<uint32_t>& u, uint32_t x) {
    return (size_t)(std::lower_bound(u.begin(), u.end(), x) - u.begin());
  };
  for (uint32_t j = 0; j < k; ++j) {
    const uint32_t v = hi - j;
    for (uint64_t e = dn.off[v]; e < dn.off[v + 1]; ++e) {
      const uint32_t s = dn.end[e];
      uint32_t* at;
      if (s > hi) {
        const size_t q = find(uni[0], s);
        at = t + q * ks + j;
        em[q] |= (uint16_t)(1u << j);
      } else {
        at = tri + (size_t)(hi - s) * ks + j;
        tm[s] |= (uint16_t)(1u << j);
      }
      put(at, out.w, out.len, dn, e);
    }
    for (uint64_t e = up.off[v]; e < up.off[v + 1]; ++e) {
      const uint32_t d = up.end[e];
      uint32_t* at = d < top ? ut + find(uni[1], d) * ks + j : utri + (size_t)j * ks + (d - top);
      put(at, out.up_w, out.up_len, up, e);
    }
  }
  out.pan.push_back(p);
}

template <class T>
bf_status upload(T** d, const std::vector<T>& h, Panels& P) {
  const size_t bytes = std::max<size_t>(h.size(), 1) * sizeof(T);
  if (test_fail_alloc("panels") || cudaMalloc((void**)d, bytes) != cudaSuccess) {
    cudaGetLastError();
    *d = nullptr;
    return BF_ERR_OOM;
  }
  P.bytes += bytes;
  if (!h.empty()) BF_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
  return BF_OK;
}

__global__ void __launch_bounds__(256)
    k_pack_weights(const uint32_t* __restrict__ w, uint64_t m, uint32_t absent, uint32_t cap,
                   uint32_t* __restrict__ out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = w[i] == absent ? cap : min(w[i], cap);
    out[i] = x | x << 16;
  }
}

// The weight tiles for 16-bit lanes, from d_w.
bf_status pack_weights(Panels& P, uint64_t m) {
  for (uint32_t** p : {&P.d_w16, &P.d_w16s}) {
    if (cudaMalloc((void**)p, m * 4) != cudaSuccess) {
      cudaGetLastError();
      *p = nullptr;
      return BF_ERR_OOM;
    }
    P.bytes += m * 4;
    k_pack_weights<<<152 * 8, 256>>>(P.d_w, m, P.absent, p == &P.d_w16 ? 0x7FFFu : 0xFFFFu, *p);
    BF_CUDA(cudaGetLastError());
  }
  BF_CUDA(cudaDeviceSynchronize());
  return BF_OK;
}

}  // namespace

void free_panels(Panels& P) {
  void* q[] = {P.d_a, P.d_b, P.d_of, P.d_hibits, P.d_lvl, P.d_lvl_small, P.d_src, P.d_w, P.d_em,
               P.d_tm, P.d_up, P.d_up_end, P.d_up_w, P.d_w16,
               P.d_w16s, P.d_len, P.d_up_len};
  for (void* x : q)
    if (x) cudaFree(x);
  P = Panels();
}

static bf_status make_panels(Graph* g, const std::vector<uint32_t>& run_end,
                             const std::vector<uint32_t>& parent,
                             const std::vector<uint32_t>& depth, const std::vector<uint64_t>& off,
                             const std::vector<uint32_t>& src, const std::vector<uint32_t>& w,
                             const std::vector<uint64_t>& up_off, const std::vector<uint2>& up_rec,
                             uint64_t max_up, const uint32_t* len, const uint32_t* up_len) {
  Panels& P = g->panels;
  const uint32_t n = g->n;
  bf_status rc;
  if (!n || off[n] >= 0x20000000ull || up_off[n] >= 0x20000000ull) return BF_OK;
  std::vector<uint32_t> up_end(up_off[n]), up_w(up_off[n]);
  parallel_for((n + 65535) / 65536, [&](uint64_t c) {
    for (uint64_t v = c << 16; v < std::min<uint64_t>(n, (c + 1) << 16); ++v)
      for (uint64_t e = up_off[v]; e < up_off[v + 1]; ++e) {
        up_end[e] = depth[v] - up_rec[e].x;
        up_w[e] = up_rec[e].y;
      }
  });
  const Edges dn{off.data(), src.data(), w.data(), len};
  const Edges up{up_off.data(), up_end.data(), up_w.data(), up_len};
  // chunks of whole runs
  std::vector<uint32_t> cut{0};
  const uint32_t step = std::max<uint32_t>(4096, n / 512);
  while (cut.back() < n) {
    const uint64_t at = std::min<uint64_t>((uint64_t)cut.back() + step, n);
    cut.push_back(at >= n ? n : run_end[at - 1] + 1);
  }
  const uint32_t nc = (uint32_t)cut.size() - 1;
  std::vector<Chunk> ch(nc);
  std::vector<uint16_t> tm(n, 0);  // by rank: the rows of its panel it has an edge into
  parallel_for(nc, [&](uint64_t c) {
    if (test_fail_alloc("panel_tiles")) throw std::bad_alloc();
    std::vector<uint32_t> uni[2];
    // runs from the highest rank down; a run's panels from its end down
    for (uint32_t v = cut[c + 1]; v > cut[c];) {
      const uint32_t e = v - 1;
      uint32_t a = e;
      while (a > cut[c] && run_end[a - 1] == e) --a;
      for (uint32_t hi = e;;) {
        const uint32_t lo = hi - a >= PANEL_ROWS ? hi - PANEL_ROWS + 1 : a;
        emit_panels(lo, hi, (uint32_t)c, dn, up, depth.data(), ch[c], uni, tm.data());
        if (lo == a) break;
        hi = lo - 1;
      }
      v = a;
    }
  });
  uint64_t np = 0, ns = 0, nw = 0, up_ns = 0, up_nw = 0;
  std::vector<uint64_t> sbase(nc), wbase(nc), up_sbase(nc), up_wbase(nc);
  for (uint32_t c = 0; c < nc; ++c) {
    sbase[c] = ns;
    wbase[c] = nw;
    np += ch[c].pan.size();
    ns += ch[c].src.size();
    nw += ch[c].w.size();
    up_sbase[c] = up_ns;
    up_wbase[c] = up_nw;
    up_ns += ch[c].up_end.size();
    up_nw += ch[c].up_w.size();
  }
  if (std::max(nw, up_nw) >= 0xFFFFFFFFull || std::max(ns, up_ns) >= 0xFFFFFFFFull) return BF_OK;
  // the graph's budget holds the panels beside what its calls take at least
  // without them (the plain engine's two slabs, 32 lanes of every row, schedules
  // of work items and their builder's scratch): else a budget that serves a call
  // without panels would be too small with them
  const uint64_t bytes = 56 * np + 6ull * n + n / 8 + 8ull * (g->n_levels + 1) + 6 * ns +
                         12 * nw + 4 * (up_ns + up_nw) + (len ? 4 * (nw + up_nw) : 0) + 65536;
  const uint64_t beside = n * (2ull * PLAIN_K * 4 + 32 * (len ? 8 : 4) + 128) + 40 * off[n];
  if (g->device_bytes + bytes + beside > g->hbm_budget) return BF_OK;
  for (const Chunk& c : ch)
    for (const HostPanel& p : c.pan)
      if (p.nu >= MAX_SOURCES) return BF_OK;
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
  P.n_src = ns;
  P.lvl_small.clear();
  P.lvl_first.assign(L + 1, 0);
  for (uint32_t l : lvl) ++P.lvl_first[l + 1];
  for (uint32_t l = 0; l < L; ++l) P.lvl_first[l + 1] += P.lvl_first[l];
  std::vector<uint4> a(np);
  std::vector<uint2> b(np);
  std::vector<uint4> up_a(2 * np);
  std::vector<uint32_t> of(n, NONE), hib((n + 31) / 32 + 1, 0);
  // panels of a level: heaviest bucket first (a level then does not end on a
  // long item that started last), those of at most four rows last, from the highest rank down in each (so
  // neighbours share sources)
  {
    std::vector<uint32_t> at((size_t)L * BUCKETS + 1, 0);
    size_t i = 0;
    for (uint32_t c = nc; c-- > 0;)
      for (const HostPanel& p : ch[c].pan)
        ++at[lvl[i++] * (size_t)BUCKETS + bucket_of(p.k, (uint64_t)p.nu * p.k) + 1];
    for (size_t k = 1; k < at.size(); ++k) at[k] += at[k - 1];
    for (uint32_t l = 0; l < L; ++l) P.lvl_small.push_back(at[l * (size_t)BUCKETS + BUCKETS - 1]);
    i = 0;
    for (uint32_t c = nc; c-- > 0;)
      for (const HostPanel& p : ch[c].pan) {
        const uint32_t l = lvl[i++], ks = stride_of(p.k);
        const uint32_t id = at[l * (size_t)BUCKETS + bucket_of(p.k, (uint64_t)p.nu * p.k)]++;
        a[id] = make_uint4(p.hi, p.k | ks << 8, p.nu, 0);
        b[id] = make_uint2((uint32_t)(sbase[c] + p.u0), (uint32_t)(wbase[c] + p.w0));
        up_a[2 * (size_t)id] = make_uint4(depth[p.hi], p.k | ks << 8, p.up_n, NONE);
        up_a[2 * (size_t)id + 1] = make_uint4(p.hi, (uint32_t)(up_sbase[c] + p.up_u0),
                                              (uint32_t)(up_wbase[c] + p.up_w0), 0);
        for (uint32_t j = 0; j < p.k; ++j) of[p.hi - j] = id;
        hib[p.hi >> 5] |= 1u << (p.hi & 31);
      }
  }
  // the next panel of a root path, and the row it enters at
  for (size_t i = 0; i < np; ++i) {
    const uint32_t x = parent[a[i].x];
    if (x == NONE) continue;
    up_a[2 * i].w = of[x];
    up_a[2 * i + 1].w = a[of[x]].x - x;
  }
  P.n = (uint32_t)np;
  // where no label of a sweep from the graph's own nodes reaches FAR, absent
  // edges weigh FAR, which the one-instruction relaxation needs
  P.absent = P.max_label < FAR ? FAR : INF;
  nw += PANEL_ROWS * PANEL_ROWS;  // (a tile of 12 rows may be read as one of 16)
  std::vector<uint32_t> s(ns), t(nw, P.absent), us(up_ns), ut(up_nw);
  std::vector<uint16_t> em(ns);
  std::vector<uint32_t> tl(len ? nw : 0, INF), utl(len ? up_nw : 0);
  parallel_for(nc, [&](uint64_t c) {
    std::copy(ch[c].src.begin(), ch[c].src.end(), s.begin() + sbase[c]);
    std::copy(ch[c].em.begin(), ch[c].em.end(), em.begin() + sbase[c]);
    std::transform(ch[c].w.begin(), ch[c].w.end(), t.begin() + wbase[c],
                   [&](uint32_t x) { return x == INF ? P.absent : x; });
    std::copy(ch[c].up_end.begin(), ch[c].up_end.end(), us.begin() + up_sbase[c]);
    std::copy(ch[c].up_w.begin(), ch[c].up_w.end(), ut.begin() + up_wbase[c]);
    std::copy(ch[c].len.begin(), ch[c].len.end(), tl.begin() + (len ? wbase[c] : 0));
    std::copy(ch[c].up_len.begin(), ch[c].up_len.end(), utl.begin() + (len ? up_wbase[c] : 0));
    ch[c] = Chunk();
  });
  if ((rc = upload(&P.d_a, a, P)) || (rc = upload(&P.d_b, b, P)) ||
      (rc = upload(&P.d_of, of, P)) || (rc = upload(&P.d_hibits, hib, P)) ||
      (rc = upload(&P.d_lvl, P.lvl_first, P)) ||
      (rc = upload(&P.d_lvl_small, P.lvl_small, P)) || (rc = upload(&P.d_src, s, P)) ||
      (rc = upload(&P.d_w, t, P)) || (rc = upload(&P.d_em, em, P)) ||
      (rc = upload(&P.d_tm, tm, P)) ||
      (rc = upload(&P.d_up, up_a, P)) || (rc = upload(&P.d_up_end, us, P)) ||
      (rc = upload(&P.d_up_w, ut, P)) || (len && (rc = upload(&P.d_len, tl, P))) ||
      (len && (rc = upload(&P.d_up_len, utl, P))) || (rc = pack_weights(P, nw))) {
    free_panels(P);
    return rc == BF_ERR_OOM ? BF_OK : rc;
  }
  g->device_bytes += P.bytes;
  return BF_OK;
}

// Panels of the DOWN edges by target rank (in-edges of v: off, src, w; src > v)
// and the UP edges by source rank (records {depth difference, w}), on runs given
// by run_end. Leaves P empty (items and paths then serve every call) when the
// tiles do not fit 32-bit offsets, the graph's budget, the device or the host's
// memory.
bf_status build_panels(Graph* g, const std::vector<uint32_t>& run_end,
                       const std::vector<uint32_t>& parent, const std::vector<uint32_t>& depth,
                       const std::vector<uint64_t>& off, const std::vector<uint32_t>& src,
                       const std::vector<uint32_t>& w, const std::vector<uint64_t>& up_off,
                       const std::vector<uint2>& up_rec, uint64_t max_up, const uint32_t* len,
                       const uint32_t* up_len) {
  bf_status rc;
  if ((rc = panel_kernels_init()) || (rc = upward_kernel_init()) ||
      (rc = upward_2ch_kernel_init()))
    return rc;
  try {
    return make_panels(g, run_end, parent, depth, off, src, w, up_off, up_rec, max_up, len,
                       up_len);
  } catch (const std::bad_alloc&) {
    free_panels(g->panels);
    return BF_OK;
  }
}

namespace {

// ---- restricted schedule ----------------------------------------------------

// Mark the targets' root paths (rank bitmap `rows`), a warp per target, whole
// runs at once, stopping where another warp has been: a set bit at x was set
// by a warp that marks x's run to its end and goes on at the parent. Each
// word of bits that a warp sets first names the panels it opened (their
// highest rank is in the word): their bits are set and their sources counted.
__global__ void __launch_bounds__(128)
    k_pn_mark(const uint32_t* __restrict__ tgt, uint32_t T, const uint32_t* __restrict__ parent,
              const uint32_t* __restrict__ run_end, uint32_t n, const uint32_t* __restrict__ hib,
              const uint32_t* __restrict__ of, const uint4* __restrict__ pan,
              uint32_t* __restrict__ rows, uint32_t* __restrict__ pbits,
              uint32_t* __restrict__ n_src, uint32_t* __restrict__ err) {
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
      uint32_t ns = 0;
      while (f) {
        const uint32_t p = of[wd * 32 + __ffs(f) - 1];
        f &= f - 1;
        atomicOr(&pbits[p >> 5], 1u << (p & 31));
        ns += pan[p].z;
      }
      if (ns) atomicAdd(n_src, ns);
    }
    __syncwarp();
    x = parent[e];
  }
}

// Exclusive scans of the bit counts of the two bitmaps, both in each launch
// (blockIdx.y, or the block): block sums, their scan, then the words'.
struct TwoBitmaps {
  const uint32_t* bits[2];
  uint32_t words[2];
  uint32_t* bsum[2];  // room for a sum per block and the total
  uint32_t* pre[2];   // [words + 1]
};
__global__ void __launch_bounds__(SCAN_TPB) k_pn_sums(TwoBitmaps b) {
  const uint32_t y = blockIdx.y, i0 = blockIdx.x * SCAN_BLOCK;
  if (i0 >= b.words[y]) return;
  uint32_t s = 0;
  for (uint32_t j = 0; j < SCAN_ITEMS; ++j) {
    const uint32_t i = i0 + j * SCAN_TPB + threadIdx.x;
    if (i < b.words[y]) s += __popc(b.bits[y][i]);
  }
  uint32_t tot;
  block_exscan<uint32_t>(s, &tot);
  if (threadIdx.x == 0) b.bsum[y][blockIdx.x] = tot;
}
__global__ void __launch_bounds__(SCAN_TPB) k_pn_top(TwoBitmaps b) {
  __shared__ uint32_t carry;
  const uint32_t y = blockIdx.x, nb = (b.words[y] + SCAN_BLOCK - 1) / SCAN_BLOCK;
  uint32_t* bsum = b.bsum[y];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b0 = 0; b0 < nb; b0 += SCAN_TPB) {
    const uint32_t i = b0 + threadIdx.x, v = i < nb ? bsum[i] : 0u;
    uint32_t tot;
    const uint32_t ex = block_exscan<uint32_t>(v, &tot), c = carry;
    if (i < nb) bsum[i] = c + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry = c + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) b.pre[y][b.words[y]] = carry;
}
__global__ void __launch_bounds__(SCAN_TPB) k_pn_out(TwoBitmaps b) {
  const uint32_t y = blockIdx.y, i0 = blockIdx.x * SCAN_BLOCK + threadIdx.x * SCAN_ITEMS;
  if (blockIdx.x * SCAN_BLOCK >= b.words[y]) return;
  uint32_t v[SCAN_ITEMS], s = 0;
  for (uint32_t j = 0; j < SCAN_ITEMS; ++j) {
    v[j] = i0 + j < b.words[y] ? __popc(b.bits[y][i0 + j]) : 0u;
    s += v[j];
  }
  uint32_t tot;
  uint32_t run = b.bsum[y][blockIdx.x] + block_exscan<uint32_t>(s, &tot);
  for (uint32_t j = 0; j < SCAN_ITEMS; ++j) {
    if (i0 + j < b.words[y]) b.pre[y][i0 + j] = run;
    run += v[j];
  }
}

// Panels in order (ids ascending, so level by level), level -> first item, and
// the row count behind the table.
__global__ void __launch_bounds__(256)
    k_pn_list(TwoBitmaps b, const uint32_t* __restrict__ lvl_first, uint32_t L,
              uint32_t* __restrict__ list, uint32_t* __restrict__ lvl, uint32_t* __restrict__ n_r) {
  const uint32_t *pbits = b.bits[1], *ppre = b.pre[1], words = b.words[1];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words || i <= L;
       i += gridDim.x * blockDim.x) {
    if (i == 0) *n_r = b.pre[0][b.words[0]];
    if (i <= L) {
      const uint32_t p = lvl_first[i];  // (one word of slack behind the bits)
      lvl[i] = ppre[p >> 5] + __popc(pbits[p >> 5] & ((1u << (p & 31)) - 1u));
    }
    if (i >= words) continue;
    uint32_t m = pbits[i], at = ppre[i];
    while (m) {
      list[at++] = i * 32 + __ffs(m) - 1;
      m &= m - 1;
    }
  }
}

__device__ __forceinline__ uint32_t row_at(const uint32_t* __restrict__ rows,
                                           const uint32_t* __restrict__ wpre, uint32_t r) {
  return wpre[r >> 5] + __popc(rows[r >> 5] & ((1u << (r & 31)) - 1u));
}

// Items with the slab rows of their sources (a warp per panel), and the target
// rows.
__global__ void __launch_bounds__(256)
    k_pn_items(const uint32_t* __restrict__ list, uint32_t m, const uint4* __restrict__ pan,
               const uint2* __restrict__ panb, const uint32_t* __restrict__ psrc,
               const uint32_t* __restrict__ rows, const uint32_t* __restrict__ wpre,
               const uint32_t* __restrict__ cidx, uint32_t* __restrict__ n_row, uint4* __restrict__ item,
               uint32_t* __restrict__ prow, const uint32_t* __restrict__ tgt, uint64_t T,
               uint32_t* __restrict__ trow, uint32_t* __restrict__ live) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t threads = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < T; i += threads) {
    const uint32_t r = cidx[tgt[i]];
    trow[i] = r;
    atomicOr(&live[r >> 5], 1u << (r & 31));
  }
  const uint32_t lane = threadIdx.x & 31;
  for (uint64_t i = tid >> 5; i < m; i += threads >> 5) {
    const uint32_t p = list[i];
    const uint4 a = pan[p];
    const uint2 b = panb[p];
    uint32_t at = 0;
    if (lane == 0) {
      const uint32_t hi = a.x, lo = hi - (a.y & 0xFF) + 1;
      const uint32_t r1 = row_at(rows, wpre, hi), r0 = row_at(rows, wpre, lo);
      const uint32_t live = r1 - r0 + 1;  // the set ranks of [lo, hi] are its top part
      at = atomicAdd(n_row, a.z);
      item[i] = make_uint4(r1, live | (a.y >> 8) << 5 | a.z << 10, b.y, at);
    }
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    for (uint32_t q = lane; q < a.z; q += 32) prow[at + q] = cidx[psrc[b.x + q]];
  }
}

__global__ void __launch_bounds__(256)
    k_pn_cidx(uint32_t n, const uint32_t* __restrict__ rows, const uint32_t* __restrict__ wpre,
              uint32_t* __restrict__ cidx) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    cidx[r] = (rows[r >> 5] >> (r & 31)) & 1u ? row_at(rows, wpre, r) : NONE;
}

// Rows that reach a target (the others are swept in vain) and their in-edges,
// counted for the call's statistics beside the sweep: one cooperative launch
// walks the levels from the last to the first. A panel's live rows are its
// targets, what its live rows pull from inside the panel, and what panels of
// later levels marked; it marks its sources with an edge into one of them. A
// warp takes a panel; levels of at most one block's warps are run by block 0
// alone, the others by all blocks, with the bounded grid barrier between.
// Bound by about four dependent loads a level. (Peeling rows without live
// out-edges off the ancestors, as the item builder does, took 608 blocks and a
// round per peeled layer: with it beside the sweep a 37 x 421 table on the
// region took 0.80 ms, without any counting 0.61 ms.)
constexpr uint32_t LIVE_TPB = 1024, LIVE_WARPS = LIVE_TPB / 32;
__global__ void __launch_bounds__(LIVE_TPB)
    k_pn_live(const uint32_t* __restrict__ lvl, uint32_t L, const uint32_t* __restrict__ list,
              const uint4* __restrict__ pan, const uint2* __restrict__ panb,
              const uint4* __restrict__ item, const uint32_t* __restrict__ prow,
              const uint16_t* __restrict__ em, const uint16_t* __restrict__ tm,
              const uint32_t* __restrict__ pos_of, const uint64_t* __restrict__ in_off,
              uint32_t* __restrict__ live, unsigned long long* __restrict__ tot,
              uint32_t* __restrict__ bar, long long timeout, uint32_t withhold,
              uint32_t* __restrict__ err) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long rows = 0, edges = 0;
  auto level = [&](uint32_t l, uint32_t w, uint32_t warps) {
    for (uint32_t i = lvl[l] + w; i < lvl[l + 1]; i += warps) {
      const uint4 it = item[i];
      const uint32_t p = list[i], k = item_live(it), nu = item_sources(it), r = it.x;
      const uint32_t hi = pan[p].x, e0 = panb[p].x;
      const uint32_t w0 = __ldcg(&live[r >> 5]), w1 = r >= 32 ? __ldcg(&live[(r >> 5) - 1]) : 0u;
      const uint32_t in = __brev(__funnelshift_l(w1, w0, 31 - (r & 31))) & ((1u << k) - 1u);
      const uint32_t feeds = lane < k ? tm[hi - lane] : 0u;
      uint32_t m = in;
      for (uint32_t j = k; j-- > 0;)
        if (__shfl_sync(0xFFFFFFFFu, feeds, j) & m) m |= 1u << j;
      if (!m) continue;
      if ((m >> lane) & 1u) {
        if (!((in >> lane) & 1u)) atomicOr(&live[(r - lane) >> 5], 1u << ((r - lane) & 31));
        const uint32_t q = pos_of[hi - lane];
        ++rows;
        edges += in_off[q + 1] - in_off[q];
      }
      for (uint32_t q = lane; q < nu; q += 32) {
        if (!(em[e0 + q] & m)) continue;
        const uint32_t s = prow[it.w + q], b = 1u << (s & 31);
        if (!(__ldcg(&live[s >> 5]) & b)) atomicOr(&live[s >> 5], b);
      }
    }
  };
  uint32_t n_bar = 0;
  bool ok = true;
  for (uint32_t l = L; ok && l-- > 0;) {
    if (lvl[l + 1] - lvl[l] > LIVE_WARPS) {
      level(l, blockIdx.x * LIVE_WARPS + warp, gridDim.x * LIVE_WARPS);
    } else {
      uint32_t first = l;
      while (first > 0 && lvl[first] - lvl[first - 1] <= LIVE_WARPS) --first;
      if (blockIdx.x == 0)
        for (uint32_t x = l + 1; x-- > first;) {
          level(x, warp, LIVE_WARPS);
          __syncthreads();
        }
      l = first;
    }
    if (!l) break;
    // (test hook: block `withhold` leaves before its first arrival)
    ok = blockIdx.x != withhold && grid_barrier(bar, n_bar++, timeout, err);
  }
  for (int o = 16; o > 0; o >>= 1) {
    rows += __shfl_down_sync(0xFFFFFFFFu, rows, o);
    edges += __shfl_down_sync(0xFFFFFFFFu, edges, o);
  }
  if (lane == 0 && rows) {
    atomicAdd(&tot[0], rows);
    atomicAdd(&tot[1], edges);
  }
}

}  // namespace

// Scratch of the panel schedule builder (per context; sized by the graph).
struct PanelScratch {
  // [W + 1] rank bitmap, [PW + 1] panel bitmap, the count of sources and a
  // cursor over them (zeroed together), rows, level table [levels + 1]
  uint32_t* bits = nullptr;
  uint32_t* pre = nullptr;    // [W + 1] and [PW + 1] bit counts before each word
  uint32_t* bsum = nullptr;
  uint32_t* list = nullptr;   // [panels] opened panels
  // [W + 1] rows that reach a target; two counters, the grid-barrier words, the
  // count's own error bits (COUNT_WORDS together)
  uint32_t* live = nullptr;
  uint32_t* tgt = nullptr;    // uploaded targets
  unsigned long long* h_counts = nullptr;  // page-locked: rows, edges, barrier, error bits
  bool counting = false;      // start_counts has work on the side stream
  uint64_t bytes = 0;         // device memory of the graph-sized arrays and the targets
  uint32_t* h_back = nullptr;  // page-locked: sources, cursor, rows, level table
  size_t cap_tgt = 0;
};

void free_panel_scratch(PanelScratch* s) {
  if (!s) return;
  void* p[] = {s->bits, s->pre, s->bsum, s->list, s->live, s->tgt};
  for (void* q : p)
    if (q) cudaFree(q);
  if (s->h_back) cudaFreeHost(s->h_back);
  if (s->h_counts) cudaFreeHost(s->h_counts);
  delete s;
}

namespace {

// Words of the live bitmap, even: two 64-bit counters lie behind it.
size_t live_words(uint32_t n) { return (((size_t)n + 31) / 32 + 2) & ~(size_t)1; }
constexpr size_t COUNT_WORDS = 8, COUNT_ERR = 6;

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

// The graph-sized scratch of a context, all of it or none.
bf_status make_scratch(Graph* g, Ctx& c) {
  const Panels& P = g->panels;
  const uint32_t W = (g->n + 31) / 32, PW = (P.n + 31) / 32, L = P.n_levels;
  const size_t meta = (size_t)W + PW + 2, nb = (std::max(W, PW) + SCAN_BLOCK - 1) / SCAN_BLOCK;
  PanelScratch* s = new (std::nothrow) PanelScratch();
  if (!s) {
    set_error("out of host memory");
    return BF_ERR_OOM;
  }
  size_t cap[5] = {};
  bf_status rc;
  if ((rc = grow(&s->bits, cap[0], meta + 3 + L + 1, g, false)) ||
      (rc = grow(&s->pre, cap[1], meta, g, false)) ||
      (rc = grow(&s->bsum, cap[2], 2 * nb, g, false)) ||
      (rc = grow(&s->live, cap[3], live_words(g->n) + COUNT_WORDS, g, false)) ||
      (rc = test_fail_alloc("panel_schedule") ? BF_ERR_OOM : BF_OK) ||
      (rc = grow(&s->list, cap[4], P.n, g, false))) {
  } else if (cudaHostAlloc((void**)&s->h_counts, COUNT_WORDS * 4, cudaHostAllocDefault) !=
                 cudaSuccess ||
             cudaHostAlloc((void**)&s->h_back, ((size_t)L + 5) * 4, cudaHostAllocDefault) !=
                 cudaSuccess) {
    cudaGetLastError();
    set_error("cannot allocate the schedule read-back buffers");
    rc = BF_ERR_OOM;
  }
  for (size_t m : cap) s->bytes += m * 4;
  if (rc) {
    g->device_bytes -= s->bytes;
    free_panel_scratch(s);
    return rc;
  }
  c.ps = s;
  return BF_OK;
}

}  // namespace

// Give a context's panel scratch and a schedule's panel items back (the budget
// holds no panel rows: what the item form had before is its again).
void drop_panel_schedule(Graph* g, Ctx& c, Sched& sc) {
  if (c.ps) {
    if (c.ps->counting) cudaStreamSynchronize(c.cnt);
    g->device_bytes -= c.ps->bytes + c.ps->cap_tgt * 4;
    free_panel_scratch(c.ps);
    c.ps = nullptr;
  }
  g->device_bytes -= sc.cap_pitem * sizeof(uint4) + sc.cap_prow * 4;
  if (sc.d_pitem) cudaFree(sc.d_pitem);
  if (sc.d_prow) cudaFree(sc.d_prow);
  sc.d_pitem = nullptr;
  sc.d_prow = nullptr;
  sc.cap_pitem = sc.cap_prow = 0;
  sc.lvl_pan.clear();
}

bf_status start_counts(Graph* g, Ctx& c, Sched& sc, cudaStream_t st) {
  if (!sc.panel) {
    sc.n_live = sc.n_r;
    return BF_OK;
  }
  if (sc.counted) return BF_OK;
  PanelScratch& s = *c.ps;
  const Panels& P = g->panels;
  const uint32_t m = sc.lvl_pan.back();
  uint32_t* lvl = s.bits + ((size_t)g->n + 31) / 32 + (P.n + 31) / 32 + 2 + 3;
  uint32_t* tot = s.live + live_words(g->n);
  if (sc.uses) {  // (a reused schedule: the counters are those of its build)
    BF_CUDA(cudaStreamSynchronize(c.cnt));
    BF_CUDA(cudaMemsetAsync(tot, 0, COUNT_WORDS * 4, st));
  }
  BF_CUDA(cudaEventRecord(c.cnt_fork, st));
  BF_CUDA(cudaStreamWaitEvent(c.cnt, c.cnt_fork, 0));
  const bool hook = test_withhold_arrival();
  const unsigned blocks =
      persistent_blocks(g, (const void*)k_pn_live, LIVE_TPB, m < 8192 ? 16 : 64);
  BF_CUDA(launch_persistent(k_pn_live, blocks, LIVE_TPB, c.cnt, (const uint32_t*)lvl, P.n_levels,
                            (const uint32_t*)s.list, (const uint4*)P.d_a, (const uint2*)P.d_b,
                            (const uint4*)sc.d_pitem, (const uint32_t*)sc.d_prow,
                            (const uint16_t*)P.d_em, (const uint16_t*)P.d_tm,
                            (const uint32_t*)g->d_pos_of, (const uint64_t*)g->d_in_off, s.live,
                            reinterpret_cast<unsigned long long*>(tot), tot + 4,
                            hook ? 2000000ll : BARRIER_TIMEOUT_CYCLES, hook ? 1u : NONE,
                            tot + COUNT_ERR));
  BF_CUDA(cudaMemcpyAsync(s.h_counts, tot, COUNT_WORDS * 4, cudaMemcpyDeviceToHost, c.cnt));
  s.counting = true;
  return BF_OK;
}

bf_status finish_counts(Ctx& c, Sched& sc) {
  if (!c.ps || !c.ps->counting) return BF_OK;
  c.ps->counting = false;
  BF_CUDA(cudaStreamSynchronize(c.cnt));
  // (a count that gave up is partial: the next call counts again)
  if (reinterpret_cast<const uint32_t*>(c.ps->h_counts)[COUNT_ERR]) {
    set_error("a bounded device wait ran out (row counts)");
    return BF_ERR_TIMEOUT;
  }
  sc.n_live = (uint32_t)c.ps->h_counts[0];
  sc.n_edges = c.ps->h_counts[1];
  sc.counted = true;
  return BF_OK;
}

// The panel schedule of h_tgt (host) / d_tgt (the same targets on the device,
// or null). Rows are the targets' ancestors in rank order (a superset of the
// rows that reach a target: 1.28 times as many for 10k targets on the country
// graph, 9 % more gathers; peeling them off first costs a small call more
// than it saves).
bf_status build_schedule_panels(Graph* g, Ctx& c, Sched& sc, const uint32_t* h_tgt,
                                const uint32_t* d_tgt, uint64_t T, uint64_t key, cudaStream_t st) {
  const Panels& P = g->panels;
  const uint32_t n = g->n, W = (n + 31) / 32, L = P.n_levels;
  const uint32_t PW = (P.n + 31) / 32;
  const unsigned nb = (unsigned)((std::max(W, PW) + SCAN_BLOCK - 1) / SCAN_BLOCK);
  const size_t meta = (size_t)W + PW + 2;  // words of the two bitmaps
  bf_status rc;
  if (!c.ps && (rc = make_scratch(g, c))) return rc;
  PanelScratch& s = *c.ps;
  // a count of the schedule before may still run (a call that failed midway)
  if (s.counting) {
    BF_CUDA(cudaStreamSynchronize(c.cnt));
    s.counting = false;
  }
  if ((rc = grow(&sc.d_cidx, sc.cap_cidx, n, g, false)) ||
      (rc = grow(&sc.d_trow, sc.cap_t, T, g, true)))
    return rc;
  if (!d_tgt) {
    if ((rc = grow(&s.tgt, s.cap_tgt, T, g, true))) return rc;
    BF_CUDA(cudaMemcpyAsync(s.tgt, h_tgt, T * 4, cudaMemcpyHostToDevice, st));
    d_tgt = s.tgt;
  }
  uint32_t *rows = s.bits, *pbits = rows + W + 1, *n_src = pbits + PW + 1, *wpre = s.pre;
  const TwoBitmaps bm{{rows, pbits}, {W, PW}, {s.bsum, s.bsum + nb}, {wpre, wpre + W + 1}};
  BF_CUDA(cudaMemsetAsync(s.bits, 0, (meta + 2) * 4, st));
  k_pn_mark<<<(unsigned)((T + 3) / 4), 128, 0, st>>>(d_tgt, (uint32_t)T, g->d_parent, g->d_run_end,
                                                     n, P.d_hibits, P.d_of, P.d_a, rows, pbits,
                                                     n_src, g->d_err);
  k_pn_sums<<<dim3(nb, 2), SCAN_TPB, 0, st>>>(bm);
  k_pn_top<<<2, SCAN_TPB, 0, st>>>(bm);
  k_pn_out<<<dim3(nb, 2), SCAN_TPB, 0, st>>>(bm);
  k_pn_list<<<std::min<uint32_t>((std::max(PW, L + 1) + 255) / 256, 152 * 8), 256, 0, st>>>(
      bm, P.d_lvl, L, s.list, n_src + 3, n_src + 2);
  BF_CUDA(cudaMemcpyAsync(s.h_back, n_src, ((size_t)L + 4) * 4, cudaMemcpyDeviceToHost, st));
  // (the map is not waited for: it runs while the host reads the counts)
  BF_CUDA(cudaEventRecord(c.cnt_fork, st));
  k_pn_cidx<<<std::min<uint32_t>((n + 255) / 256, 152 * 16), 256, 0, st>>>(n, rows, wpre,
                                                                          sc.d_cidx);
  BF_CUDA(cudaGetLastError());
  BF_CUDA(cudaEventSynchronize(c.cnt_fork));
  const uint32_t n_rows = s.h_back[0], n_r = s.h_back[2], *lvl = s.h_back + 3, m = lvl[L];
  if (m > P.n || n_r > n) {
    set_error("panel schedule: inconsistent counts");
    return BF_ERR_DEVICE;
  }
  if ((rc = grow(&sc.d_pitem, sc.cap_pitem, m, g, true)) ||
      (rc = grow(&sc.d_prow, sc.cap_prow, n_rows, g, true)))
    return rc;
  BF_CUDA(cudaMemsetAsync(s.live, 0, (live_words(n) + COUNT_WORDS) * 4, st));
  const uint64_t threads = std::max<uint64_t>((uint64_t)m * 32, T);
  k_pn_items<<<(unsigned)std::min<uint64_t>((threads + 255) / 256, 152 * 32), 256, 0, st>>>(
      s.list, m, P.d_a, P.d_b, P.d_src, rows, wpre, sc.d_cidx, n_src + 1, sc.d_pitem,
      sc.d_prow, d_tgt, T, sc.d_trow, s.live);
  BF_CUDA(cudaGetLastError());
  sc.lvl_pan.assign(lvl, lvl + L + 1);
  sc.panel = true;
  sc.n_r = n_r;
  sc.n_prow = n_rows;
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

template <uint32_t N>
__device__ __forceinline__ void store_lanes(uint32_t* p, const uint32_t (&v)[N]) {
  if constexpr (N == 4)
    *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
  else if constexpr (N == 2)
    *reinterpret_cast<uint2*>(p) = make_uint2(v[0], v[1]);
  else
    *p = v[0];
}

// the same from shared memory
template <uint32_t N>
__device__ __forceinline__ void load_tile(const uint32_t* p, uint32_t (&v)[N]) {
  if constexpr (N == 4) {
    const uint4 x = *reinterpret_cast<const uint4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    v[0] = x.x, v[1] = x.y;
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

// A weight of a tile as relax<SAT>() takes it.
template <bool SAT>
__device__ __forceinline__ uint32_t weight(uint32_t w, uint32_t absent) {
  return SAT && w == absent ? INF : w;
}

// Rows i < j of a panel into row j, in order: tri[i * stride + j] is the weight
// of the edge inside the panel (16-byte loads where the stride allows).
template <uint32_t K, uint32_t N, bool SAT>
__device__ __forceinline__ void solve_triangle(const uint32_t* tri, uint32_t stride,
                                               uint32_t absent, uint32_t (&acc)[K][N]) {
#pragma unroll
  for (uint32_t i = 0; i + 1 < K; ++i) {
    if constexpr (K >= 4) {
#pragma unroll
      for (uint32_t v = (i + 1) / 4; v < K / 4; ++v) {
        const uint4 x = *reinterpret_cast<const uint4*>(tri + i * stride + 4 * v);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          if (4 * v + q > i) {
            const uint32_t wq = weight<SAT>(w[q], absent);
#pragma unroll
            for (uint32_t l = 0; l < N; ++l)
              acc[4 * v + q][l] = relax<SAT>(acc[i][l], wq, acc[4 * v + q][l]);
          }
      }
    } else {
#pragma unroll
      for (uint32_t j = i + 1; j < K; ++j) {
        const uint32_t w = weight<SAT>(tri[i * stride + j], absent);
#pragma unroll
        for (uint32_t l = 0; l < N; ++l) acc[j][l] = relax<SAT>(acc[i][l], w, acc[j][l]);
      }
    }
  }
}

// ---- few lanes or few panels: the warps of a block share a panel's sources --

constexpr uint32_t SPLIT_WARPS = 8;
constexpr uint32_t SPLIT_CH = 256;  // sources staged at a time

template <uint32_t LPT>
struct SplitSmem {
  uint32_t w[SPLIT_CH * PANEL_ROWS];
  uint32_t tri[PANEL_ROWS * PANEL_ROWS];
  uint32_t row[SPLIT_CH];
  uint32_t red[PANEL_ROWS * 32 * LPT];
};

template <uint32_t K, uint32_t LPT, bool SAT>
__device__ __forceinline__ void split_item(const uint4 a, const uint32_t* __restrict__ prow,
                                           const uint32_t* __restrict__ pw, uint32_t absent,
                                           uint32_t* __restrict__ slab, uint32_t Kp,
                                           const uint32_t* __restrict__ seeded,
                                           SplitSmem<LPT>& sm) {
  constexpr uint32_t FARV = SAT ? INF : FAR + 1;
  constexpr uint32_t LANES = 32 * LPT, TPB = 32 * SPLIT_WARPS;
  const uint32_t t = threadIdx.x, warp = t >> 5;
  const uint32_t live = item_live(a), stride = item_stride(a), nu = item_sources(a);
  const uint32_t lane0 = blockIdx.y * LANES, lane = lane0 + (t & 31) * LPT;
  const bool on = lane < Kp;
  auto stage = [&](uint32_t c0, uint32_t m) {
    for (uint32_t i = t; i < m; i += TPB) sm.row[i] = prow[a.w + c0 + i];
    for (uint32_t i = t; i < m * K; i += TPB)
      sm.w[i] = weight<SAT>(pw[a.z + (size_t)(c0 + i / K) * stride + i % K], absent);
  };
  // all of this is static: staged before the previous level is done
  stage(0, min(nu, SPLIT_CH));
  const uint32_t* tri = pw + a.z + (size_t)nu * stride;
  for (uint32_t i = t; i < K * K; i += TPB)
    sm.tri[i] = tri[(i / K) * stride + i % K];
  // (seeds too: they are written before the first level is launched)
  for (uint32_t i = t; i < K * LANES; i += TPB) {
    const uint32_t j = i / LANES, x = lane0 + i % LANES, r = a.x - j;
    sm.red[i] = j < live && x < Kp && ((seeded[r >> 5] >> (r & 31)) & 1u)
                    ? __ldcg(slab + (size_t)r * Kp + x) : FARV;
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t acc[K][LPT];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j)
#pragma unroll
    for (uint32_t l = 0; l < LPT; ++l) acc[j][l] = FARV;
  for (uint32_t c0 = 0; c0 < nu; c0 += SPLIT_CH) {
    const uint32_t m = min(nu - c0, SPLIT_CH);
    if (c0) {
      __syncthreads();
      stage(c0, m);
      __syncthreads();
    }
    if (on) {
      constexpr uint32_t U = 16 / LPT;  // source rows in flight per thread
      for (uint32_t s0 = warp; s0 < m; s0 += U * SPLIT_WARPS) {
        uint32_t d[U][LPT];
#pragma unroll
        for (uint32_t q = 0; q < U; ++q) {
          const uint32_t s = s0 + q * SPLIT_WARPS;
          if (s < m) load_lanes<LPT>(slab + (size_t)sm.row[s] * Kp + lane, d[q]);
        }
#pragma unroll
        for (uint32_t q = 0; q < U; ++q) {
          const uint32_t s = s0 + q * SPLIT_WARPS;
          if (s >= m) break;
          uint32_t w[K];
          load_weights<K>(sm.w + s * K, w);
#pragma unroll
          for (uint32_t l = 0; l < LPT; ++l)
#pragma unroll
            for (uint32_t j = 0; j < K; ++j) acc[j][l] = relax<SAT>(d[q][l], w[j], acc[j][l]);
        }
      }
    }
  }
  // the warps hold minima over different sources: combine them, then a thread
  // per lane solves the triangle
  if (on) {
#pragma unroll
    for (uint32_t j = 0; j < K; ++j)
#pragma unroll
      for (uint32_t l = 0; l < LPT; ++l)
        if (acc[j][l] < FARV) atomicMin(&sm.red[j * LANES + (t & 31) * LPT + l], acc[j][l]);
  }
  __syncthreads();
  const uint32_t x = lane0 + t;
  if (t >= LANES || x >= Kp) return;
  uint32_t v[K][1];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j) v[j][0] = sm.red[j * LANES + t];
  solve_triangle<K, 1, SAT>(sm.tri, K, absent, v);
#pragma unroll
  for (uint32_t j = 0; j < K; ++j)
    if (j < live) slab[(size_t)(a.x - j) * Kp + x] = v[j][0];
}

// One level of panels: blockIdx.x = item, blockIdx.y = block of 32 * LPT lanes.
// Bound by the chain of dependent levels, 3 us each: what it must still do once
// the level before it is done is one round of row loads, the combination and
// the triangle; everything else, seeds too, is staged before. Against the item
// sweep (a level of rows, a gather per edge), sweep time: 37 x 421 on the
// 1000 x 1250 region 1.69 -> 0.16 ms, 100 x 100 on grid100 1.59 -> 0.14 ms; with
// four rows in flight per thread, seeds read at the end and 128 lanes a block
// for any level 0.25 and 0.28.
template <uint32_t LPT, bool SAT>
__global__ void __launch_bounds__(32 * SPLIT_WARPS)
    k_sweep_panels(const uint4* __restrict__ item, uint32_t i0, const uint32_t* __restrict__ prow,
                   const uint32_t* __restrict__ pw, uint32_t absent,
                   uint32_t* __restrict__ slab, uint32_t Kp, const uint32_t* __restrict__ seeded) {
  __shared__ __align__(16) SplitSmem<LPT> sm;
  asm volatile("griddepcontrol.launch_dependents;");
  const uint4 a = item[i0 + blockIdx.x];
  const uint32_t live = item_live(a);
#define BF_PANEL(K) split_item<K, LPT, SAT>(a, prow, pw, absent, slab, Kp, seeded, sm)
  if (live > 12) BF_PANEL(16);
  else if (live > 8) BF_PANEL(12);
  else if (live > 4) BF_PANEL(8);
  else if (live > 2) BF_PANEL(4);
  else if (live == 2) BF_PANEL(2);
  else BF_PANEL(1);
#undef BF_PANEL
}

// ---- many lanes: source rows through a ring of bulk copies ------------------

constexpr uint32_t RING = 4;         // groups of rows in flight per block
constexpr uint32_t GROUP = 8;        // rows of a group (half of a panel's)
constexpr uint32_t RING_WARPS = 8;   // consumer warps
constexpr uint32_t RING_LPT = 2;     // lanes of a consumer thread
constexpr uint32_t RING_TILE = RING_WARPS * 32 * RING_LPT;  // lanes of a row in a group
constexpr uint32_t RING_POLLS = 1u << 22;                   // bound on a wait

struct RingSmem {
  uint32_t row[RING][GROUP][RING_TILE];
  uint32_t w[RING][GROUP][PANEL_ROWS];             // the sources' weights
  uint32_t tri[RING][PANEL_ROWS * PANEL_ROWS];     // with a unit's last group
  uint4 meta[RING];                                // with a unit's first group
  uint64_t full[RING], empty[RING];
  int abort;
};

__device__ __forceinline__ uint32_t sm_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sm_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sm_addr(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_addr(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(sm_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Wait for a phase, bounded: past the limit, or once another warp gave up, the
// block is abandoned (false).
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, int* abort, uint32_t* err) {
  if (bar_try(b, parity)) return true;
  for (uint32_t i = 0; i < RING_POLLS; ++i) {
    if (bar_try(b, parity)) return true;
    if (*(volatile int*)abort) return false;
  }
  *(volatile int*)abort = 1;
  atomicOr(err, DEVERR_TIMEOUT);
  return false;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          sm_addr(dst)),
      "l"(src), "r"(bytes), "r"(sm_addr(bar))
      : "memory");
}

// A consumer thread's view of the ring: group `at`, phase bit of its pass.
struct RingPos {
  uint32_t at = 0, phase = 0;
  __device__ __forceinline__ void next() {
    if (++at == RING) {
      at = 0;
      phase ^= 1u;
    }
  }
};

// One unit (a panel, a tile of lanes) for this thread's lanes: its groups in
// order - the seeds of rows 0 to 7, those of rows 8 to 15, the sources, each
// if there are any - and the triangle, which comes with the last. The first
// group has been waited for. False: the block is abandoned.
template <uint32_t K, bool SAT>
__device__ __forceinline__ bool ring_unit(const uint4 m, RingSmem& sm, RingPos& p,
                                          uint32_t absent, uint32_t* __restrict__ slab,
                                          uint32_t Kp, uint32_t lane, uint32_t* err) {
  constexpr uint32_t FARV = SAT ? INF : FAR + 1, N = RING_LPT;
  const uint32_t tl = threadIdx.x * N;
  const uint32_t live = item_live(m), stride = item_stride(m), nu = item_sources(m), seeds = m.z;
  auto release = [&]() {  // this warp is done with the current group
    __syncwarp();
    if ((threadIdx.x & 31) == 0) bar_arrive(&sm.empty[p.at]);
    p.next();
  };
  auto next = [&]() {
    release();
    return bar_wait(&sm.full[p.at], p.phase, &sm.abort, err);
  };
  uint32_t acc[K][N];
#pragma unroll
  for (uint32_t j = 0; j < K; ++j)
#pragma unroll
    for (uint32_t l = 0; l < N; ++l) acc[j][l] = FARV;
#pragma unroll
  for (uint32_t j0 = 0; j0 < K; j0 += GROUP) {
    const uint32_t in = seeds >> j0 & ((1u << GROUP) - 1);
    if (!in) continue;
    const uint32_t* row = &sm.row[p.at][0][tl];
#pragma unroll
    for (uint32_t j = j0; j < j0 + GROUP && j < K; ++j)
      if ((seeds >> j) & 1u) {
        load_tile<N>(row, acc[j]);
        row += RING_TILE;
      }
    if ((nu || seeds >> j0 >> GROUP) && !next()) return false;
  }
  for (uint32_t s0 = 0; s0 < nu;) {
    const uint32_t* row = &sm.row[p.at][0][tl];
    const uint32_t* wt = sm.w[p.at][0];
#pragma unroll
    for (uint32_t q = 0; q < GROUP; ++q) {
      if (s0 + q >= nu) break;
      uint32_t x[N], w[K];
      load_tile<N>(row + q * RING_TILE, x);
      load_weights<K>(wt + q * PANEL_ROWS, w);
#pragma unroll
      for (uint32_t j = 0; j < K; ++j) {
        const uint32_t wj = weight<SAT>(w[j], absent);
#pragma unroll
        for (uint32_t l = 0; l < N; ++l) acc[j][l] = relax<SAT>(x[l], wj, acc[j][l]);
      }
    }
    s0 += GROUP;
    if (s0 >= nu) break;
    if (!next()) return false;
  }
  if constexpr (K > 1) solve_triangle<K, N, SAT>(sm.tri[p.at], stride, absent, acc);
  release();
  if (lane < Kp) {
    uint32_t* row = slab + (size_t)m.x * Kp + lane;
#pragma unroll
    for (uint32_t j = 0; j < K; ++j) {
      if (j >= live) break;
      store_lanes<N>(row, acc[j]);
      row -= Kp;
    }
  }
  return true;
}

// One level of panels for many lanes: blocks walk the level's units (panel,
// 512 lanes). A producer warp keeps a ring of four groups of eight row tiles
// (2 KB each) in flight by bulk copies, across unit boundaries, and eight warps
// consume them; the loads take no registers of the threads that hold the
// labels, and a warp's work per row is one 8-byte shared load, the weights and
// the add-mins. Bound by the integer pipe (an add-min per weight and lane, 64 a
// cycle and SM: 4.9 ms for 10k x 10k on the country graph) and HBM (37 GB, 5.4
// ms: 32 GB of source rows and rows written, the rest seeded rows read back)
// together; a level of 4347 panels at 4000 lanes ran at 57 % of the first and 60 %
// of the second. 10k x 10k sweep 14.4 -> 9.5 ms against a thread that loads its
// own rows into registers; measured on the way: four warps of four lanes a thread
// 11.3 ms (code for 64 labels misses the instruction cache), groups of four rows
// 11.0, seeds as sources with one-hot weights 10.4, scalar loads of the triangle
// 10.0.
template <bool SAT>
__global__ void __launch_bounds__(32 * (RING_WARPS + 1), 3)
    k_sweep_panels_ring(const uint4* __restrict__ item, uint32_t i0, uint32_t n_item,
                        uint32_t tiles, const uint32_t* __restrict__ prow,
                        const uint32_t* __restrict__ pw, uint32_t absent, uint32_t* __restrict__ slab,
                        uint32_t Kp, const uint32_t* __restrict__ seeded,
                        uint32_t* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char ring_smem[];
  RingSmem& sm = *reinterpret_cast<RingSmem*>(ring_smem);
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t warp = threadIdx.x >> 5, wl = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (uint32_t i = 0; i < RING; ++i) {
      bar_init(&sm.full[i], 1);
      bar_init(&sm.empty[i], RING_WARPS);
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const uint32_t units = n_item * tiles;
  if (warp < RING_WARPS) {
    // (the bounded ring waits below then only wait for this block's producer)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    RingPos p;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
      if (!bar_wait(&sm.full[p.at], p.phase, &sm.abort, err)) return;
      const uint4 m = sm.meta[p.at];
      const uint32_t lane = m.w + threadIdx.x * RING_LPT, live = item_live(m);
      bool ok;
#define BF_UNIT(K) ok = ring_unit<K, SAT>(m, sm, p, absent, slab, Kp, lane, err)
      if (live > 12) BF_UNIT(16);
      else if (live > 8) BF_UNIT(12);
      else if (live > 4) BF_UNIT(8);
      else if (live > 2) BF_UNIT(4);
      else if (live == 2) BF_UNIT(2);
      else BF_UNIT(1);
#undef BF_UNIT
      if (!ok) return;
    }
    return;
  }
  // producer: what a unit needs before its copies can start is loaded while
  // earlier units are filled: the item two units ahead, the words of its
  // seeded bits and its first 32 source rows one unit ahead
  struct Ahead {
    uint32_t s0, s1, row;
  };
  auto item_of = [&](uint32_t x) {
    return x < units ? item[i0 + x / tiles] : make_uint4(0, 0, 0, 0);
  };
  auto ahead_of = [&](const uint4& it) {
    Ahead h;
    h.s0 = seeded[it.x >> 5];
    h.s1 = it.x >= 32 ? seeded[(it.x >> 5) - 1] : 0u;
    h.row = wl < item_sources(it) ? prow[it.w + wl] : 0u;
    return h;
  };
  uint32_t head = 0;  // groups filled so far
  uint32_t u = blockIdx.x;
  uint4 a = item_of(u), na = item_of(u + gridDim.x);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");
  Ahead h = ahead_of(a);
  bool ok = true;
  for (; ok && u < units; u += gridDim.x) {
    const uint4 nna = item_of(u + 2 * gridDim.x);
    const Ahead nh = ahead_of(na);
    const uint32_t live = item_live(a), stride = item_stride(a);
    const uint32_t lane0 = (u % tiles) * RING_TILE;
    const uint32_t bytes = min(RING_TILE, Kp - lane0) * 4;
    // the panel's rows with seeds (bit j: row j, which is j rows below row a.x)
    const uint32_t seeds = __brev(__funnelshift_l(h.s1, h.s0, 31 - (a.x & 31))) &
                           ((1u << live) - 1u);
    const uint32_t nu = item_sources(a), low = seeds & ((1u << GROUP) - 1);
    const uint32_t gs = (low ? 1u : 0u) + (seeds >> GROUP ? 1u : 0u);  // seed groups
    const uint32_t ng = max(1u, gs + (nu + GROUP - 1) / GROUP);
    uint32_t row = h.row, chunk = 0;  // slab rows of 32 sources, from `chunk`
    for (uint32_t gi = 0; gi < ng; ++gi) {
      const uint32_t slot = head % RING, pass = head / RING;
      const bool seed = gi < gs;
      // a seed group's rows: bits of `in`, from row j0 of the panel
      const uint32_t j0 = seed && !(gi == 0 && low) ? GROUP : 0u;
      const uint32_t in = j0 ? seeds >> GROUP : low;
      const uint32_t s0 = seed ? 0u : (gi - gs) * GROUP;
      const uint32_t cnt = seed ? __popc(in) : min(GROUP, nu - s0);
      const uint32_t tri = gi + 1 == ng && live > 1 ? stride * stride * 4 : 0u;
      if (s0 - chunk == 32) {
        chunk = s0;
        row = s0 + wl < nu ? prow[a.w + s0 + wl] : 0u;
      }
      uint32_t src = __shfl_sync(0xFFFFFFFFu, row, (s0 - chunk + wl) & 31);
      if (seed && wl < cnt) src = a.x - j0 - __fns(in, 0, (int)wl + 1);
      uint64_t* full = &sm.full[slot];
      bool free = true;
      if (wl == 0) {
        free = bar_wait(&sm.empty[slot], (pass & 1u) ^ 1u, &sm.abort, err);
        if (free) {
          if (gi == 0) sm.meta[slot] = make_uint4(a.x, a.y, seeds, lane0);
          const uint32_t tx = cnt * (bytes + (seed ? 0u : stride * 4)) + tri;
          if (tx)
            bar_expect(full, tx);
          else
            bar_arrive(full);
        }
      }
      ok = __shfl_sync(0xFFFFFFFFu, free, 0);
      if (!ok) break;
      if (wl < cnt) {
        if (!seed)
          bulk_load(sm.w[slot][wl], pw + a.z + (size_t)(s0 + wl) * stride, stride * 4, full);
        bulk_load(sm.row[slot][wl], slab + (size_t)src * Kp + lane0, bytes, full);
      } else if (wl == GROUP && tri) {
        bulk_load(sm.tri[slot], pw + a.z + (size_t)nu * stride, tri, full);
      }
      ++head;
    }
    a = na;
    na = nna;
    h = nh;
  }
  // abandoned: no copy may still be writing this block's shared memory when
  // it exits, so wait (bounded) for the groups filled last
  if (!ok && wl < RING && head > wl) {
    const uint32_t q = head - 1 - wl;
    for (uint32_t i = 0; i < RING_POLLS && !bar_try(&sm.full[q % RING], (q / RING) & 1u); ++i) {
    }
  }
}

// Units per SM from which a wave of 68 to 128 lanes takes the ring form.
constexpr uint64_t RING_NARROW = 8;

template <bool SAT>
cudaError_t launch_panels(const Graph* g, const Sched& sc, uint32_t i0, uint32_t m, uint32_t* slab,
                          uint32_t Kp, const uint32_t* seeded, bool pdl, cudaStream_t st) {
  const Panels& P = g->panels;
  const uint32_t tiles = (Kp + RING_TILE - 1) / RING_TILE;
  // A thread of the ring form walks all sources of its panel (up to a few
  // hundred at the top of the tree): with few units in a level that chain is
  // the level's time, so the split form takes levels of fewer than two units
  // per SM (fewer than eight at up to 128 lanes, whose tile is mostly empty; at
  // up to 64 it wins in any level). 100 sources: to 10,000 ends on the country
  // graph 1.29 ms against 1.49 by the split form alone, to 5000 on the region
  // 0.60 against 0.68, on grid100 0.38 either way (0.40 from two units).
  const uint64_t units = (uint64_t)m * tiles;
  const uint64_t enough = (Kp > 128 ? 2ull : RING_NARROW) * g->sm_count;
  if (units >= enough && units < 0x80000000ull && Kp > 64) {
    const uint32_t grid = std::min<uint32_t>(m * tiles, 3 * g->sm_count);
    return launch_level_smem(k_sweep_panels_ring<SAT>, dim3(grid), 32 * (RING_WARPS + 1),
                             sizeof(RingSmem), pdl, st, (const uint4*)sc.d_pitem, i0, m, tiles, (const uint32_t*)sc.d_prow,
                        (const uint32_t*)P.d_w, P.absent, slab, Kp, seeded, g->d_err);
  }
  auto go = [&](auto kern, uint32_t lanes) {
    return launch_level(kern, dim3(m, (Kp + lanes - 1) / lanes), 32 * SPLIT_WARPS, pdl, st,
                        (const uint4*)sc.d_pitem, i0, (const uint32_t*)sc.d_prow,
                        (const uint32_t*)P.d_w, P.absent, slab, Kp, seeded);
  };
  // lanes a block: as many as still give two blocks an SM (fewer lanes a thread
  // keep more rows in flight), else 32. 100 lanes on grid100, whole call: 344 us
  // against 420 with 128 lanes a block
  const uint64_t few = 2ull * g->sm_count;
  if (Kp <= 32 || m * (uint64_t)((Kp + 63) / 64) < few) return go(k_sweep_panels<1, SAT>, 32);
  if (Kp <= 64 || m * (uint64_t)((Kp + 127) / 128) < few) return go(k_sweep_panels<2, SAT>, 64);
  return go(k_sweep_panels<4, SAT>, 128);
}

}  // namespace

// The ring form's shared memory on the current device (at graph creation).
bf_status panel_kernels_init() {
  BF_CUDA(cudaFuncSetAttribute(k_sweep_panels_ring<false>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(RingSmem)));
  BF_CUDA(cudaFuncSetAttribute(k_sweep_panels_ring<true>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(RingSmem)));
  return BF_OK;
}

// Whether a sweep from seed costs of at most max_seed may hold finite labels
// beyond the one-instruction relaxation's range.
bool panels_saturate(const Graph* g, uint64_t max_seed) {
  return g->panels.max_label + max_seed >= FAR;
}

// What a lane without a seed holds in the rows that a panel sweep reads.
uint32_t panel_fill(const Graph* g, uint64_t max_seed) {
  return panels_saturate(g, max_seed) ? INF : FAR + 1;
}

// The least label that means "unreachable" in the rows that a sweep from seed
// costs of at most max_seed leaves.
uint32_t unreachable_from(const Graph* g, const Sched& sc, uint64_t max_seed) {
  return sc.panel && !panels_saturate(g, max_seed) ? FAR : INF;
}

// The level launches of a panel schedule on `st`. sat: labels may pass the
// range of the one-instruction relaxation (seed costs, or the graph's own
// longest paths).
cudaError_t sweep_panels(Graph* g, Sched& sc, uint32_t* slab, uint32_t Kp, bool sat,
                         cudaStream_t st, uint64_t* launches, const uint32_t* seeded) {
  // the first level waits for what ran before it, so that every level may read
  // the seeds while the level before it drains
  bool pdl = false;
  for (uint32_t l = 0; l + 1 < sc.lvl_pan.size(); ++l) {
    const uint32_t i0 = sc.lvl_pan[l], m = sc.lvl_pan[l + 1] - i0;
    if (!m) continue;
    const cudaError_t e = sat ? launch_panels<true>(g, sc, i0, m, slab, Kp, seeded, pdl, st)
                              : launch_panels<false>(g, sc, i0, m, slab, Kp, seeded, pdl, st);
    if (e != cudaSuccess) return e;
    pdl = g->tune.pdl != 0;
    ++*launches;
  }
  return cudaSuccess;
}

}  // namespace bf
