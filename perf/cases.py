"""What users of the engine have it do, as cases that can be timed.

Every case goes through the public Python entry points of bfphast on seeded
synthetic road graphs of the repository's own families. A graph is built and
loaded once per process and kept, as a routing service keeps it; a state holds
the inputs of one request (new for every seed) and the output buffers that
such a caller owns.

  graph     lattice               CCH ranks
  grid100   100 x 100 grid           35 724
  town      200 x 250 country       119 249
  district  500 x 600 country       715 293
  region    1000 x 1250 country   2 983 382
  country   2000 x 2500 country  11 936 709

Durations are deciseconds: 30 minutes are 18 000.
"""
import pathlib
import sys

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "butterfly-osm_gb300"))

import bfphast  # noqa: E402
import cchbuild  # noqa: E402
import workload  # noqa: E402

INF = bfphast.INF

# kind, rows, cols, CCH ranks, finite UP edges (DOWN: as many within a percent)
GRAPHS = {
    "grid100": (cchbuild.KIND_GRID, 100, 100, 35724, 648864),
    "town": (cchbuild.KIND_COUNTRY, 200, 250, 119249, 369762),
    "district": (cchbuild.KIND_COUNTRY, 500, 600, 715293, 2254797),
    "region": (cchbuild.KIND_COUNTRY, 1000, 1250, 2983382, 9582325),
    "country": (cchbuild.KIND_COUNTRY, 2000, 2500, 11936709, 38900000),
}


def listed():
    return [
        # the smallest table a client asks for, on a small graph: latency and
        # launches are all of it (the repository's first configuration)
        {"name": "grid_matrix", "kind": "matrix", "graph": "grid100", "S": 100, "T": 100,
         "threshold": INF},
        # one-to-all distances of a batch of sources, every node returned
        {"name": "town_one_to_all", "kind": "one_to_all", "graph": "town", "S": 29},
        # a table request as the serving mix draws them (10 to 5000 a side)
        {"name": "region_request", "kind": "matrix", "graph": "region", "S": 37, "T": 421,
         "threshold": INF},
        # a planner's table on the device, cells above 30 minutes cut off
        {"name": "region_bounded", "kind": "matrix_device", "graph": "region", "S": 1000,
         "T": 1500, "threshold": 18000},
        # the headline: a national 10k x 10k table on the device, new targets
        {"name": "country_matrix", "kind": "matrix_device", "graph": "country", "S": 10000,
         "T": 10000, "threshold": INF},
        # bulk reachability sets on the device: a full wave and a ragged one,
        # thresholds from 5 minutes to an hour
        {"name": "country_isochrones", "kind": "isochrones_device", "graph": "country", "S": 1500},
        # a handful of isochrones for one page of a map, host buffers
        {"name": "region_isochrones", "kind": "isochrones", "graph": "region", "S": 5},
        # isochrone outlines drawn on a map, 30 minutes by car
        {"name": "region_polygons", "kind": "polygons", "graph": "region", "S": 24,
         "threshold_s": 1800},
        # durations and lengths between points snapped onto roads: each end
        # has one to three candidate states with an offset
        {"name": "region_phantoms", "kind": "phantoms", "graph": "region", "S": 60, "T": 90,
         "threshold": INF},
        # new weights for every road (a traffic update): the weights and
        # middles of the whole hierarchy
        {"name": "region_customize", "kind": "customize", "graph": "region"},
        # a table with lengths as record batch columns, every cell, odd widths
        {"name": "tile_dense", "kind": "tile", "S": 5003, "T": 4001, "sparse": False,
         "lengths": True, "threshold": INF, "keep": 1.0},
        # the 10k x 10k table as columns: destinations within a radius only,
        # 30 minutes at most, cells beyond dropped
        {"name": "tile_sparse", "kind": "tile", "S": 10000, "T": 10000, "sparse": True,
         "lengths": False, "threshold": 18000, "keep": 0.2},
    ]


def _log(rng, lo, hi):
    """A whole number, uniform over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["matrix", "one_to_all", "matrix_device", "isochrones_device", "isochrones",
                       "polygons", "phantoms", "customize", "tile"])
    small = ["grid100", "town", "district", "region"]
    if kind == "matrix":
        return {"kind": kind, "graph": rng.choice(small), "S": _log(rng, 1, 2000),
                "T": _log(rng, 1, 5000), "threshold": rng.choice([INF, INF, 6000, 36000])}
    if kind == "one_to_all":
        g = rng.choice(small)
        return {"kind": kind, "graph": g, "S": _log(rng, 1, 8 if g == "region" else 64)}
    if kind == "matrix_device":
        return {"kind": kind, "graph": rng.choice(["district", "region", "country"]),
                "S": _log(rng, 100, 10000), "T": _log(rng, 100, 10000),
                "threshold": rng.choice([INF, INF, 9000, 18000])}
    if kind == "isochrones_device":
        return {"kind": kind, "graph": rng.choice(["district", "region", "country"]),
                "S": _log(rng, 64, 1500)}
    if kind == "isochrones":
        return {"kind": kind, "graph": rng.choice(small), "S": _log(rng, 1, 64)}
    if kind == "polygons":
        return {"kind": kind, "graph": rng.choice(["district", "region"]), "S": _log(rng, 1, 64),
                "threshold_s": rng.choice([300, 900, 1800, 3600])}
    if kind == "phantoms":
        return {"kind": kind, "graph": rng.choice(["town", "district", "region"]),
                "S": _log(rng, 1, 200), "T": _log(rng, 1, 300),
                "threshold": rng.choice([INF, 18000])}
    if kind == "customize":
        return {"kind": kind, "graph": "district" if rng.random() < 0.4 else
                rng.choice(["town", "region"])}
    sparse = rng.random() < 0.5
    return {"kind": "tile", "S": _log(rng, 50, 10000), "T": _log(rng, 50, 10000),
            "sparse": sparse, "lengths": rng.random() < 0.5,
            "threshold": 18000 if sparse else rng.choice([INF, 18000]),
            "keep": rng.choice([1.0, 0.2, 0.5])}


# ---- what a service keeps: graphs, topologies, road geometry ----------------

_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _fixture(name):
    kind, rows, cols = GRAPHS[name][:3]
    return _keep(("fixture", name), lambda: cchbuild.build_synthetic(
        kind, rows, cols, seed=42, with_topo=name != "country"))


def _graph(name):
    return _keep(("graph", name), lambda: bfphast.Graph.from_cch(_fixture(name)[1]))


def _graph_2ch(name):
    """The graph with a length on every edge (metres that vary by road)."""
    def make():
        cch = _fixture(name)[1]
        ln = []
        for key in ("up_w", "down_w"):
            w = cch[key]
            f = np.random.default_rng(9).integers(5, 34, len(w)).astype(np.uint32)
            ln.append(np.where(w == INF, np.uint32(INF), w * f // np.uint32(10)))
        return bfphast.Graph.from_cch(cch, up_len=ln[0], down_len=ln[1])
    return _keep(("graph2", name), make)


def _geometry(name):
    """A straight road from tail to head per rank, lattice coordinates."""
    def make():
        ebg, cch = _fixture(name)
        cols = GRAPHS[name][2]
        r2s = cch["rank_to_state"]
        ii = np.arange(ebg["n_intersections"], dtype=np.int64)
        lat = (500_000_000 + (ii // cols) * 9000).astype(np.int32)
        lon = (30_000_000 + (ii % cols) * 14000).astype(np.int32)
        tail, head = ebg["state_tail"][r2s], ebg["state_head"][r2s]
        pts = np.stack([lat[tail], lon[tail], lat[head], lon[head]], 1).reshape(-1, 2)
        return bfphast.Geometry(np.arange(0, 2 * len(r2s) + 1, 2, dtype=np.uint64), pts,
                                ebg["node_weight"][r2s])
    return _keep(("geometry", name), make)


def _topology(name):
    """(Cch, original UP weights, original DOWN weights) of the whole hierarchy."""
    def make():
        u = _fixture(name)[1]["topo"]
        n = len(u["off"]) - 1
        tgt = torch.from_numpy(u["tgt"].astype(np.int64)).cuda()
        order = torch.sort(tgt, stable=True).indices.cpu().numpy()
        src = np.repeat(np.arange(n, dtype=np.uint32), np.diff(u["off"].astype(np.int64)))
        off = np.zeros(n + 1, np.uint64)
        off[1:] = np.cumsum(np.bincount(u["tgt"], minlength=n))
        cch = bfphast.Cch(n, u["off"], u["tgt"], off, src[order])
        return cch, u["orig_up"], u["orig_down"][order]
    return _keep(("topology", name), make)


# ---- one request ------------------------------------------------------------

def _pinned(n):
    return torch.empty(n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)


def _dev(a):
    return torch.from_numpy(a.view(np.int32)).cuda()


def _ids(rng, n, count):
    return rng.integers(0, n, count).astype(np.uint32)


def _seeds(rng, n, count):
    """Candidate states of snapped points: (rank, offset time, offset length)."""
    out = []
    for _ in range(count):
        k = int(rng.integers(1, 4))
        out.append([(int(rng.integers(0, n)), int(rng.integers(0, 120)),
                     int(rng.integers(0, 400))) for _ in range(k)])
    return out


def _thresholds(rng, count):
    return rng.choice(np.asarray(workload.ISO_THRESHOLDS_S, np.uint32) * 10, count).astype(np.uint32)


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "tile":
        S, T = case["S"], case["T"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        dur = torch.empty(S * T, device="cuda").log_normal_(11.4, 0.8, generator=g)
        dur = dur.clamp_(max=2e6).to(torch.int32)
        dur[torch.rand(S * T, device="cuda", generator=g) < 0.002] = -1  # unreachable
        st.update(S=S, T=T, dur=dur, sparse=case["sparse"], threshold=case["threshold"],
                  src=torch.randperm(S, device="cuda", generator=g).to(torch.int32),
                  dst=torch.randperm(T, device="cuda", generator=g).to(torch.int32), len=None,
                  cols=[torch.zeros(S * T, dtype=torch.int32, device="cuda") for _ in range(4)],
                  off=None, mask=None)
        if case["lengths"]:
            st["len"] = torch.where(dur == -1, dur, dur // 3)
        if case["keep"] < 1.0:  # the destinations within each source's radius, by index
            near = torch.rand(S, T, device="cuda", generator=g) < case["keep"]
            st["off"] = torch.zeros(S + 1, dtype=torch.int64, device="cuda")
            st["off"][1:] = near.sum(1).cumsum(0)
            st["mask"] = near.nonzero()[:, 1].to(torch.int32)
        return st
    name = case["graph"]
    n = GRAPHS[name][3]
    if kind == "customize":
        cch, up, down = _topology(name)
        st.update(cch=cch, up=_pinned(len(up)), down=_pinned(len(down)),
                  out=[_pinned(len(x)) for x in (up, down, up, down)])
        for src, dst in ((up, st["up"]), (down, st["down"])):  # 70 % to 150 % of the free flow
            f = torch.randint(70, 151, (len(src),), generator=torch.Generator().manual_seed(seed))
            w = torch.from_numpy(src.astype(np.int64))
            dst[:] = torch.where(w == INF, w, w * f // 100 + 1).numpy().astype(np.uint32)
        return st
    if kind == "phantoms":
        st.update(graph=_graph_2ch(name), src=_seeds(rng, n, case["S"]),
                  tgt=_seeds(rng, n, case["T"]), threshold=case["threshold"])
        return st
    st.update(graph=_graph(name), src=_ids(rng, n, case["S"]))
    if kind in ("matrix", "matrix_device"):
        st.update(tgt=_ids(rng, n, case["T"]), threshold=case["threshold"])
    if kind == "matrix_device":
        st.update(d_src=_dev(st["src"]), d_tgt=_dev(st["tgt"]),
                  out=torch.empty(case["S"], case["T"], dtype=torch.int32, device="cuda"))
    if kind in ("isochrones", "isochrones_device"):
        st["thr"] = _thresholds(rng, case["S"])
    if kind == "isochrones_device":
        st.update(d_src=_dev(st["src"]), d_thr=_dev(st["thr"]),
                  bits=torch.empty(case["S"], (n + 63) // 64, dtype=torch.int64, device="cuda"),
                  counts=torch.empty(case["S"], dtype=torch.int64, device="cuda"))
    if kind == "polygons":
        s = case["threshold_s"]
        st.update(geometry=_geometry(name), thr=np.full(case["S"], 10 * s, np.uint32),
                  tier=np.full(case["S"], s, np.uint32),
                  rings=np.zeros((8192 * max(8, case["S"]), 2)))
    return st


def _whole(a):
    """Unsigned results as signed ones of the same bytes."""
    return a.view(np.int32 if a.dtype == np.uint32 else np.int64)


def run(st):
    kind = st["kind"]
    if kind == "matrix":
        return _whole(st["graph"].matrix(st["src"], st["tgt"], st["threshold"]))
    if kind == "one_to_all":
        return _whole(st["graph"].query_batch(st["src"]))
    if kind == "matrix_device":
        st["graph"].matrix_device(st["d_src"].data_ptr(), len(st["src"]), st["d_tgt"].data_ptr(),
                                  len(st["tgt"]), st["out"].data_ptr(), st["threshold"],
                                  torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if kind == "isochrones_device":
        st["graph"].isochrone_bitsets_device(
            st["d_src"].data_ptr(), st["d_thr"].data_ptr(), len(st["src"]), st["bits"].data_ptr(),
            st["counts"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return [st["bits"], st["counts"]]
    if kind == "isochrones":
        return [_whole(a) for a in st["graph"].isochrone_bitsets(st["src"], st["thr"])]
    if kind == "polygons":
        rings, _ = bfphast.isochrone_polygons(st["graph"], st["geometry"], st["src"], st["thr"],
                                              st["tier"])
        sizes = np.array([len(r) for r in rings])
        np.concatenate(rings, out=st["rings"][:sizes.sum()])
        return [st["rings"], sizes]
    if kind == "phantoms":
        t, ln = st["graph"].matrix_seeded_2ch(st["src"], st["tgt"], st["threshold"])
        return [_whole(t), _whole(ln)]
    if kind == "customize":
        return [_whole(a) for a in st["cch"].customize(st["up"], st["down"], out=st["out"])]
    at = lambda x: None if x is None else x.data_ptr()  # noqa: E731
    rows = bfphast.tile_emit_device(
        st["dur"].data_ptr(), st["S"], st["T"], st["src"].data_ptr(), st["dst"].data_ptr(),
        [c.data_ptr() for c in st["cols"]], st["threshold"], at(st["off"]), at(st["mask"]),
        0 if st["off"] is None else st["S"], 0 if st["mask"] is None else st["mask"].numel(),
        at(st["len"]), st["sparse"], 0, torch.cuda.current_stream().cuda_stream)
    return st["cols"] + [rows]


def work(case):
    """Inputs read once, outputs written once. A road graph is read where the
    whole of it is needed (8 bytes an edge); of a table's graph only what
    leads to its ends is, which no formula gives: those bytes are left out."""
    kind = case["kind"]
    if kind == "tile":
        cells = case["S"] * case["T"]
        inputs = (8 if case["lengths"] else 4) * cells
        if case["keep"] < 1.0:
            inputs += 4 * case["keep"] * cells
        # about 2.1 % of the durations are within 30 minutes
        rows = cells * case["keep"] * 0.021 if case["sparse"] else cells
        return {"bytes": inputs + 16 * rows, "flops": 0}
    n, edges = GRAPHS[case["graph"]][3:]
    if kind in ("matrix", "matrix_device"):
        return {"bytes": 4 * (case["S"] * case["T"] + case["S"] + case["T"]), "flops": 0}
    if kind == "one_to_all":
        return {"bytes": 4 * case["S"] * (n + 1) + 16 * edges, "flops": 0}
    if kind in ("isochrones", "isochrones_device"):
        return {"bytes": case["S"] * (n / 8 + 16) + 16 * edges, "flops": 0}
    if kind == "polygons":  # roads within 30 minutes, two points each; a ring's vertices
        roads = min(n, 242000 * (case["threshold_s"] / 1800) ** 2)
        return {"bytes": case["S"] * (32 * roads + 16 * 1300), "flops": 0}
    if kind == "phantoms":
        return {"bytes": 8 * case["S"] * case["T"] + 24 * (case["S"] + case["T"]), "flops": 0}
    # customize: the hierarchy's pairs are about 2.2 times its finite edges;
    # an original weight in, a weight and a middle out, both directions
    return {"bytes": 24 * 2.2 * edges, "flops": 0}


def exact(case, seed):
    """Durations, lengths, bits and columns are whole numbers, which have to
    be equal; a ring's vertices follow from which cells of a raster are set,
    for which there is no value in 64 bits but the path's own."""
    return None
