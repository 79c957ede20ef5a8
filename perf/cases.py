"""Performance cases of the walk engine: what a user's program calls, by size.

Five kinds of work, each through a public entry point:

  walk    a long-lived program keeps a WalkEngine on a graph that is already
          on the GPU and walks it again and again (one pass = set the walker
          population, run, read the result into pinned host memory);
  device  the caller owns every buffer (gw_walk_noalloc): walks of a CSR on
          the GPU into the caller's device tensors, paths included;
  app     a one-shot program, as the Node2vec / SOPR / SOSR command lines are:
          make the engine, give it the graph, walk once, read the walks, close;
  ooc     a graph larger than the device cache, in blocks of pinned host memory;
  edges   an edge list on the GPU to a CSR (gw_edges_csr), the step before all
          of the above.

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05) like the benchmark's, 16 edges drawn
per vertex, the generator seeded by the case's seed.  All outputs are whole
numbers: vertex ids, lengths, 64-bit path hashes, step counts, CSR arrays.
"""
import ctypes
import math

import numpy as np
import torch

import gowalker_b200 as gw
from gowalker_b200.preprocess import split_equal_edge_mass


def listed():
    return [
        # The smallest walk anyone asks for (a test-sized graph, the default
        # p, q and length, every path read back): launches and waits.
        dict(name="n2v_tiny", kind="walk", algo=0, scale=10, nverts=1024, wps=1, length=30, p=0.5, q=2.0, term=0.0,
             init=0, numwalks=0, read="paths"),
        # A corpus for embeddings: ten walks per vertex of a mid-size graph
        # that fits L2, the paper's p, q and length.
        dict(name="n2v_corpus", kind="walk", algo=0, scale=16, nverts=60001, wps=10, length=80, p=0.5, q=2.0,
             term=0.0, init=0, numwalks=0, read="hashes"),
        # Node2vec on a graph larger than L2 (the benchmark's in-core
        # workload, one size up, hashes read back).
        dict(name="n2v_large", kind="walk", algo=0, scale=21, nverts=1 << 21, wps=1, length=80, p=2.0, q=0.5,
             term=0.0, init=0, numwalks=0, read="hashes"),
        # Second-order PageRank walks of uneven length, four per vertex.
        dict(name="sopr_mid", kind="walk", algo=1, scale=18, nverts=250007, wps=4, length=20, p=0.5, q=2.0, term=0.15,
             init=0, numwalks=0, read="hashes"),
        # The same on a graph of 128 M edges: the benchmark's SOPR workload at
        # a quarter of its size.
        dict(name="sopr_large", kind="walk", algo=1, scale=22, nverts=1 << 22, wps=4, length=20, p=0.5, q=2.0,
             term=0.15, init=0, numwalks=0, read="hashes"),
        # SOSR from its fixed sources (the reference's own start for SOPR and
        # SOSR): every walker begins at the same two vertices.
        dict(name="sosr_source", kind="walk", algo=2, scale=20, nverts=1 << 20, wps=1, length=20, p=0.5, q=2.0,
             term=0.15, init=1, numwalks=400000, read="paths"),
        # Walks for a consumer on the GPU: paths, lengths and hashes into the
        # caller's tensors (the benchmark's in-core Node2vec workload).
        dict(name="n2v_device", kind="device", algo=0, scale=20, nverts=1 << 20, wps=1, length=80, p=2.0, q=0.5,
             term=0.0, init=0, numwalks=0),
        # The command-line app: host CSR in, every path out, once.
        dict(name="n2v_app", kind="app", algo=0, scale=16, nverts=1 << 16, wps=1, length=30, p=0.5, q=2.0, term=0.0,
             weighted=False),
        # Weighted Node2vec in one shot: the alias tables are built for it.
        dict(name="weighted_app", kind="app", algo=0, scale=18, nverts=200003, wps=1, length=80, p=2.0, q=0.5,
             term=0.0, weighted=True),
        # A graph four times the device cache, blocks compressed and fetched
        # ahead, GOWalker's zero mode for the tail: the headline's options.
        dict(name="ooc_n2v", kind="ooc", algo=0, scale=21, nverts=1300007, wps=1, length=80, p=0.5, q=2.0, term=0.0,
             blocks=24, cache=0.45, compress=1, prefetch=1, zero=1),
        # SOPR out of core with the default options: plain copies, no prefetch.
        dict(name="ooc_sopr", kind="ooc", algo=1, scale=19, nverts=500009, wps=2, length=20, p=0.5, q=2.0, term=0.15,
             blocks=12, cache=0.6, compress=0, prefetch=0, zero=0),
        # Edge list to a sorted, deduplicated, undirected CSR.
        dict(name="edges_large", kind="edges", scale=22, pairs=50_000_003, given=1, symmetric=1, sort=1, dedup=1),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "device", "app", "ooc", "edges"])
    if kind == "edges":
        pairs = _log(rng, 20_000, 40_000_000)
        dedup = rng.randint(0, 1)
        return dict(kind=kind, scale=max(10, min(23, int(math.log2(pairs)) - rng.randint(2, 5))), pairs=pairs,
                    given=rng.randint(0, 1), symmetric=rng.randint(0, 1), sort=1 if dedup else rng.randint(0, 1),
                    dedup=dedup)
    algo = rng.choice([0, 0, 1, 2])
    c = dict(kind=kind, algo=algo)
    top = {"walk": 2_000_000, "device": 1_000_000, "app": 200_000, "ooc": 1_000_000}[kind]
    c["nverts"] = _log(rng, 1000 if kind != "ooc" else 100_000, top)
    c["scale"] = max(10, (c["nverts"] - 1).bit_length())
    p, q = rng.choice([(0.5, 2.0), (2.0, 0.5), (1.0, 1.0), (0.25, 4.0), (4.0, 0.25), (1.0, 2.0)])
    c.update(p=p, q=q)
    if algo == 0:
        c.update(wps=rng.choice([1, 1, 2]) if kind == "walk" else 1, length=rng.choice([10, 30, 40, 80]), term=0.0)
    else:
        c.update(wps=rng.choice([1, 2, 4]) if kind == "walk" else rng.choice([1, 2]), length=20,
                 term=rng.choice([0.15, 0.15, 0.2]))
    if kind in ("walk", "device"):
        init = rng.choice([0, 0, 0, 1, 2])
        c.update(init=init, numwalks=0 if init == 0 else _log(rng, 1000, 400_000))
    if kind == "walk":
        big = c["nverts"] * c["wps"] * (c["length"] + 1) > 30_000_000
        c["read"] = "hashes" if big else rng.choice(["paths", "hashes"])
    if kind == "app":
        c["weighted"] = algo == 0 and rng.random() < 0.4
    if kind == "ooc":
        c.update(blocks=rng.randint(8, 24), cache=round(rng.uniform(0.5, 0.8), 2), compress=rng.randint(0, 1),
                 prefetch=rng.randint(0, 1), zero=rng.randint(0, 1))
    return c


def _graph(case, seed, symmetric=True):
    return gw.DeviceGraph(case["scale"], nverts=case["nverts"], edgefactor=16, seed=seed & 0x7FFFFFFF,
                          symmetric=symmetric)


def _options(case, seed):
    """Engine options of a case; the walk seed comes from the case's seed."""
    return dict(algorithm=case["algo"], maxhops=case["length"], p=case["p"], q=case["q"], alpha=0.2,
                term_prob=case["term"], walkpersource=case["wps"], seed=(seed * 2654435761 + 12345) & 0xFFFFFFFF)


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _rmat_pairs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["pairs"]
    src = torch.zeros(n, dtype=torch.int32, device="cuda")
    dst = torch.zeros(n, dtype=torch.int32, device="cuda")
    for _ in range(case["scale"]):
        u = torch.rand(n, device="cuda", generator=g)
        src.mul_(2).add_(u >= 0.76)
        dst.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    src[0], dst[0] = (1 << case["scale"]) - 1, 0  # the last vertex has an edge, so the vertex count can be found
    return src, dst


class _Array:
    """A CSR array on the GPU, for torch.as_tensor; keeps its graph alive."""

    def __init__(self, graph, ptr, n, kind):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "edges":
        src, dst = _rmat_pairs(case, seed)
        most = case["pairs"] * (2 if case["symmetric"] else 1)
        return dict(case=case, src=src, dst=dst, csr=torch.zeros(most, dtype=torch.int32, device="cuda"))
    s = dict(case=case, opt=_options(case, seed))
    if kind == "ooc":
        dg = _graph(case, seed, symmetric=case["algo"] != 0)
        s["beg"], s["csr"] = dg.to_host(pinned=True)
        nedges = dg.nedges
        dg.free()
        beg = s["beg"].numpy().view(np.uint64)
        vb, eb = split_equal_edge_mass(beg, case["blocks"])
        largest = 4 * int(np.diff(eb.astype(np.int64)).max())
        # the vertex offsets, then the case's share of the blocks (at least
        # what a prefetching run with two staging buffers needs)
        slots = max(5, int(case["cache"] * case["blocks"]))
        cache = 8 * (case["nverts"] + 1) + (slots + 2 * case["compress"]) * (largest + 64)
        eng = gw.WalkEngine(cache_size=cache, compress_blocks=case["compress"], prefetch=case["prefetch"],
                            zero_copy=case["zero"], zero_threshold=largest // 128 // 24 if case["zero"] else 0,
                            **s["opt"])
        eng.set_host_graph(s["beg"], s["csr"][:nedges], vb, eb)
        s.update(eng=eng, hashes=_pinned(case["nverts"] * case["wps"], torch.int64))
        return s
    s["graph"] = dg = _graph(case, seed)
    if kind == "walk":
        eng = gw.WalkEngine(init_mode=case["init"], numwalks=case["numwalks"],
                            record_paths=1 if case["read"] == "paths" else 0, **s["opt"])
        eng.set_device_graph(dg.nverts, dg.nedges, dg.beg_ptr, dg.csr_ptr)
        n = case["numwalks"] or case["nverts"] * case["wps"]
        s.update(eng=eng, n=n, lens=_pinned(n, torch.int32))
        if case["read"] == "paths":
            s["paths"] = _pinned((n, case["length"] + 1), torch.int32)
        else:
            s["hashes"] = _pinned(n, torch.int64)
    elif kind == "device":
        n = case["numwalks"] or case["nverts"] * case["wps"]
        s.update(n=n, cfg=gw.default_config(init_mode=case["init"], numwalks=case["numwalks"], record_paths=1,
                                            **s["opt"]),
                 hashes=torch.empty(n, dtype=torch.int64, device="cuda"),
                 lens=torch.empty(n, dtype=torch.int32, device="cuda"),
                 paths=torch.empty((n, case["length"] + 1), dtype=torch.int32, device="cuda"))
    elif kind == "app":
        if case["weighted"]:
            g = torch.Generator(device="cuda")
            g.manual_seed(seed)
            s["w"] = torch.empty(max(dg.nedges, 1), dtype=torch.float32, device="cuda").log_normal_(0, 1, generator=g)
        else:
            s["beg"], s["csr"] = dg.to_host(pinned=True)
            s["csr"] = s["csr"][: dg.nedges]
            dg.free()
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "edges":
        g = gw.DeviceGraph.from_edges(s["src"], s["dst"], nverts=(1 << case["scale"]) if case["given"] else 0,
                                      symmetric=bool(case["symmetric"]), sort=bool(case["sort"]),
                                      dedup=bool(case["dedup"]))
        # the program's own array, sized for an input without repeats, takes
        # the neighbour ids; the offsets say how much of it is used
        s["csr"][: g.nedges].copy_(torch.as_tensor(_Array(g, g.csr_ptr, g.nedges, "<i4"), device="cuda"))
        return {"beg": torch.as_tensor(_Array(g, g.beg_ptr, g.nverts + 1, "<i8"), device="cuda"), "csr": s["csr"]}
    if kind == "device":
        L, g, st = gw.load(), s["graph"], gw.GwStats()
        rc = L.gw_walk_noalloc(ctypes.byref(s["cfg"]), ctypes.c_void_p(g.beg_ptr), ctypes.c_void_p(g.csr_ptr),
                               g.nverts, g.nedges, s["n"], _ptr(s["hashes"]), _ptr(s["lens"]), _ptr(s["paths"]),
                               None, ctypes.byref(st))
        if rc != 0:
            raise gw.GwError(rc, "gw_walk_noalloc failed")
        return {"hashes": s["hashes"], "lens": s["lens"], "paths": s["paths"], "steps": int(st.steps)}
    if kind == "app":
        with gw.WalkEngine(record_paths=1, **s["opt"]) as eng:
            if case["weighted"]:
                g = s["graph"]
                eng.set_device_graph(g.nverts, g.nedges, g.beg_ptr, g.csr_ptr)
                eng.set_device_weights(s["w"].data_ptr())
            else:
                eng.set_host_graph(s["beg"], s["csr"])
            eng.init_walkers()
            st = eng.run()
            paths, lens = eng.paths()
        return {"paths": paths.view(np.int32), "lens": lens.view(np.int32), "steps": st["steps"]}
    eng, L = s["eng"], gw.load()
    eng.init_walkers()
    st = eng.run()
    if kind == "walk":
        out = {"steps": st["steps"], "lens": s["lens"]}
        if case["read"] == "paths":
            eng._check(L.gw_get_paths(eng.h, 0, s["n"], _ptr(s["paths"]), _ptr(s["lens"])))
            out["paths"] = s["paths"]
        else:
            eng._check(L.gw_path_lengths(eng.h, 0, s["n"], _ptr(s["lens"])))
            eng._check(L.gw_path_hashes(eng.h, 0, s["n"], _ptr(s["hashes"])))
            out["hashes"] = s["hashes"]
        return out
    eng._check(L.gw_path_hashes(eng.h, 0, s["hashes"].numel(), _ptr(s["hashes"])))
    return {"hashes": s["hashes"], "steps": st["steps"]}


L2_BYTES = 126 << 20


def work(case):
    """What a pass cannot do without, from the case alone: the outputs, and
    the graph's arrays once, or, on a graph larger than L2, one 32-byte sector
    for each step's offsets and one for its neighbour where that is more.  The
    walkers of an R-MAT graph's isolated vertices (about 0.4 of them when
    symmetric) take no step; SOPR and SOSR walks end early by their termination
    probability; walks of a directed R-MAT graph end at vertices without
    out-edges."""
    if case["kind"] == "edges":
        m = case["pairs"] * (2 if case["symmetric"] else 1)
        return {"bytes": 8 * case["pairs"] + 4 * m + (8 << case["scale"]), "flops": 0}
    walkers = case.get("numwalks") or case["nverts"] * case["wps"]
    mean = case["length"]
    if case["term"] > 0:
        mean = sum((1 - case["term"]) ** h for h in range(case["length"]))
    alive = 1.0 if case.get("init") else 0.6
    steps = walkers * mean * alive * (0.8 if case["kind"] == "ooc" else 1.0)
    out = 12 * walkers
    if case["kind"] in ("device", "app") or case.get("read") == "paths":
        out += 4 * walkers * (case["length"] + 1)
    edges = 16 * case["nverts"] * (1 if case["kind"] == "ooc" and case["algo"] == 0 else 2)
    graph = 8 * case["nverts"] + 4 * edges * (2 if case.get("weighted") else 1)
    gathers = 64 * steps
    if case["kind"] in ("ooc", "app"):
        graph = max(graph, gathers) if graph > L2_BYTES else graph
    else:
        graph = gathers if graph > L2_BYTES else min(graph, gathers)
    return {"bytes": int(out + graph), "flops": 0}
