"""Performance cases: what programs that use this partitioner have it do.

Every case is one call (or one short sequence of calls) through the package's
public functions, on synthetic graphs of the kinds the package generates:
2D and 3D grids, random geometric graphs (RGG) and R-MAT power-law graphs.
A case is a dict of plain values:

  call    partition | host | batch | refine | coarsen | stats
  graph   grid2d | grid3d | rgg | rmat, with its sizes (nx, ny, nz / n / scale)
  tier    i32 | big | biggest (integer widths)
  k, alg (0 two-hop matching, 1 HEC, 2 matching), imb, ultra, vw (vertex weights)

All results are whole numbers that do not depend on timing, so they are
compared exactly.
"""
import importlib.util
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package (its folder's name is not a Python identifier), from the
    working folder, which holds the tree that is measured."""
    if "jet_b200" in sys.modules:
        return sys.modules["jet_b200"]
    home = os.path.join(os.getcwd(), "jet-partitioner-official-fork_b200")
    if not os.path.isdir(home):
        home = os.path.join(ROOT, "jet-partitioner-official-fork_b200")
    spec = importlib.util.spec_from_file_location("jet_b200", os.path.join(home, "__init__.py"),
                                                  submodule_search_locations=[home])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["jet_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# Batch workers are host threads with a stream each; without this they share
# hardware queues (the setting INTEGRATION.md gives to users of the batch call).
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")


def listed():
    return [
        # A very small graph with the default coarsening: what a call costs
        # when there is next to no work (launches, synchronisation, Metis).
        dict(name="rgg2k", call="partition", graph="rgg", n=2003, weighted=True, tier="i32", k=8, alg=0, imb=1.03),
        # The small plain configuration: 256 x 256 grid, unit weights, HEC.
        dict(name="grid256", call="partition", graph="grid2d", nx=256, ny=256, weighted=False, tier="i32", k=32, alg=1,
             imb=1.03),
        # A small mesh with ultra_settings, the option for better cuts at the
        # price of many more refinement iterations.
        dict(name="grid301_ultra", call="partition", graph="grid2d", nx=301, ny=211, weighted=True, tier="i32", k=24, alg=1,
             imb=1.03, ultra=True),
        # A mid-size geometric graph (a mesh or road-like network) with vertex
        # weights and pure matching.
        dict(name="rgg150k_match", call="partition", graph="rgg", n=150001, weighted=True, vw=True, tier="i32", k=48, alg=2,
             imb=1.03),
        # A solver's mesh in host memory, cut into many parts (more than the
        # shared-memory tables of one warp take), 64-bit offsets and weights.
        dict(name="mesh717k_host_k768", call="host", graph="grid3d", nx=96, ny=90, nz=83, weighted=True, tier="big", k=768,
             alg=0, imb=1.05),
        # The large mesh configuration: 128^3 7-point grid, HEC.
        dict(name="grid128", call="partition", graph="grid3d", nx=128, ny=128, nz=128, weighted=True, tier="i32", k=64, alg=1,
             imb=1.03),
        # A mid-size power-law graph in the widest integer tier.
        dict(name="rmat20_biggest", call="partition", graph="rmat", scale=20, tier="biggest", k=96, alg=0, imb=1.05),
        # The large power-law configuration (social network / web graph):
        # 2^24 vertices, 2.6e8 entries, two-hop matching.
        dict(name="rmat24", call="partition", graph="rmat", scale=24, tier="big", k=256, alg=0, imb=1.10),
        # The batched configuration: independent geometric graphs of uneven
        # size in one call, 16 workers (48 graphs of the configuration's 512).
        dict(name="batch48", call="batch", graph="rgg", count=48, lo=1000, hi=200000, weighted=True, tier="i32", alg=1,
             imb=1.03, workers=16),
        # Improving a partition that a program already has (slabs of a mesh
        # ordering after some vertices moved): one level of refinement.
        dict(name="refine700k", call="refine", graph="grid2d", nx=1000, ny=701, weighted=True, tier="i32", k=64, imb=1.03),
        # One coarsening step on its own: a two-hop map and the contraction.
        dict(name="coarsen_rmat21", call="coarsen", graph="rmat", scale=21, tier="big", alg=0),
        # Evaluating a partition (cut, sizes, communication volume).
        dict(name="stats3m", call="stats", graph="grid3d", nx=160, ny=150, nz=131, weighted=True, tier="i32", k=128),
    ]


def _logint(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["partition", "partition", "partition", "partition", "host", "batch", "refine", "coarsen", "stats"])
    if call == "batch":
        lo = _logint(rng, 1000, 4000)
        return dict(call=call, graph="rgg", count=rng.randint(6, 48), lo=lo, hi=_logint(rng, 20000, 200000), weighted=True,
                    tier=rng.choice(["i32", "i32", "big"]), alg=rng.choice([0, 1, 1, 2]), imb=1.03,
                    workers=rng.choice([8, 16]))
    graph = rng.choice(["grid2d", "grid3d", "rgg", "rmat"])
    if call == "refine" and graph == "rmat":
        graph = "grid3d"
    c = dict(call=call, graph=graph, tier=rng.choice(["i32", "i32", "big", "biggest"]))
    if graph == "grid2d":
        n = _logint(rng, 3000, 2000000)
        c["nx"] = max(16, int(n ** 0.5 * rng.uniform(0.6, 1.6)))
        c["ny"] = max(16, n // c["nx"])
        c["weighted"] = rng.random() < 0.6
    elif graph == "grid3d":
        n = _logint(rng, 5000, 3000000)
        c["nx"] = max(8, int(n ** (1 / 3) * rng.uniform(0.7, 1.4)))
        c["ny"] = max(8, int(n ** (1 / 3) * rng.uniform(0.7, 1.4)))
        c["nz"] = max(8, n // (c["nx"] * c["ny"]))
        c["weighted"] = rng.random() < 0.8
    elif graph == "rgg":
        c["n"] = _logint(rng, 2000, 800000)
        c["weighted"] = rng.random() < 0.8
    else:
        c["scale"] = rng.randint(12, 22)
    if call in ("partition", "host", "coarsen"):
        c["alg"] = rng.choice([0, 0, 1, 2])
    if call != "coarsen":
        n = _vertices(c)
        # power-law graphs into up to 256 parts (the range of the serving configuration), meshes into more
        c["k"] = max(2, min(_logint(rng, 4, 256 if graph == "rmat" else 800), n // 60))
    if call in ("partition", "host", "refine"):
        c["imb"] = rng.choice([1.03, 1.03, 1.05, 1.10])
        c["vw"] = rng.random() < 0.25
    if call in ("partition", "host") and _vertices(c) < 300000 and graph != "rmat":
        c["ultra"] = rng.random() < 0.15
    return c


def _vertices(c):
    g = c["graph"]
    if g == "grid2d":
        return c["nx"] * c["ny"]
    if g == "grid3d":
        return c["nx"] * c["ny"] * c["nz"]
    if g == "rgg":
        return c["n"]
    return 1 << c["scale"]


def _entries(c):
    """Stored entries (both directions); expected values for random graphs."""
    g = c["graph"]
    if g == "grid2d":
        x, y = c["nx"], c["ny"]
        return 2 * ((x - 1) * y + x * (y - 1))
    if g == "grid3d":
        x, y, z = c["nx"], c["ny"], c["nz"]
        return 2 * ((x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1))
    if g == "rgg":
        return 10 * c["n"]
    return int(15.5 * (1 << c["scale"]))


def _graph(jet, c, seed, device):
    G = jet.graphs
    g = c["graph"]
    if g == "grid2d":
        r = G.grid2d(c["nx"], c["ny"], weighted=c["weighted"], seed=seed, device=device)
    elif g == "grid3d":
        r = G.grid3d(c["nx"], c["ny"], c["nz"], weighted=c["weighted"], seed=seed, device=device)
    elif g == "rgg":
        r = G.rgg(c["n"], 10.0, seed=seed, weighted=c["weighted"], device=device)
    else:
        r = G.rmat(c["scale"], 8, seed=seed, tier=c["tier"], device=device)
    r = r.as_tier(c["tier"])
    if c.get("vw"):
        gen = torch.Generator().manual_seed(seed + 77)
        r.vw = torch.randint(1, 6, (r.n,), generator=gen).to(r.vw.dtype).to(r.vw.device)
    return r


def _config(jet, c, k):
    return jet.config_t(coarsening_alg=c["alg"], num_parts=k, max_imb_ratio=c["imb"], ultra_settings=bool(c.get("ultra")))


def prepare(case, seed):
    jet = _package()
    c = case
    s = dict(jet=jet, call=c["call"], seed=seed + 1)
    if c["call"] == "batch":
        # the sizes and part counts belong to the case, the graphs to the seed
        rng = random.Random(c["count"] * 1000003 + c["lo"] * 1009 + c["hi"])
        graphs, configs = [], []
        for i in range(c["count"]):
            n = _logint(rng, c["lo"], c["hi"])
            k = rng.choice((8, 16, 32, 64))
            graphs.append(_graph(jet, dict(c, graph="rgg", n=n), seed * 1000 + i, "cuda"))
            configs.append(_config(jet, c, k))
        s.update(graphs=graphs, configs=configs, seeds=[seed + i for i in range(c["count"])], workers=c["workers"],
                 tier=c["tier"])
        return s
    g = _graph(jet, c, seed, "cuda")
    if c["call"] == "partition":
        fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[c["tier"]]
        s.update(fn=fn, g=g, config=_config(jet, c, c["k"]))
    elif c["call"] == "host":
        fn = {"i32": jet.partition_host, "big": jet.partition_host_big, "biggest": jet.partition_host_biggest}[c["tier"]]
        s.update(fn=fn, g=g.to("cpu"), config=_config(jet, c, c["k"]))
    elif c["call"] in ("refine", "stats"):
        # slabs of the vertex order, a fiftieth of the vertices elsewhere
        k = c["k"]
        gen = torch.Generator().manual_seed(seed + 5)
        part = (torch.arange(g.n) * k // g.n).to(torch.int32)
        part = torch.where(torch.rand(g.n, generator=gen) < 0.02, torch.randint(0, k, (g.n,), generator=gen).to(torch.int32), part)
        s.update(g=g, part=part.cuda(), k=k, imb=c.get("imb", 1.03))
    else:
        # the program's own buffers for the coarse graph, at most as large as the fine one
        cap = {"grid2d": _entries(c), "grid3d": _entries(c), "rgg": 11 * g.n + 4096}.get(c["graph"], 16 * g.n)
        into = {"row": torch.zeros(g.n + 1, dtype=g.row.dtype, device="cuda"),
                "adj": torch.zeros(cap, dtype=g.adj.dtype, device="cuda"),
                "val": torch.zeros(cap, dtype=g.val.dtype, device="cuda"),
                "vw": torch.zeros(g.n, dtype=g.vw.dtype, device="cuda")}
        s.update(g=g, alg=c["alg"], into=into)
    return s


def run(state):
    s = state
    jet = s["jet"]
    if s["call"] in ("partition", "host"):
        part, cut, _ = s["fn"](s["config"], s["g"], seed=s["seed"])
        return {"part": part, "cut": cut}
    if s["call"] == "batch":
        out = jet.partition_batch(s["configs"], s["graphs"], seeds=s["seeds"], workers=s["workers"], tier=s["tier"])
        return {"part": torch.cat([p for p, _, _ in out]), "cut": torch.tensor([c for _, c, _ in out])}
    if s["call"] == "refine":
        part, cut, _ = jet.refine_level(s["g"], s["part"], s["k"], s["imb"])
        return {"part": part, "cut": cut}
    if s["call"] == "coarsen":
        cmap, nc, _ = jet.coarsen_map(s["g"], s["alg"], level=1, seed=s["seed"])
        c = jet.contract(s["g"], cmap, nc)
        into = s["into"]
        for name, t in (("row", c.row), ("adj", c.adj), ("val", c.val), ("vw", c.vw)):
            into[name][:t.numel()].copy_(t)
        return dict(into, map=cmap, nc=nc)
    return {"stats": torch.tensor(jet.pstat(s["g"], s["part"], s["k"]))}


_BYTES = {"i32": (4, 4, 4), "big": (4, 8, 8), "biggest": (8, 8, 8)}


def work(case):
    """Bytes of the graph read once and the results written once."""
    c = case
    o, e, w = _BYTES[c["tier"]]
    if c["call"] == "batch":
        # mean of a log-uniform size
        n = c["count"] * (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"])
        m = 10 * n
    else:
        n, m = _vertices(c), _entries(c)
    b = (n + 1) * e + m * (o + w) + n * w
    if c["call"] == "coarsen":
        b += n * o + 0.5 * ((n + 1) * e + m * (o + w) + n * w)  # the map, and a coarse graph of about half the size
    else:
        b += 4 * n
    return {"bytes": float(b), "flops": 0.0}


def tolerance(case):
    return "exact"


def _exact_stats(s):
    g, part, k = s["g"], s["part"].long(), s["k"]
    src = torch.repeat_interleave(torch.arange(g.n, device=part.device), (g.row[1:] - g.row[:-1]).long())
    dst = g.adj.long()
    out = part[src] != part[dst]
    w = g.val.long()
    cut = int(w[out].sum())
    per = torch.zeros(k, dtype=torch.int64, device=part.device).index_add_(0, part[src[out]], w[out])
    comm = torch.unique(src[out] * k + part[dst[out]]).numel()
    sizes = torch.zeros(k, dtype=torch.int64, device=part.device).index_add_(0, part, g.vw.long())
    return [cut // 2, int(per.max()), comm, int(sizes.max()), int(sizes.min()), int(sizes.sum())]


def exact(case, seed):
    """The statistics restated with torch; partitions and maps are whole
    numbers whose value only the method itself defines."""
    if case["call"] != "stats":
        return None
    return {"stats": torch.tensor(_exact_stats(prepare(case, seed)))}
