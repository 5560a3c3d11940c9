"""Parity of the CUDA path (through the C ABI) with the CPU oracle.

Exact (bit-for-bit) where the computation is deterministic:
  * contraction given a map (rows compared sorted), coarse vertex weights
  * connectivity tables given a partition (sizes and {part: weight} sets)
  * heavy-edge / matching proposals given the seed
  * LP refinement iterations from a balanced partition: parts, part sizes,
    cut and tables after every iteration
  * pstat quantities and projection
Properties where the reference itself races (aggregation CAS rounds).
"""
import numpy as np
import pytest
import torch

from conftest import sorted_rows, table_multisets

pytestmark = pytest.mark.gpu

TIERS = ["i32", "big", "biggest"]


def host(t):
    return t.detach().cpu().numpy()


def make(graphs, kind, tier):
    if kind == "grid2d":
        g = graphs.grid2d(48, 40, weighted=True, seed=3)
    elif kind == "grid3d":
        g = graphs.grid3d(14, 12, 10, weighted=True, seed=5)
    elif kind == "rgg":
        g = graphs.rgg(3000, 10.0, seed=2)
    elif kind == "rmat":
        g = graphs.rmat(11, 8, seed=4, tier=tier)
    elif kind == "star":
        # a hub of degree 5000 plus a ring: exercises the CTA-per-vertex paths
        n = 6001
        u = torch.cat([torch.zeros(5000, dtype=torch.long), torch.arange(1, 6000)])
        v = torch.cat([torch.arange(1, 5001), torch.arange(2, 6001)])
        g = graphs.from_undirected(n, u, v, torch.randint(1, 5, (u.numel(),), generator=torch.Generator().manual_seed(1)))
    elif kind == "dense":
        # 1500 rows of about 100 edges, three hubs of 5000, a ring: over a
        # thousand rows above 32 edges, so the tables go through the
        # persistent longest-first build (whole-block and single-warp rows)
        n = 6000
        gen = torch.Generator().manual_seed(2)
        u = torch.cat([torch.arange(1500).repeat_interleave(100), torch.tensor([1500, 1501, 1502]).repeat_interleave(5000),
                       torch.arange(n)])
        v = torch.cat([torch.randint(0, n, (150000,), generator=gen),
                       torch.cat([torch.randperm(n, generator=gen)[:5000] for _ in range(3)]), (torch.arange(n) + 1) % n])
        a, b = torch.minimum(u, v), torch.maximum(u, v)
        pairs = torch.unique((a * n + b)[a != b])
        g = graphs.from_undirected(n, pairs // n, pairs % n, torch.randint(1, 5, (pairs.numel(),), generator=gen))
    else:
        raise ValueError(kind)
    return g.as_tier(tier)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind", ["grid2d", "rgg", "rmat", "star"])
def test_contract_bit_exact(jet, graphs, orc, tier, kind):
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    m, nc, _ = orc.coarsen(og, 1 if kind != "rmat" else 0, level=2, seed=7, uniform=False)
    want = orc.contract(og, m, nc)
    got = jet.contract(g.to("cuda"), torch.from_numpy(m).cuda(), nc)
    assert got.nnz == len(want.adj)
    assert np.array_equal(host(got.row), want.row)
    assert np.array_equal(host(got.vw), want.vw)
    # every row, hub rows included, comes out in neighbour order
    assert np.array_equal(host(got.adj), want.adj)
    assert np.array_equal(host(got.val), want.val)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind", ["grid3d", "rmat", "star", "dense"])
@pytest.mark.parametrize("k", [8, 64, 300, 700])
def test_conn_tables_bit_exact(jet, graphs, orc, tier, kind, k):
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    rng = np.random.default_rng(k)
    part = rng.integers(0, k, g.n).astype(np.int32)
    off, ent, val, size = orc.conn_build(og, part, k)
    goff, gent, gval, gsize = jet.conn_build(g.to("cuda"), torch.from_numpy(part).cuda(), k)
    assert np.array_equal(host(goff), off)
    assert np.array_equal(host(gsize), size)
    assert table_multisets(host(goff), host(gent), host(gval), host(gsize)) == table_multisets(off, ent, val, size)


@pytest.mark.parametrize("tier", ["i32", "big"])
@pytest.mark.parametrize("uniform", [True, False])
def test_hec_proposals_bit_exact(jet, graphs, orc, tier, uniform):
    g = make(graphs, "grid3d", tier)
    og = orc.G.from_csr(g)
    _, _, hn = orc.coarsen(og, 1, level=3, seed=11, uniform=uniform)
    _, _, ghn = jet.coarsen_map(g.to("cuda"), 1, level=3, seed=11, uniform=uniform)
    assert np.array_equal(host(ghn), hn)


@pytest.mark.parametrize("kind", ["rgg", "rmat", "star"])
@pytest.mark.parametrize("uniform", [True, False])
def test_match_proposals_bit_exact(jet, graphs, orc, kind, uniform):
    tier = "big" if kind == "rmat" else "i32"
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    _, _, hn = orc.coarsen(og, 2, level=1, seed=5, uniform=uniform)
    _, _, ghn = jet.coarsen_map(g.to("cuda"), 2, level=1, seed=5, uniform=uniform)
    assert np.array_equal(host(ghn), hn)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind", ["grid2d", "grid3d", "rgg", "rmat", "star"])
@pytest.mark.parametrize("alg,uniform", [(1, True), (1, False), (2, True), (2, False), (0, True), (0, False)])
def test_coarsen_map_bit_exact(jet, graphs, orc, tier, kind, alg, uniform):
    """HEC, pure matching and 2-hop matching produce the oracle's (in-order)
    map exactly."""
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    m, nc, _ = orc.coarsen(og, alg, level=2, seed=13, uniform=uniform)
    gm, gnc, _ = jet.coarsen_map(g.to("cuda"), alg, level=2, seed=13, uniform=uniform)
    assert gnc == nc
    assert np.array_equal(host(gm), m)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("alg", [0, 1, 2])
@pytest.mark.parametrize("kind", ["grid2d", "rmat", "star"])
def test_coarsen_map_properties(jet, graphs, tier, alg, kind):
    g = make(graphs, kind, tier)
    m, nc, _ = jet.coarsen_map(g.to("cuda"), alg, level=1, seed=3, uniform=g.uniform)
    m = host(m)
    assert 0 < nc <= g.n
    assert m.min() == 0 and m.max() == nc - 1
    assert len(np.unique(m)) == nc
    sizes = np.bincount(m, minlength=nc)
    if alg == 2:
        assert sizes.max() <= 2
    row, adj = host(g.row), host(g.adj)
    deg = np.diff(row)
    # isolated vertices propose a random vertex under HEC (src/heuristics.hpp:205),
    # so an aggregate may hold a vertex plus isolated ones
    has_isolated = np.zeros(nc, dtype=bool)
    has_isolated[m[deg == 0]] = True
    for i in range(0, g.n, 17):
        if sizes[m[i]] > 1 and alg != 0 and deg[i] > 0 and not has_isolated[m[i]]:
            assert np.any(m[adj[row[i]:row[i + 1]]] == m[i])


def balanced_start(orc, og, k):
    return orc.metis(og, k)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind,k", [("grid2d", 8), ("grid3d", 16), ("rgg", 32), ("rmat", 16)])
def test_lp_iterations_bit_exact(jet, graphs, orc, tier, kind, k):
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    part = balanced_start(orc, og, k)
    imb = 1.10 if kind == "rmat" else 1.03
    fr = 0.25 if g.uniform else 0.75
    for iters in (1, 3, 8):
        want = orc.refine_iters(og, part, k, imb, fr, iters)
        if any(kk != 0 for kk in want["kinds"]):
            continue  # this prefix reached a rebalancing step: checked statistically elsewhere
        got = jet.refine_iters(g.to("cuda"), torch.from_numpy(part).cuda(), k, imb, fr, iters)
        assert got["kinds"] == list(want["kinds"])
        assert got["moves"] == list(want["moves"])
        assert np.array_equal(host(got["part"]), want["part"])
        assert np.array_equal(host(got["sizes"]), want["sizes"])
        assert got["cut"] == want["cut"]
        assert np.array_equal(host(got["size"]), want["size"])
        assert np.array_equal(host(got["dest_cache"]), want["dest_cache"])
        gm = table_multisets(host(got["off"]), host(got["ent"]), host(got["val"]), host(got["size"]))
        wm = table_multisets(want["off"], want["ent"], want["val"], want["size"])
        assert gm == wm


@pytest.mark.parametrize("queue", [True, False], ids=["queue", "fullsort"])
@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind,k", [("grid2d", 8), ("grid3d", 16), ("rgg", 32), ("rmat", 16), ("star", 4), ("dense", 64)])
def test_rebalance_iterations_bit_exact(jet, graphs, orc, tier, kind, k, queue):
    """Weak and strong rebalancing reproduce the oracle's in-order bucket
    scores and destination draws: parts, sizes, cut and tables match after
    every iteration of runs that start badly unbalanced (30% and 90% of the
    vertices piled into part 0; from the latter two weak iterations do not
    restore balance, so strong rebalancing runs).  Both eviction forms: the
    queue of the candidates whose in-bucket order matters, and the sort of
    every candidate."""
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    imb = 1.10 if kind == "rmat" else 1.03
    seen = set()
    prev = jet.set_refine_drivers(jet.DRIVER_ALL if queue else jet.DRIVER_ALL & ~jet.DRIVER_REB_QUEUE)
    try:
        for skew in (0.3, 0.9):
            seen.update(_skewed_runs(jet, orc, g, og, k, imb, skew))
    finally:
        jet.set_refine_drivers(prev)
    assert 1 in seen
    if kind not in ("grid2d", "star"):
        assert 2 in seen


def _skewed_runs(jet, orc, g, og, k, imb, skew, iters_list=(1, 2, 3, 6, 10)):
    """refine_iters from a Metis partition with a share `skew` of the
    vertices moved to part 0, against the oracle after each count of
    iterations; returns the iteration kinds seen."""
    seen = set()
    rng = np.random.default_rng(1)
    part = orc.metis(og, k)
    part[rng.random(g.n) < skew] = 0
    for iters in iters_list:
        want = orc.refine_iters(og, part, k, imb, 0.75, iters)
        got = jet.refine_iters(g.to("cuda"), torch.from_numpy(part).cuda(), k, imb, 0.75, iters)
        assert got["kinds"] == list(want["kinds"])
        assert got["moves"] == list(want["moves"])
        assert np.array_equal(host(got["part"]), want["part"])
        assert np.array_equal(host(got["sizes"]), want["sizes"])
        assert got["cut"] == want["cut"]
        gm = table_multisets(host(got["off"]), host(got["ent"]), host(got["val"]), host(got["size"]))
        assert gm == table_multisets(want["off"], want["ent"], want["val"], want["size"])
    seen.update(want["kinds"])
    # the cut bookkeeping matches a fresh recomputation
    assert got["cut"] // 2 == orc.pstat(og, host(got["part"]), k)[0]
    return seen


@pytest.mark.parametrize("nx,ny,k", [(33, 1, 2), (43, 3, 4), (64, 64, 3), (1621, 1500, 5)],
                         ids=["one_over_a_warp", "one_over_a_stretch", "whole_stretches", "two_rounds"])
def test_vertex_pass_edges(jet, graphs, orc, nx, ny, k):
    """The grid kernels give each warp a stretch of at most 128 vertices:
    sizes around a warp and a stretch, and one above what the whole grid
    covers in a round (18,944 warps), in iterations that rebalance and then
    run LP; parts, moves and cut equal the oracle's."""
    g = graphs.grid2d(nx, ny, weighted=True, seed=2)
    og = orc.G.from_csr(g)
    part = (np.arange(g.n) * k // g.n).astype(np.int32)
    part[np.random.default_rng(4).random(g.n) < 0.05] = 0
    for iters in (1, 4):
        want = orc.refine_iters(og, part, k, 1.03, 0.75, iters)
        got = jet.refine_iters(g.to("cuda"), torch.from_numpy(part).cuda(), k, 1.03, 0.75, iters)
        assert got["kinds"] == list(want["kinds"])
        assert got["moves"] == list(want["moves"])
        assert np.array_equal(host(got["part"]), want["part"])
        assert got["cut"] == want["cut"]


@pytest.mark.parametrize("n", [8192, 8194, 8450, 130001], ids=["whole_steps", "one_over", "one_step_over", "two_or_more_chunks"])
@pytest.mark.parametrize("tier", TIERS)
def test_contract_dense_rows(jet, graphs, orc, tier, n):
    """Hub rows through the dense accumulator: coarse id counts at and just
    past a multiple of a warp's sweep step (128 ids in 32 bits, 64 in 64) and
    past one chunk of the array; rows that touch every id and a few."""
    gen = torch.Generator().manual_seed(n)
    far = torch.randint(n // 2, n, (4200,), generator=gen)
    u = torch.cat([torch.zeros(n - 1, dtype=torch.long), torch.full((4200,), 2), torch.arange(3, n - 1)])
    v = torch.cat([torch.arange(1, n), far, torch.arange(4, n)])
    g = graphs.from_undirected(n, u, v, torch.randint(1, 9, (u.numel(),), generator=gen)).as_tier(tier)
    m = (np.arange(n) // 2).astype(np.int64 if tier == "biggest" else np.int32)
    nc = (n + 1) // 2
    want = orc.contract(orc.G.from_csr(g), m, nc)
    got = jet.contract(g.to("cuda"), torch.from_numpy(m).cuda(), nc)
    assert np.array_equal(host(got.row), want.row) and np.array_equal(host(got.adj), want.adj)
    assert np.array_equal(host(got.val), want.val) and np.array_equal(host(got.vw), want.vw)


def test_moves_many_rounds(jet, graphs, orc):
    """More moves than the group kernels' grid has groups of four lanes (16
    blocks of 64 on each SM): their loop over the moves takes several rounds. A
    random partition of a 2.4 M-vertex mesh, one iteration of the host-driven
    loop; parts, moves and cut equal the oracle's."""
    g = graphs.grid2d(1621, 1500, weighted=True, seed=2)
    part = np.random.default_rng(4).integers(0, 5, g.n).astype(np.int32)
    want = orc.refine_iters(orc.G.from_csr(g), part, 5, 1.10, 0.75, 1)
    got = jet.refine_iters(g.to("cuda"), torch.from_numpy(part).cuda(), 5, 1.10, 0.75, 1)
    assert want["moves"][0] > 2 * 16 * 64 * torch.cuda.get_device_properties(0).multi_processor_count
    assert got["moves"] == list(want["moves"])
    assert np.array_equal(host(got["part"]), want["part"])
    assert got["cut"] == want["cut"]


@pytest.mark.parametrize("tier", ["i32", "big"])
def test_rebalance_queue_overflow_falls_back(jet, graphs, orc, tier):
    """A 250 x 250 mesh with 90% of its vertices piled into one part: the
    evictions' in-bucket order matters for tens of thousands of candidates,
    more than the ordering block holds, so the iterations take the full sort
    after the classification has already queued moves; the result is still
    the oracle's."""
    g = graphs.grid2d(250, 250, weighted=False).as_tier(tier)
    og = orc.G.from_csr(g)
    prev = jet.set_refine_drivers(jet.DRIVER_ALL)
    try:
        seen = _skewed_runs(jet, orc, g, og, 8, 1.03, 0.9, iters_list=(1, 2, 3, 4))
    finally:
        jet.set_refine_drivers(prev)
    assert 1 in seen


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind,alg,k", [("grid2d", 1, 16), ("grid3d", 1, 32), ("rgg", 1, 8), ("rgg", 2, 16),
                                        ("grid2d", 2, 8), ("rmat", 0, 16), ("star", 0, 8), ("rmat", 1, 32),
                                        ("dense", 0, 64), ("dense", 1, 300)])
def test_full_partition_bit_exact(jet, graphs, orc, tier, kind, alg, k):
    """HEC, pure and 2-hop matching: the whole multilevel run (coarsening,
    Metis, refinement, projection) returns the oracle's partition for the
    same seed."""
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    for seed in (1, 2):
        want, wcut, _ = orc.partition(og, k, alg=alg, imb=1.03, seed=seed)
        cfg = jet.config_t(coarsening_alg=alg, num_parts=k, max_imb_ratio=1.03)
        fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
        part, cut, _ = fn(cfg, g.to("cuda"), seed=seed)
        assert cut == wcut
        assert np.array_equal(host(part), want)


@pytest.mark.parametrize("tier", TIERS)
def test_pstat_and_project_exact(jet, graphs, orc, tier):
    g = make(graphs, "rgg", tier)
    og = orc.G.from_csr(g)
    k = 12
    rng = np.random.default_rng(3)
    part = rng.integers(0, k, g.n).astype(np.int32)
    assert jet.pstat(g.to("cuda"), torch.from_numpy(part).cuda(), k) == orc.pstat(og, part, k).tolist()
    m, nc, _ = orc.coarsen(og, 1, level=2, seed=1, uniform=False)
    cp = rng.integers(0, k, nc).astype(np.int32)
    fine = jet.project(torch.from_numpy(m).cuda(), torch.from_numpy(cp).cuda(), tier)
    assert np.array_equal(host(fine), cp[m])


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("alg", [0, 1, 2])
def test_partition_valid_and_cut_exact(jet, graphs, orc, tier, alg):
    g = make(graphs, "grid2d" if alg != 0 else "rmat", tier)
    og = orc.G.from_csr(g)
    k = 16
    imb = 1.03 if alg != 0 else 1.10
    cfg = jet.config_t(coarsening_alg=alg, num_parts=k, max_imb_ratio=imb)
    fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    part, cut, exp = fn(cfg, g.to("cuda"), seed=2)
    p = host(part)
    assert p.min() >= 0 and p.max() < k
    st = orc.pstat(og, p, k)
    assert st[0] == cut  # reported cut equals the recomputed cut
    opt = (st[5] + k - 1) // k
    assert st[3] <= int(opt * imb)
    assert abs(exp.imb_ratio - st[3] / opt) < 1e-12
    assert len(exp.coarseLevels) >= 1


def test_partition_host_memory_roundtrip(jet, graphs, orc):
    g = make(graphs, "grid2d", "i32")
    cfg = jet.config_t(coarsening_alg=1, num_parts=8)
    part_h, cut_h, _ = jet.partition_host(cfg, g, seed=4)
    assert part_h.device.type == "cpu"
    assert orc.pstat(orc.G.from_csr(g), part_h.numpy(), 8)[0] == cut_h


def test_quality_median_within_two_percent(jet, graphs, ref):
    """Median cut over 8 seeds within 2% of the reference's own code (the
    256x256 grid, k = 32, HEC, unit weights, imbalance 1.03), every GPU
    partition within the imbalance."""
    g = graphs.grid2d(256, 256)
    og = ref.G.from_csr(g)
    cfg = jet.config_t(coarsening_alg=1, num_parts=32, max_imb_ratio=1.03)
    gd = g.to("cuda")
    gpu = []
    for s in range(8):
        part, cut, exp = jet.partition(cfg, gd, seed=s)
        gpu.append(cut)
        assert exp.imb_ratio <= 1.03 + 1e-12
    theirs = [ref.partition(og, 32, alg=1, imb=1.03, seed=s)[1] for s in range(8)]
    assert np.median(gpu) <= 1.02 * np.median(theirs), (gpu, theirs)


def test_invalid_inputs_rejected(jet, graphs):
    g = graphs.grid2d(8, 8).to("cuda")
    bad = graphs.CSRGraph(g.n, g.row.clone(), g.adj.clone(), g.val.clone(), g.vw.clone(), False, "i32")
    bad.adj[3] = 10_000
    with pytest.raises(jet.JetError) as e:
        jet.partition(jet.config_t(num_parts=4), bad)
    assert e.value.code == jet.JET_ERR_INVALID
    bad2 = graphs.CSRGraph(g.n, g.row.clone(), g.adj.clone(), g.val.clone(), g.vw.clone() * 0, False, "i32")
    with pytest.raises(jet.JetError) as e:
        jet.partition(jet.config_t(num_parts=4), bad2)
    assert e.value.code == jet.JET_ERR_INVALID
    with pytest.raises(jet.JetError):
        jet.partition(jet.config_t(num_parts=0), g)


def test_edge_cases(jet, graphs, orc):
    # k = 1: everything in one part, nothing cut
    g = graphs.grid2d(10, 10).to("cuda")
    part, cut, _ = jet.partition(jet.config_t(num_parts=1), g)
    assert cut == 0 and int(part.max()) == 0
    # isolated vertices and a graph smaller than the coarsening cutoff
    u = torch.tensor([0, 1, 2, 5])
    v = torch.tensor([1, 2, 3, 6])
    small = graphs.from_undirected(12, u, v)
    part, cut, _ = jet.partition(jet.config_t(coarsening_alg=1, num_parts=3), small.to("cuda"))
    p = host(part)
    assert p.min() >= 0 and p.max() < 3
    assert orc.pstat(orc.G.from_csr(small), p, 3)[0] == cut


@pytest.mark.parametrize("drivers", ["all", "all_fullsort", "cta_global", "cluster", "coop", "graph", "host", "host_fullsort"])
@pytest.mark.parametrize("tier,kind,k", [("i32", "grid2d", 16), ("big", "rgg", 64), ("biggest", "grid2d", 300),
                                         ("i32", "rgg", 600)])
def test_level_drivers_bit_exact(jet, graphs, orc, drivers, tier, kind, k):
    """Every level-loop driver (one CTA with its state in shared or in global
    memory, one thread-block cluster, cooperative grid kernel, CUDA graph
    with conditional nodes, host loop) returns the oracle's partition on
    graphs whose finer levels exceed the one-CTA bound."""
    q = jet.DRIVER_REB_QUEUE
    mask = {"all": jet.DRIVER_ALL, "all_fullsort": jet.DRIVER_ALL & ~q, "cta_global": jet.DRIVER_CTA | q,
            "cluster": jet.DRIVER_CLUSTER | q, "coop": jet.DRIVER_COOP | jet.DRIVER_GRAPH | q, "graph": jet.DRIVER_GRAPH | q,
            "host": q, "host_fullsort": 0}[drivers]
    g = graphs.grid2d(170, 150, weighted=True, seed=7) if kind == "grid2d" else graphs.rgg(30000, 9.0, seed=5)
    g = g.as_tier(tier)
    og = orc.G.from_csr(g)
    want, wcut, _ = orc.partition(og, k, alg=1, imb=1.03, seed=3)
    prev = jet.set_refine_drivers(mask)
    try:
        cfg = jet.config_t(coarsening_alg=1, num_parts=k, max_imb_ratio=1.03)
        fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
        part, cut, _ = fn(cfg, g.to("cuda"), seed=3)
    finally:
        jet.set_refine_drivers(prev)
    assert cut == wcut
    assert np.array_equal(host(part), want)


@pytest.mark.parametrize("wl", ["grid3d128_k64", "rmat16_k64_2hop", "rmat20_k256_2hop"])
def test_full_size_partition_bit_exact(jet, graphs, orc, wl):
    """Large inputs (2M-vertex mesh; 2^16-vertex R-MAT with 2-hop matching;
    the power-law config's settings -- k = 256, 2-hop, imbalance 1.10, int64
    offsets and weights -- on R-MAT 2^20): the large-level paths drive every
    fine level and the result is still the oracle's partition, run after run."""
    if wl == "grid3d128_k64":
        g = graphs.grid3d(128, 128, 128, weighted=True, seed=1)
        k, alg, imb, fn = 64, 1, 1.03, jet.partition
    elif wl == "rmat16_k64_2hop":
        g = graphs.rmat(16, 8, seed=1, tier="big")
        k, alg, imb, fn = 64, 0, 1.10, jet.partition_big
    else:
        g = graphs.rmat(20, 8, seed=1, tier="big")
        k, alg, imb, fn = 256, 0, 1.10, jet.partition_big
    og = orc.G.from_csr(g)
    want, wcut, _ = orc.partition(og, k, alg=alg, imb=imb, seed=1)
    cfg = jet.config_t(coarsening_alg=alg, num_parts=k, max_imb_ratio=imb)
    gd = g.to("cuda")
    for _ in range(2):
        part, cut, _ = fn(cfg, gd, seed=1)
        assert cut == wcut
        assert np.array_equal(host(part), want)


@pytest.mark.parametrize("tier", ["i32", "big"])
@pytest.mark.parametrize("n", [20001, 1200001])
def test_contract_hub_rows_both_paths(jet, graphs, orc, tier, n):
    """A ring plus a hub of degree 6000: with few coarse vertices the hub row
    goes through the dense shared-memory accumulator, with many (> 8 chunks
    of ids) through the global hash table and the hub-row sort.  Both give
    the oracle's rows exactly."""
    hub_deg = 6000
    u = torch.cat([torch.zeros(hub_deg, dtype=torch.long), torch.arange(1, n - 1)])
    v = torch.cat([torch.arange(1, hub_deg + 1) * ((n - 1) // hub_deg), torch.arange(2, n)])
    w = torch.randint(1, 9, (u.numel(),), generator=torch.Generator().manual_seed(n))
    g = graphs.from_undirected(n, u, v, w).as_tier(tier)
    og = orc.G.from_csr(g)
    m, nc, _ = orc.coarsen(og, 1, level=2, seed=3, uniform=False)
    want = orc.contract(og, m, nc)
    got = jet.contract(g.to("cuda"), torch.from_numpy(m).cuda(), nc)
    assert np.array_equal(host(got.row), want.row)
    assert np.array_equal(host(got.adj), want.adj)
    assert np.array_equal(host(got.val), want.val)
    assert np.array_equal(host(got.vw), want.vw)


@pytest.mark.parametrize("tier", TIERS)
def test_contract_wide_id_range_rows(jet, graphs, orc, tier):
    """Coarse rows of 257 to 4096 member edges whose neighbours spread over
    more coarse ids than a shared-memory bitmap covers (about 644,000 ids): the
    per-row radix sort path.  Rows equal the oracle's exactly."""
    n = 1_300_000
    gen = torch.Generator().manual_seed(9)
    spokes = torch.arange(0, 600, 2) * 2131  # 300 vertices spread over the range
    deg = torch.randint(300, 3000, (spokes.numel(),), generator=gen)
    u = torch.cat([spokes.repeat_interleave(deg), torch.arange(n)])
    v = torch.cat([torch.randint(0, n, (int(deg.sum()),), generator=gen), (torch.arange(n) + 1) % n])
    a, b = torch.minimum(u, v), torch.maximum(u, v)
    pairs = torch.unique((a * n + b)[a != b])
    g = graphs.from_undirected(n, pairs // n, pairs % n, torch.randint(1, 9, (pairs.numel(),), generator=gen)).as_tier(tier)
    og = orc.G.from_csr(g)
    # pairs of consecutive vertices, and groups of 16 in the last 1% of ids
    m = np.arange(n, dtype=np.int64) // 2
    tail = n - n // 100
    m[tail:] = tail // 2 + (np.arange(n - tail) // 16)
    nc = int(m.max()) + 1
    m = m.astype(np.int64 if tier == "biggest" else np.int32)
    want = orc.contract(og, m, nc)
    got = jet.contract(g.to("cuda"), torch.from_numpy(m).cuda(), nc)
    assert np.array_equal(host(got.row), want.row)
    assert np.array_equal(host(got.adj), want.adj)
    assert np.array_equal(host(got.val), want.val)
    assert np.array_equal(host(got.vw), want.vw)


@pytest.mark.parametrize("tier", ["big", "biggest"])
def test_wide_weights_exact(jet, graphs, orc, tier):
    """Edge weights of 2^26 to 2^27 (total far above 2^31): the shared-memory
    accumulators must take the 64-bit path, not the 32-bit one.  Tables,
    contraction and refinement iterations equal the oracle's."""
    g = make(graphs, "dense", "i32")
    gen = torch.Generator().manual_seed(12)
    und = torch.randint(1 << 26, 1 << 27, (g.nnz,), generator=gen, dtype=torch.int64)
    # symmetric weights: the weight of (u, v) and (v, u) from the smaller endpoint's edge index
    src = torch.repeat_interleave(torch.arange(g.n), (g.row[1:] - g.row[:-1]).long())
    dst = g.adj.long()
    key = torch.minimum(src, dst) * g.n + torch.maximum(src, dst)
    _, inv = torch.unique(key, return_inverse=True)
    w = und[inv]
    g = graphs.CSRGraph(g.n, g.row, g.adj, w, g.vw.to(torch.int64), False, "i32").as_tier(tier)
    og = orc.G.from_csr(g)
    assert int(w.sum()) > (1 << 31)
    for k in (64, 300):
        part = (np.arange(g.n) % k).astype(np.int32)
        off, ent, val, size = orc.conn_build(og, part, k)
        goff, gent, gval, gsize = jet.conn_build(g.to("cuda"), torch.from_numpy(part).cuda(), k)
        assert np.array_equal(host(gsize), size)
        assert table_multisets(host(goff), host(gent), host(gval), host(gsize)) == table_multisets(off, ent, val, size)
    m = (np.arange(g.n) // 2).astype(np.int64 if tier == "biggest" else np.int32)
    want = orc.contract(og, m, g.n // 2)
    got = jet.contract(g.to("cuda"), torch.from_numpy(m).cuda(), g.n // 2)
    assert np.array_equal(host(got.row), want.row) and np.array_equal(host(got.adj), want.adj)
    assert np.array_equal(host(got.val), want.val)
    part = (np.arange(g.n) % 64).astype(np.int32)
    part[: g.n // 3] = 0  # badly unbalanced: rebalancing iterations with large updates
    for iters in (1, 3, 6):
        want = orc.refine_iters(og, part, 64, 1.03, 0.75, iters)
        got = jet.refine_iters(g.to("cuda"), torch.from_numpy(part).cuda(), 64, 1.03, 0.75, iters)
        assert got["kinds"] == list(want["kinds"])
        assert np.array_equal(host(got["part"]), want["part"])
        assert got["cut"] == want["cut"]
        gm = table_multisets(host(got["off"]), host(got["ent"]), host(got["val"]), host(got["size"]))
        assert gm == table_multisets(want["off"], want["ent"], want["val"], want["size"])


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind,alg,k", [("grid2d", 1, 16), ("rgg", 2, 8), ("rmat", 0, 16)])
def test_ultra_settings_partition_bit_exact(jet, graphs, orc, tier, kind, alg, k):
    """ultra_settings (src/jet_refiner.hpp:1090-1093): the filter ratio steps
    from 0.85 down by 0.05 with 12 patience iterations each; the whole run
    equals the oracle's."""
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    imb = 1.10 if alg == 0 else 1.03
    want, wcut, _ = orc.partition(og, k, alg=alg, imb=imb, seed=3, ultra=True)
    plain, pcut, _ = orc.partition(og, k, alg=alg, imb=imb, seed=3)
    cfg = jet.config_t(coarsening_alg=alg, num_parts=k, max_imb_ratio=imb, ultra_settings=1)
    fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    part, cut, exp = fn(cfg, g.to("cuda"), seed=3)
    assert cut == wcut
    assert np.array_equal(host(part), want)
    # the schedule runs more LP iterations than the default one
    assert sum(cl.lpIterations for cl in exp.coarseLevels) > 0


def _tie_free(og, tier):
    """64-bit symmetric pseudo-random weights below 2^30: no two parts are
    ever equally connected, so the reference's first-slot tie rule and the
    lowest-part-id rule here cannot differ."""
    n = og.n
    rid = np.repeat(np.arange(n, dtype=np.int64), np.diff(og.row))
    a = np.minimum(rid, og.adj).astype(np.uint64)
    b = np.maximum(rid, og.adj).astype(np.uint64)
    x = a * np.uint64(0x9E3779B97F4A7C15) ^ b * np.uint64(0xC2B2AE3D27D4EB4F)
    x ^= x >> np.uint64(29)
    w = (x % np.uint64(1 << 30)).astype(np.int64) + 1
    od, ed, wd = {"big": (np.int32, np.int64, np.int64), "biggest": (np.int64, np.int64, np.int64)}[tier]
    return og.row.astype(ed), og.adj.astype(od), w.astype(wd), og.vw.astype(wd)


@pytest.mark.parametrize("tier", ["big", "biggest"])
@pytest.mark.parametrize("kind,k", [("grid3d", 16), ("rgg", 32), ("rmat", 16)])
def test_gpu_matches_reference_directly(jet, graphs, orc, ref, tier, kind, k):
    """The GPU path against the reference's own code (oracle/_ref, Serial):
    pstat, connectivity tables, contraction of the GPU's own coarsening map,
    and ten refinement iterations from a skewed start (LP, weak and strong
    rebalancing) with weights under which no two parts tie."""
    base = make(graphs, kind, tier)
    row, adj, val, vw = _tie_free(orc.G.from_csr(base), tier)
    g = graphs.CSRGraph(base.n, torch.from_numpy(row), torch.from_numpy(adj), torch.from_numpy(val),
                        torch.from_numpy(vw), False, tier)
    rg = ref.G(row, adj, val, vw, False)
    gd = g.to("cuda")
    rng = np.random.default_rng(2)
    part = rng.integers(0, k, g.n).astype(np.int32)
    pd = torch.from_numpy(part).cuda()
    assert jet.pstat(gd, pd, k) == ref.pstat(rg, part, k).tolist()
    goff, gent, gval, gsize = jet.conn_build(gd, pd, k)
    r = ref.conn_build(rg, part, k)
    assert np.array_equal(host(goff), r[0]) and np.array_equal(host(gsize), r[3])
    assert table_multisets(host(goff), host(gent), host(gval), host(gsize)) == table_multisets(*r)
    cmap, nc, _ = jet.coarsen_map(gd, 1, level=1, seed=1)
    c = jet.contract(gd, cmap, nc)
    rc = ref.contract(rg, host(cmap), nc)
    assert np.array_equal(host(c.row), rc.row) and np.array_equal(host(c.vw), rc.vw)
    ra, rv = sorted_rows(rc.row, rc.adj, rc.val)
    assert np.array_equal(host(c.adj), ra) and np.array_equal(host(c.val), rv)
    skew = part.copy()
    skew[rng.random(g.n) < 0.6] = 0
    imb = 1.10 if kind == "rmat" else 1.03
    want = ref.refine_iters(rg, skew, k, imb, 0.75, 10)
    got = jet.refine_iters(gd, torch.from_numpy(skew).cuda(), k, imb, 0.75, 10)
    assert got["kinds"] == list(want["kinds"])
    assert got["moves"] == list(want["moves"])
    assert np.array_equal(host(got["part"]), want["part"])
    assert np.array_equal(host(got["sizes"]), want["sizes"])
    assert got["cut"] == want["cut"]


def test_class_profiling_pass_leaves_results_unchanged(jet, graphs, orc):
    """The profiling pass (every level on the host-driven loop with the
    rebalance queue, event brackets per kernel class, device-side counts for the byte model) returns the same
    partition as a normal call, and accounts time and bytes to the classes
    that ran."""
    g = graphs.grid3d(40, 40, 30, weighted=True, seed=4)
    og = orc.G.from_csr(g)
    cfg = jet.config_t(coarsening_alg=1, num_parts=16, max_imb_ratio=1.03)
    want, wcut, _ = orc.partition(og, 16, alg=1, imb=1.03, seed=2)
    prev = jet.set_refine_drivers(jet.DRIVER_REB_QUEUE)
    try:
        jet.prof_enable(True)
        part, cut, _ = jet.partition(cfg, g.to("cuda"), seed=2)
        torch.cuda.synchronize()
        prof = jet.prof_read()
        jet.prof_enable(False)
    finally:
        jet.set_refine_drivers(prev)
    assert cut == wcut and np.array_equal(host(part), want)
    for c in ("conn_build", "lp_select", "afterburn", "apply", "cut_after"):
        assert prof[c]["launches"] > 0 and prof[c]["ms"] > 0 and prof[c]["bytes"] > 0, (c, prof[c])
    assert prof["update"]["launches"] > 0


def test_rmat24_k256_full_size_equals_oracle_fixture(jet, graphs):
    """The power-law config at full size -- R-MAT 2^24, k = 256, 2-hop,
    imbalance 1.10, int64 offsets and weights -- against the oracle's
    partition recorded in tests/golden/rmat24_k256_oracle.json (made by
    tests/golden/make_rmat24_fixture.py; the oracle needs about 12 minutes on
    one host thread).  The graph is generated on the GPU by the same
    counter-based generator and checked against the fixture's digests."""
    import hashlib
    import json
    import os
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "rmat24_k256_oracle.json")
    if not os.path.exists(path):
        pytest.skip("fixture not generated")
    want = json.load(open(path))
    g = graphs.rmat(24, 8, seed=1, tier="big", device="cuda")
    assert hashlib.sha256(host(g.row).tobytes()).hexdigest() == want["row_sha256"]
    assert hashlib.sha256(host(g.adj).tobytes()).hexdigest() == want["adj_sha256"]
    cfg = jet.config_t(coarsening_alg=0, num_parts=256, max_imb_ratio=1.10)
    part, cut, exp = jet.partition_big(cfg, g, seed=1)
    assert cut == want["cut"]
    assert hashlib.sha256(host(part).astype(np.int32).tobytes()).hexdigest() == want["part_sha256"]
    assert exp.imb_ratio <= 1.10 + 1e-12


def test_inputs_still_being_written_on_the_default_stream(jet, graphs):
    """A call on torch's default stream waits for the work queued there: the
    graph's arrays are filled behind a long kernel, with no synchronisation
    before the call."""
    g = make(graphs, "grid2d", "i32").to("cuda")
    cfg = jet.config_t(coarsening_alg=1, num_parts=8, max_imb_ratio=1.03)
    want, cut, _ = jet.partition(cfg, g, seed=5)
    late = graphs.CSRGraph(g.n, torch.zeros_like(g.row), torch.zeros_like(g.adj), torch.ones_like(g.val),
                           torch.ones_like(g.vw), g.uniform, g.tier)
    torch.cuda.synchronize()
    torch.cuda._sleep(50_000_000)  # about 25 ms
    late.row.copy_(g.row)
    late.adj.copy_(g.adj)
    late.val.copy_(g.val)
    late.vw.copy_(g.vw)
    got, got_cut, _ = jet.partition(cfg, late, seed=5)
    assert got_cut == cut and torch.equal(got, want)


@pytest.mark.parametrize("alg", [0, 1, 2])
@pytest.mark.parametrize("tier", ["big", "biggest"])
@pytest.mark.parametrize("kind,k", [("grid2d", 7), ("rgg", 16), ("rmat", 16), ("star", 8), ("dense", 300)])
def test_64_bit_tiers_in_32_bits(jet, graphs, tier, kind, k, alg, tmp_path, monkeypatch):
    """A 64-bit-tier graph whose sums fit 32 bits is partitioned in 32 bits;
    a run that dumps its hierarchy keeps the tier's own types.  Both give the
    same partition, with vertex weights and from host memory too."""
    monkeypatch.chdir(tmp_path)
    g = make(graphs, kind, tier)
    g.vw = torch.randint(1, 6, (g.n,), generator=torch.Generator().manual_seed(3)).to(g.vw.dtype)
    fn = {"big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    hfn = {"big": jet.partition_host_big, "biggest": jet.partition_host_biggest}[tier]
    for ultra in (False, True):
        a = dict(coarsening_alg=alg, num_parts=k, max_imb_ratio=1.05, ultra_settings=ultra)
        part, cut, _ = fn(jet.config_t(**a), g.to("cuda"), seed=3)
        want, wcut, _ = fn(jet.config_t(dump_coarse=True, **a), g.to("cuda"), seed=3)
        assert cut == wcut and torch.equal(part, want)
        for verbose in (False, True):  # without it the wide copies are given back before the partition
            hpart, hcut, _ = hfn(jet.config_t(verbose=verbose, **a), g, seed=3)
            assert hcut == wcut and torch.equal(hpart, want.cpu())


@pytest.mark.parametrize("tier", ["big", "biggest"])
@pytest.mark.parametrize("which,off", [("edges", -2), ("edges", 0), ("edges", 4), ("vertices", -1), ("vertices", 0),
                                       ("single", 0)])
def test_32_bit_rule_at_its_edges(jet, graphs, orc, tier, which, off):
    """Weight sums just below, at and above what the 32-bit form takes (edge
    sum 2^30, vertex sum 2^28, one weight of 2^31): all equal the oracle."""
    g = graphs.grid2d(40, 30, weighted=True, seed=8).as_tier(tier)
    row, adj = g.row.long(), g.adj.long()
    src = torch.repeat_interleave(torch.arange(g.n), row[1:] - row[:-1])

    def set_edge(u, v, w):
        g.val[(src == u) & (adj == v)] = w
        g.val[(src == v) & (adj == u)] = w

    if which == "edges":
        g.val = g.val * ((1 << 30) // int(g.val.sum()))
        u, v = 0, int(adj[0])
        set_edge(u, v, int(g.val[0]) + ((1 << 30) + off - int(g.val.sum())) // 2)
        assert int(g.val.sum()) == (1 << 30) + off
    elif which == "vertices":
        g.vw = g.vw * ((1 << 28) // g.n)
        g.vw[17] += (1 << 28) + off - int(g.vw.sum())
        assert int(g.vw.sum()) == (1 << 28) + off
    else:
        set_edge(0, int(adj[0]), 1 << 31)
    og = orc.G.from_csr(g)
    fn = {"big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    for alg in (0, 1):
        want, wcut, _ = orc.partition(og, 8, alg=alg, imb=1.03, seed=2)
        part, cut, _ = fn(jet.config_t(coarsening_alg=alg, num_parts=8, max_imb_ratio=1.03), g.to("cuda"), seed=2)
        assert cut == wcut and np.array_equal(host(part), want)


@pytest.mark.parametrize("tier", TIERS)
@pytest.mark.parametrize("kind", ["grid2d", "grid3d", "rgg", "rmat", "star", "dense"])
@pytest.mark.parametrize("k", [2, 31, 33, 700, 5000])
def test_pstat_row_classes(jet, graphs, orc, tier, kind, k):
    """Statistics of rows in every class (register compare, warp and block
    bitmaps; histograms in shared and in global memory), of slabs and of
    scattered parts; a part id out of range is refused."""
    g = make(graphs, kind, tier)
    og = orc.G.from_csr(g)
    rng = np.random.default_rng(k)
    slabs = (np.arange(g.n) * min(k, g.n) // g.n).astype(np.int32)
    for part in (rng.integers(0, k, g.n).astype(np.int32), slabs):
        assert jet.pstat(g.to("cuda"), torch.from_numpy(part).cuda(), k) == orc.pstat(og, part, k).tolist()
    part[g.n // 2] = k
    with pytest.raises(jet.JetError):
        jet.pstat(g.to("cuda"), torch.from_numpy(part).cuda(), k)


def _partition_with(jet, mask, tier, cfg, g, seed):
    prev = jet.set_refine_drivers(mask)
    try:
        fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
        part, cut, _ = fn(cfg, g.to("cuda"), seed=seed)
    finally:
        jet.set_refine_drivers(prev)
    return host(part), cut


@pytest.mark.parametrize("drivers", ["all", "cluster", "coop", "host"])
@pytest.mark.parametrize("tier,kind,k", [("i32", "grid3d", 513), ("i32", "rgg", 1024), ("i32", "rgg", 1025), ("big", "rgg", 700),
                                         ("i32", "hubs", 600)])
def test_many_parts_on_the_persistent_loops(jet, graphs, orc, drivers, tier, kind, k):
    """k above a warp table's 512 entries: levels of short rows run on the
    persistent loops with hash tables of twice the largest row ("hubs": a
    graph with longer rows, which needs k entries and keeps the other
    drivers); all equal the oracle."""
    q = jet.DRIVER_REB_QUEUE
    mask = {"all": jet.DRIVER_ALL, "cluster": jet.DRIVER_CLUSTER | q, "coop": jet.DRIVER_COOP | jet.DRIVER_GRAPH | q,
            "host": q}[drivers]
    if kind == "grid3d":
        g = graphs.grid3d(30, 30, 31, weighted=True, seed=2)
    elif kind == "rgg":
        g = graphs.rgg(30000, 9.0, seed=5)
    else:
        gen = torch.Generator().manual_seed(4)
        n = 20000
        u = torch.cat([torch.arange(n), torch.arange(20).repeat_interleave(300)])
        v = torch.cat([(torch.arange(n) + 1) % n, torch.randint(0, n, (6000,), generator=gen)])
        a, b = torch.minimum(u, v), torch.maximum(u, v)
        pairs = torch.unique((a * n + b)[a != b])
        g = graphs.from_undirected(n, pairs // n, pairs % n, torch.randint(1, 9, (pairs.numel(),), generator=gen))
    g = g.as_tier(tier)
    cfg = jet.config_t(coarsening_alg=1, num_parts=k, max_imb_ratio=1.05)
    want, wcut, _ = orc.partition(orc.G.from_csr(g), k, alg=1, imb=1.05, seed=4)
    part, cut = _partition_with(jet, mask, tier, cfg, g, 4)
    assert cut == wcut and np.array_equal(part, want)


@pytest.mark.parametrize("drivers", ["all", "cta_global", "cluster", "coop", "graph", "host_fullsort"])
@pytest.mark.parametrize("tier,k", [("big", 64), ("biggest", 600)])
def test_level_drivers_64_bit(jet, graphs, orc, drivers, tier, k):
    """The 64-bit instantiations of the level drivers: edge weights whose sum
    does not fit 32 bits."""
    q = jet.DRIVER_REB_QUEUE
    mask = {"all": jet.DRIVER_ALL, "cta_global": jet.DRIVER_CTA | q, "cluster": jet.DRIVER_CLUSTER | q,
            "coop": jet.DRIVER_COOP | jet.DRIVER_GRAPH | q, "graph": jet.DRIVER_GRAPH | q, "host_fullsort": 0}[drivers]
    g = graphs.rgg(20000, 9.0, seed=5).as_tier(tier)
    g.val = g.val * 100003
    assert int(g.val.sum()) > 1 << 31
    cfg = jet.config_t(coarsening_alg=0, num_parts=k, max_imb_ratio=1.03)
    want, wcut, _ = orc.partition(orc.G.from_csr(g), k, alg=0, imb=1.03, seed=3)
    part, cut = _partition_with(jet, mask, tier, cfg, g, 3)
    assert cut == wcut and np.array_equal(part, want)


def test_rows_that_end_at_the_largest_offset(jet, graphs):
    """An i32 graph of 2^31 - 1 entries: cursors over its last row step past
    the largest 32-bit offset. Statistics, tables and contraction equal counts
    of the rows' entries (entry j names vertex j mod 1009)."""
    m, per, v, k, members = 2 ** 31 - 1, 16384, 1009, 64, 32
    n = (m + 1) // per
    dev = "cuda"
    row = torch.arange(n + 1, device=dev, dtype=torch.int64) * per
    row[n] = m
    adj = torch.arange(m, device=dev, dtype=torch.int32).remainder_(v)
    g = graphs.CSRGraph(n, row.to(torch.int32), adj, torch.ones(m, dtype=torch.int32, device=dev),
                        torch.ones(n, dtype=torch.int32, device=dev), True, "i32")
    part = (torch.arange(n, device=dev, dtype=torch.int32) * 7) % k
    # entries of row i that name x: whole periods, and the rest from the row's first id on
    first, length = (row[:-1] % v)[:, None], (row[1:] - row[:-1])[:, None]
    ids = torch.arange(v, device=dev)[None, :]
    times = (length // v + ((ids - first) % v < length % v)).to(torch.int32)
    to_part = torch.zeros(n, k, dtype=torch.int32, device=dev).index_add_(1, part[:v].long(), times)
    own = to_part.gather(1, part[:, None].long())[:, 0]
    out = length[:, 0] - own
    per_part = torch.zeros(k, dtype=torch.int64, device=dev).index_add_(0, part.long(), out)
    sizes = torch.bincount(part, minlength=k)
    want = [int(out.sum()) // 2, int(per_part.max()), int((to_part > 0).sum() - (own > 0).sum()), int(sizes.max()), int(sizes.min()), n]
    assert jet.pstat(g, part, k) == want
    assert jet.pstat_noalloc(g, part, k) == want

    off, ent, val, size = jet.conn_build(g, part, k)
    # every row has every part, so tables are direct: k slots, a part at its own
    assert torch.equal(off, torch.arange(n + 1, device=dev, dtype=torch.int32) * k) and bool((size == k).all())
    assert torch.equal(ent.view(n, k), torch.arange(k, device=dev, dtype=torch.int32).expand(n, k))
    assert torch.equal(val.view(n, k), to_part)
    del off, ent, val, size, to_part

    nc = n // members
    cmap = torch.arange(n, device=dev, dtype=torch.int32) // members
    c = jet.contract(g, cmap, nc)
    coarse = torch.zeros(nc, (v - 1) // members + 1, dtype=torch.int32, device=dev)
    coarse.index_add_(1, cmap[:v].long(), times.view(nc, members, v).sum(1, dtype=torch.int32))
    at = torch.arange(coarse.shape[1], device=dev)
    coarse[at, at] = 0
    keep = coarse > 0
    assert torch.equal(c.row[1:] - c.row[:-1], keep.sum(1, dtype=torch.int32))
    assert torch.equal(c.adj, keep.nonzero()[:, 1].to(torch.int32)) and torch.equal(c.val, coarse[keep])
    assert bool((c.vw == members).all())
