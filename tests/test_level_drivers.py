"""Which level loop a level goes to: the bounds between the drivers, and what
each loop reserves. Results do not depend on it; the parity tests cover those."""
import ctypes
import json
import os
import subprocess
import sys

import pytest
import torch

from conftest import ROOT

CHILD = """
import json, sys
sys.path.insert(0, sys.argv[1])
from conftest import load_pkg
jet = load_pkg()
g = jet.graphs.grid2d(400, 250, weighted=True, seed=3, device="cuda")
jet.prof_phases(True)
part, cut, _ = jet.partition(jet.config_t(coarsening_alg=1, num_parts=16), g, seed=2)
print(json.dumps([cut, [d for d, p in jet.prof_phases(False).items() if p]]))
"""


def _drivers(**env):
    """Cut of one partition in a process with these variables, and the
    persistent loops that ran."""
    e = {k: v for k, v in os.environ.items() if not k.startswith("JET_")}
    e.update(env)
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "tests")], env=e, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    cut, ran = json.loads(r.stdout.splitlines()[-1])
    return cut, set(ran)


@pytest.mark.gpu
def test_a_bound_of_zero_leaves_a_driver_out():
    """100,000 vertices: the grid takes the finest levels, the cluster the
    middle ones; a bound of 0 (or below) leaves that loop without levels."""
    cut, ran = _drivers()
    assert ran == {"cta", "cluster", "coop"}
    for value in ("0", "-1"):
        assert _drivers(JET_COOP_MAX_N=value) == (cut, {"cta", "cluster"})
        assert _drivers(JET_CLUSTER_MAX_N=value) == (cut, {"cta", "coop"})
    assert _drivers(JET_COOP_MAX_N="0", JET_CLUSTER_MAX_N="0") == (cut, {"cta"})
    assert _drivers(JET_COOP_MAX_N="1000000") == (cut, {"cta", "cluster", "coop"})


# what a cluster's or grid's block has for the bucket offsets: 160 KiB with
# 32-bit weights, what its other shared memory leaves with 64-bit ones
@pytest.mark.parametrize("tier,k,budget,n,want", [
    (0, 64, 160 << 10, 3971, 50 * 64 + 1), (0, 64, 160 << 10, 1 << 20, 50 * 64 * 5 + 1), (0, 256, 160 << 10, 60000, 50 * 256 + 1),
    (0, 819, 160 << 10, 60000, 50 * 819 + 1), (0, 820, 160 << 10, 60000, 0), (1, 205, 150 << 10, 60000, 50 * 205 + 1),
    (1, 256, 150 << 10, 1 << 18, 50 * 256 + 1), (1, 256, 150 << 10, 1 << 20, 0), (2, 384, 150 << 10, 60000, 0),
    (2, 383, 150 << 10, 60000, 50 * 383 + 1)])
def test_bucket_offsets_reserved_for_the_level(jet, tier, k, budget, n, want):
    """The reservation follows the level's own size, whatever the largest
    level that the loop could take."""
    f = jet.load().jet_test_bucket_copy
    f.restype = ctypes.c_int64
    assert f(tier, ctypes.c_int64(n), ctypes.c_int32(k), ctypes.c_int64(budget)) == want


@pytest.mark.gpu
@pytest.mark.parametrize("tier", ["big", "biggest"])
@pytest.mark.parametrize("k", [380, 400, 409, 512])
def test_wide_weights_and_many_parts_keep_the_persistent_loops(jet, graphs, orc, tier, k):
    """64-bit weights: bucket offsets of 385 to 409 parts fit 160 KiB but not
    what the kernel's other shared memory leaves; such levels run on the
    cluster and the grid all the same, with the grid-wide scan."""
    g = graphs.rgg(90000, 9.0, seed=5).as_tier(tier)
    g.val = g.val * (2 ** 31 // int(g.val.sum()) + 1)
    assert int(g.val.sum()) > 2 ** 31
    want, wcut, _ = orc.partition(orc.G.from_csr(g), k, alg=1, imb=1.05, seed=4)
    fn = {"big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    jet.prof_phases(True)
    part, cut, _ = fn(jet.config_t(coarsening_alg=1, num_parts=k, max_imb_ratio=1.05), g.to("cuda"), seed=4)
    ran = {d for d, p in jet.prof_phases(False).items() if p}
    assert {"cluster", "coop"} <= ran
    assert cut == wcut and (part.cpu().numpy() == want).all()


@pytest.mark.parametrize("n,m,max_deg,n_hub,want", [
    (10000, 60000, 60, 0, 0), (10000, 60000, 5000, 1, 0),                          # a mesh; hubs among short rows
    (10000, 139999, 5000, 1, 0), (10000, 140000, 5000, 1, 1),                      # hubs and a mean of 14
    (10000, 320000, 127, 0, 0), (10000, 320000, 128, 0, 1),                        # longest row of four times the mean
    (10000, 319999, 4000, 0, 0),                                                   # a mean below 32
    (513, 16416, 60, 0, 0), (512, 16384, 60, 0, 1), (200000, 26000000, 300, 0, 0)  # small and dense; large and dense
])
def test_levels_of_long_rows(jet, n, m, max_deg, n_hub, want):
    """The rule that gives rows groups of lanes, at its edges."""
    assert jet.load().jet_test_long_rows(*(ctypes.c_int64(x) for x in (n, m, max_deg, n_hub))) == want


@pytest.fixture(scope="module")
def long_row_graphs(graphs, orc):
    """Graphs with hub rows or long uneven ones, and the oracle's partitions, made once each."""
    made = {}

    def get(tier, wide, kind, k, alg):
        key = (tier, wide, kind, k, alg)
        if key in made:
            return made[key]
        if kind == "rmat":
            g = graphs.rmat(16, 8, seed=4, tier=tier)
            assert int((g.row[1:] - g.row[:-1]).max()) > 4096
        elif kind == "star":  # short rows and one hub
            n = 9000
            u = torch.cat([torch.zeros(5000, dtype=torch.long), torch.arange(1, n - 1)])
            v = torch.cat([torch.arange(1, 5001), torch.arange(2, n)])
            g = graphs.from_undirected(n, u, v, torch.randint(1, 5, (u.numel(),), generator=torch.Generator().manual_seed(1)))
        else:  # every row a tenth of the vertices, no hub
            n = 1500
            a, b = torch.randint(0, n, (2, 110000), generator=torch.Generator().manual_seed(2))
            pairs = torch.unique((torch.minimum(a, b) * n + torch.maximum(a, b))[a != b])
            g = graphs.from_undirected(n, pairs // n, pairs % n, pairs % 8 + 1)
        g = g.as_tier(tier)
        if wide:
            g.val = g.val * (2 ** 31 // int(g.val.sum()) + 1)
        want, cut, _ = orc.partition(orc.G.from_csr(g), k, alg=alg, imb=1.05, seed=3)
        made[key] = g, want, cut
        return made[key]
    return get


@pytest.mark.gpu
@pytest.mark.parametrize("drivers", ["all", "cta", "cluster", "coop"])
@pytest.mark.parametrize("tier,wide", [("i32", False), ("big", True), ("biggest", True)])
@pytest.mark.parametrize("kind,k,alg", [("rmat", 48, 0), ("rmat", 40, 1), ("star", 8, 0), ("dense", 24, 1)])
def test_long_rows_on_the_persistent_loops(jet, long_row_graphs, drivers, tier, wide, kind, k, alg):
    """Levels with hub rows and of long uneven rows, in 32 bits and with
    weight sums above 2^31, on each loop: equal to the oracle."""
    g, want, wcut = long_row_graphs(tier, wide, kind, k, alg)
    assert not wide or int(g.val.sum()) > 2 ** 31
    q = jet.DRIVER_REB_QUEUE
    mask = {"all": jet.DRIVER_ALL, "cta": jet.DRIVER_CTA | q, "cluster": jet.DRIVER_CLUSTER | q,
            "coop": jet.DRIVER_COOP | jet.DRIVER_GRAPH | q}[drivers]
    fn = {"i32": jet.partition, "big": jet.partition_big, "biggest": jet.partition_biggest}[tier]
    prev = jet.set_refine_drivers(mask)
    try:
        part, cut, _ = fn(jet.config_t(coarsening_alg=alg, num_parts=k, max_imb_ratio=1.05), g.to("cuda"), seed=3)
    finally:
        jet.set_refine_drivers(prev)
    assert cut == wcut and (part.cpu().numpy() == want).all()


@pytest.mark.gpu
@pytest.mark.parametrize("scale,degree,tier,wide,loops", [
    (18, 8, "i32", False, {"coop"}), (19, 8, "i32", False, set()), (18, 10, "i32", False, {"coop"}),
    (19, 3, "i32", False, {"coop"}), (19, 6, "i32", False, {"coop"}), (18, 8, "big", True, {"coop"}),
    (18, 10, "big", True, set()), (19, 3, "big", True, {"coop"}), (19, 6, "big", True, set())])
def test_large_levels_of_long_rows_stay_level_graphs(jet, graphs, scale, degree, tier, wide, loops):
    """Power-law levels above 262,144 vertices, and with 64-bit weights above
    2^22 entries, are faster as level graphs than on the grid; those of mostly
    short rows only with 64-bit weights and above 2^22 entries."""
    g = graphs.rmat(scale, degree, seed=4, tier=tier, device="cuda").as_tier(tier)
    assert (g.nnz > 1 << 22) == (degree == 10 or (scale, degree) in ((19, 6), (19, 8)))
    assert int((g.row[1:] - g.row[:-1]).max()) > 4096
    if wide:
        g.val = g.val * (2 ** 31 // int(g.val.sum()) + 1)
    part = torch.randint(0, 16, (g.n,), generator=torch.Generator().manual_seed(1), dtype=torch.int32).cuda()
    jet.prof_phases(True)
    jet.refine_level(g, part, 16, 1.10)
    assert {d for d, p in jet.prof_phases(False).items() if p} == loops


@pytest.mark.gpu
@pytest.mark.parametrize("tier,wide", [("i32", False), ("big", True)])
def test_row_walk_many_rounds(jet, graphs, orc, tier, wide):
    """A level of the persistent grid whose first iteration has more moves
    than 32 for each of its warps: the walks over the rows of candidates and
    moves take several rounds. A random partition of a 700 x 700 mesh; the
    refined level equals the oracle's."""
    g = graphs.grid2d(700, 700, weighted=True, seed=2).as_tier(tier)
    if wide:
        g.val = g.val * (2 ** 31 // int(g.val.sum()) + 1)
    og = orc.G.from_csr(g)
    part = torch.randint(0, 5, (g.n,), generator=torch.Generator().manual_seed(4), dtype=torch.int32)
    warps = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    assert orc.refine_iters(og, part.numpy(), 5, 1.10, 0.75, 1)["moves"][0] > 32 * warps
    want, wcut, _ = orc.refine_level(og, part.numpy(), 5, 1.10)
    prev = jet.set_refine_drivers(jet.DRIVER_COOP | jet.DRIVER_GRAPH | jet.DRIVER_REB_QUEUE)
    try:
        jet.prof_phases(True)
        got, cut, _ = jet.refine_level(g.to("cuda"), part.cuda(), 5, 1.10)
        ran = {d for d, p in jet.prof_phases(False).items() if p}
    finally:
        jet.set_refine_drivers(prev)
    assert ran == {"coop"}
    assert cut == wcut and (got.cpu().numpy() == want).all()
