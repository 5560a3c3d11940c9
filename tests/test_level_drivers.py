"""Which level loop a level goes to: the bounds between the drivers, and what
each loop reserves. Results do not depend on it; the parity tests cover those."""
import json
import os
import subprocess
import sys

import pytest

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
