"""The degeneracy peel where its step sizes change: graphs peeled by one CTA
alone, fronts and scans just past its limits, hubs whose rows are split over
many warps, levels without vertices, windows of the bucket left empty, and paths,
whose sub-rounds of two vertices are one CTA's work for far longer than one
stretch of it."""
import numpy as np
import pytest

import kcgpu_b200 as kc
from oracle.oracle import OracleGraph
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _star(leaves: int):
    return np.zeros(leaves, np.uint32), np.arange(1, leaves + 1, dtype=np.uint32), leaves + 1


def _complete(n: int):
    s, d = G.complete(n)
    return s, d, n


def _path(n: int):
    a = np.arange(n - 1, dtype=np.uint32)
    return a, a + 1, n


CASES = {
    "one_cta": lambda: kc.gen_rmat(12, 8.0, seed=3).arrays(),
    "scan_limit": lambda: kc.gen_er(8193, 0.002, 5).arrays(),
    "front_limit": lambda: G.disjoint_union([_complete(3)] * 342),
    "star_past_edge_limit": lambda: _star(16_400),
    "star_hub_and_core": lambda: G.disjoint_union([_star(40_000), _complete(150), _star(1_023), _star(1_025)]),
    "empty_windows": lambda: G.disjoint_union([_complete(400), _complete(90), _complete(7), _star(9_000)]),
    "one_cta_star": lambda: _star(4_095),
    "several_ctas_star": lambda: _star(4_096),
    "hubs_over_leaves": lambda: G.disjoint_union([_star(600)] * 27),
    "rmat15": lambda: kc.gen_rmat(15, 16.0, seed=9).arrays(),
    "path_20k": lambda: _path(20_000),
    "path_200k": lambda: _path(200_000),
    "path_1m": lambda: _path(1_000_000),
    "paths_and_core": lambda: G.disjoint_union([_path(30_001), _complete(90), _star(9_000), _path(17_000)]),
    "isolated": lambda: (np.array([1], np.uint32), np.array([20_000], np.uint32), 30_000),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_peel_matches_oracle(ctx, name):
    s, d, n = CASES[name]()
    og = OracleGraph(s, d, n)
    og.orient("degen")
    want_prio, want_level = og.peel()
    want_core, want_max = og.kcore()
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        core, mx = g.kcore()
        g.orient("degen")
        prio, level = g.peel()
    assert np.array_equal(prio, want_prio) and np.array_equal(level, want_level)
    assert np.array_equal(core, want_core) and mx == want_max
