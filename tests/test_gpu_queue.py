"""The one-CTA queue of small graphs and the general one, at the edges of its
range: unit counts around a round and around the limit, all size classes in one
graph, unit shards, edge units, and graphs without any unit."""
import numpy as np
import pytest

import kcgpu_b200 as kc
from oracle.oracle import OracleGraph
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _mixed(isolated: int):
    """Units of all four size classes (cliques of 20, 90 and 200, a dense
    multipartite graph above 1024), then isolated vertices."""
    parts = []
    for c in (20, 90, 200):
        s, d = G.complete(c)
        parts.append((s, d, c))
    parts.append(G.multipartite([550, 550, 550]))
    parts.append((np.zeros(0, np.uint32), np.zeros(0, np.uint32), isolated))
    return G.disjoint_union(parts)


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 16_383, 16_384, 16_385])
def test_unit_counts_at_the_limits(ctx, n):
    s, d, n = kc.gen_er(n, min(0.5, 24.0 / max(1, n)), n).arrays() if n > 1 else (np.zeros(0, np.uint32),) * 2 + (1,)
    og = OracleGraph(s, d, n)
    og.orient("degree")
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degree")
        for k in (3, 4):
            want = og.count(k)
            for mode, unit in (("orient", "node"), ("pivot", "edge"), ("auto", "node")):
                assert g.count(k, mode=mode, unit=unit) == want, (n, k, mode, unit)
                assert sum(g.count(k, mode=mode, unit=unit, shard=(i, 3)) for i in range(3)) == want


@pytest.mark.parametrize("isolated", [0, 15_000])
def test_all_classes(ctx, isolated):
    s, d, n = _mixed(isolated)
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degree")
        for k in (3, 4):
            want = sum(G.comb(c, k) for c in (20, 90, 200)) + G.multipartite_kcliques([550, 550, 550], k)
            for mode in ("pivot", "auto"):
                for unit, enc in (("node", "bitmap"), ("edge", "bitmap"), ("node", "list")):
                    r = g.count(k, mode=mode, unit=unit, encoding=enc, stats=True)
                    assert r.count == want and r.stats["units"] > 0, (k, mode, unit, enc)


@pytest.mark.parametrize("n", [500, 16_384, 16_385, 2_097_152, 2_097_153])
def test_launches_are_counted(ctx, n):
    """stats["kernels"] is what the call launched: the queue is one kernel for up
    to 16,384 units, five up to 2,097,152, then seven."""
    s, d = G.complete(60)
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degree")
        g.count(5, mode="pivot", stats=True)
        before = kc.lib().kc_kernel_launches()
        r = g.count(5, mode="pivot", stats=True)
        assert r.count == G.comb(60, 5)
        assert r.stats["kernels"] == kc.lib().kc_kernel_launches() - before
