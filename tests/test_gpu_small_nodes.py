"""Clique-tree nodes that the pivoting kernel counts whole: r = k - held = 3
with up to 128 candidates and any r with up to 32, at the edges of the word
and size ranges, with pivots already dropped (dense graphs), universal
vertices (planted cliques), the largest r (19: k = 20 by node units) and ones
beyond it."""
import math

import numpy as np
import pytest

import kcgpu_b200 as kc
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu


def _dense(n: int, p: float, seed: int):
    """G(n, p) with a clique planted on n // 3 of its vertices."""
    rng = np.random.default_rng(seed)
    a = np.triu(rng.random((n, n)) < p, 1)
    c = rng.permutation(n)[: n // 3]
    a[np.ix_(c, c)] = True
    s, d = np.nonzero(np.triu(a, 1) | np.triu(a.T, 1))
    return s.astype(np.uint32), d.astype(np.uint32), n


@pytest.mark.parametrize("n", [6, 32, 33, 34, 64, 65, 66, 96, 97, 98, 128, 129, 130, 180])
@pytest.mark.parametrize("p", [0.25, 0.85])
def test_dense_graphs_match_oracle(ctx, n, p):
    s, d, n = _dense(n, p, n)
    og = OracleGraph(s, d, n)
    og.orient("degen")
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degen")
        for k in (4, 5, 6, 9):
            if k > 6 and n > 66 and p > 0.5:
                continue  # (the oracle's tree is large there)
            want = og.count(k, "pivot", closed=True)
            for mode, unit in (("pivot", "node"), ("pivot", "edge"), ("auto", "node")):
                assert g.count(k, mode=mode, unit=unit) == want, (n, p, k, mode, unit)


@pytest.mark.parametrize("n", [24, 33, 70, 140])
def test_complete_graph_deep_k(ctx, n):
    s, d = np.triu_indices(n, 1)
    with kc.Graph.from_edges(ctx, s.astype(np.uint32), d.astype(np.uint32), n) as g:
        g.orient("degree")
        for k in (4, 8, 19, 20, 21, 22, 23):
            for unit in ("node", "edge"):
                assert g.count(k, mode="pivot", unit=unit) == math.comb(n, k), (n, k, unit)


@pytest.mark.parametrize("n", [6, 32, 33, 34, 66, 97])
@pytest.mark.parametrize("p", [0.25, 0.85])
def test_several_k(ctx, n, p):
    s, d, n = _dense(n, p, n + 1)
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degen")
        for ks in ([3, 4, 5], list(range(3, 10)), [4, 16], [5, 17, 6]):
            want = [g.count(k, mode="pivot") for k in ks]
            for unit in ("node", "edge"):
                assert g.count_multi(ks, unit=unit) == want, (n, p, ks, unit)


@pytest.mark.parametrize("n", [24, 33, 70, 140])
def test_several_k_complete_graph(ctx, n):
    s, d = np.triu_indices(n, 1)
    with kc.Graph.from_edges(ctx, s.astype(np.uint32), d.astype(np.uint32), n) as g:
        g.orient("degree")
        for ks in (list(range(3, 17)), list(range(3, 34)), [15, 18]):
            assert g.count_multi(ks) == [math.comb(n, k) for k in ks], (n, ks)


@pytest.mark.parametrize("n", [24, 33, 70, 140])
def test_auto_past_the_listing_depth(ctx, n):
    """k = 19 is the last k that the automatic mode lists; past it every unit is pivoted."""
    s, d = np.triu_indices(n, 1)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    # the complete graph, padded with a sparse part so that units of every size occur
    es, ed, en = kc.gen_er(3000, 0.004, n).arrays()
    s, d = np.concatenate([s, es + n]), np.concatenate([d, ed + n])
    with kc.Graph.from_edges(ctx, s, d, n + en) as g:
        g.orient("degen")
        for k in (18, 19, 20, 21, 30):
            for unit in ("node", "edge"):
                for encoding in ("bitmap", "list"):
                    got = g.count(k, mode="auto", unit=unit, encoding=encoding, part=0)
                    assert got == math.comb(n, k), (n, k, unit, encoding)
            assert g.count_local(k, mode="auto")[:n] == [math.comb(n - 1, k - 1)] * n, (n, k)
    # one pass of a batch whose largest k is past it
    off = np.array([0, s.size, 2 * s.size], np.uint64)
    for fixed in (None, dict(mode="auto", unit="node", part=0, encoding="bitmap")):
        got = kc.batch_count(ctx, np.tile(s, 2), np.tile(d, 2), off, np.full(2, n + en, np.uint32), np.array([18, 21], np.uint32),
                             autotune=fixed is None, fixed=fixed)
        assert got == [math.comb(n, 18), math.comb(n, 21)], (n, fixed)


@pytest.mark.parametrize("n", [15, 16, 17, 18, 33, 34, 48, 70])
@pytest.mark.parametrize("p", [0.4, 0.9])
def test_several_k_past_the_histogram(ctx, n, p):
    """Largest k above 16: nodes of up to 15 candidates are counted whole all the same."""
    s, d, n = _dense(n, p, n + 2)
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degen")
        single = {k: g.count(k, mode="pivot") for k in range(3, 34)}
        for ks in (list(range(3, 34)), [5, 24], [17, 20, 31], [3, 16, 17], [33]):
            for unit in ("node", "edge"):
                assert g.count_multi(ks, unit=unit) == [single[k] for k in ks], (n, p, ks, unit)


def test_several_k_past_the_histogram_on_blocks(ctx):
    s, d, n = kc.gen_sbm(2000, 20, 0.4, 0.002, 3).plant_cliques(3, 18, 30, 7).arrays()
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        g.orient("degen")
        ks = list(range(3, 31))
        want = [g.count(k, mode="pivot") for k in ks]
        for unit in ("node", "edge"):
            assert g.count_multi(ks, unit=unit) == want
            assert g.count_multi([4, 25], unit=unit) == [want[1], want[22]]
