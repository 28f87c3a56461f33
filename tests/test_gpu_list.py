"""The list-encoded kernel, which takes the units above 1,024 vertices: a few
hubs, adjacent to each other, over 1,150 vertices that form a sparse random graph
with planted cliques (deep trees, pivot chains, irregular neighbourhoods). Leaves
on those vertices give them larger degrees than the hubs, so the degree
orientation puts them into the hubs' out-lists."""
import numpy as np
import pytest

import kcgpu_b200 as kc
from oracle.oracle import OracleGraph

pytestmark = pytest.mark.gpu

HUBS, INNER = 4, 1150


def _graph(seed: int):
    rng = np.random.default_rng(seed)
    a = np.triu(rng.random((INNER, INNER)) < 0.02, 1)
    for size in (12, 16, 20):
        c = np.sort(rng.choice(INNER, size, replace=False))
        a[np.ix_(c, c)] = True
    s, d = np.nonzero(np.triu(a, 1))
    hub = INNER + np.arange(HUBS)
    hs, hd = np.triu_indices(HUBS, 1)
    leaf_of = np.repeat(np.arange(INNER), INNER + 30)
    s = np.concatenate([s, np.tile(np.arange(INNER), HUBS), hub[hs], leaf_of])
    d = np.concatenate([d, np.repeat(hub, INNER), hub[hd], INNER + HUBS + np.arange(leaf_of.size)])
    return s.astype(np.uint32), d.astype(np.uint32), INNER + HUBS + leaf_of.size


@pytest.fixture(scope="module")
def case(ctx):
    s, d, n = _graph(5)
    og = OracleGraph(s, d, n)
    og.orient("degree")
    want = {k: og.count(k, "pivot", closed=True) for k in range(3, 9)}
    g = kc.Graph.from_edges(ctx, s, d, n)
    g.orient("degree")
    rp, _ = g.dag()
    out = np.diff(rp.astype(np.int64))[INNER : INNER + HUBS]
    assert (np.sort(out) == INNER + np.arange(HUBS)).all()  # every hub is a node unit of the list kernel, hub pairs are edge units
    assert want[8] > 1000
    yield g, want
    g.close()


# every partition size at k = 4 and 5, every k with a warp per walker (and with
# eight lanes where that is quick); the automatic mode pivots these units
PARTS = {
    "orient": [(p, k) for p in (1, 2, 4, 8, 16) for k in (4, 5)] + [(32, k) for k in range(3, 9)],
    "pivot": [(p, 4) for p in (1, 2, 4, 16)] + [(8, k) for k in (3, 4, 6)] + [(32, k) for k in range(3, 9)],
    "auto": [(0, 3), (32, 5), (8, 4)],
}


@pytest.mark.parametrize("mode", sorted(PARTS))
@pytest.mark.parametrize("unit", ["node", "edge"])
def test_counts_match_oracle(case, mode, unit):
    g, want = case
    for part, k in PARTS[mode]:
        r = g.count(k, mode=mode, unit=unit, part=part, encoding="list", stats=True)
        assert r.count == want[k], (mode, unit, part, k)
        assert r.stats["max_unit_size"] > 1024 and r.stats["ms_launch"][0] > 0


@pytest.mark.parametrize("mode", ["orient", "pivot"])
@pytest.mark.parametrize("unit", ["node", "edge"])
def test_shards_add_up(case, mode, unit):
    g, want = case
    for S in (2, 3):
        got = [g.count(5, mode=mode, unit=unit, encoding="list", shard=(i, S)) for i in range(S)]
        assert sum(got) == want[5], (mode, unit, S, got)


@pytest.mark.parametrize("mode", ["orient", "pivot"])
def test_time_limit(ctx, case, mode):
    g, want = case
    ctx.set_time_limit(1)
    try:
        with pytest.raises(kc.KCError, match="KC_ERR_DEVICE_TIMEOUT"):
            g.count(5, mode=mode, encoding="list")
    finally:
        ctx.set_time_limit(0)
    assert g.count(5, mode=mode, encoding="list") == want[5]


def test_batch_with_a_list_unit(ctx):
    s, d, n = _graph(6)
    es, ed, en = kc.gen_er(900, 0.05, 7).arrays()
    off = np.array([0, es.size, es.size + s.size], np.uint64)
    nn, ks = np.array([en, n], np.uint32), np.array([4, 6], np.uint32)
    want = []
    for (a, b, m), k in zip(((es, ed, en), (s, d, n)), ks):
        og = OracleGraph(a, b, m)
        og.orient("degree")
        want.append(og.count(int(k), "pivot", closed=True))
    for mode in ("orient", "pivot"):
        got = kc.batch_count(ctx, np.concatenate([es, s]), np.concatenate([ed, d]), off, nn, ks, autotune=False,
                             fixed=dict(mode=mode, unit="node", part=8, encoding="list"))
        assert got == want, mode
