"""Batches built from adjacency bit rows against the same graphs counted one by
one: row widths around a word, duplicate and reversed edges, self-loops, graphs
without edges or vertices, both orientations, every method, out-degrees above
1024 (which go the general way), and the sizes past which a batch is built the
general way as a whole."""
import numpy as np
import pytest

import kcgpu_b200 as kc
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _batch(graphs):
    off = np.cumsum([0] + [len(s) for s, _, _ in graphs]).astype(np.uint64)
    s = np.concatenate([g[0] for g in graphs]).astype(np.uint32)
    d = np.concatenate([g[1] for g in graphs]).astype(np.uint32)
    return s, d, off, np.array([g[2] for g in graphs], np.uint32)


def _messy_er(n, p, seed):
    s, d, n = kc.gen_er(n, p, seed).arrays()
    s, d = G.messy(s, d, n, seed)
    return s, d, n


def _small():
    none = np.zeros(0, np.uint32)
    gs = [(none, none, 0), (none, none, 5), (np.array([0], np.uint32), np.array([0], np.uint32), 1)]
    for n in (2, 31, 32, 33, 63, 64, 65, 200, 700):
        gs.append(_messy_er(n, 0.4 if n < 100 else 0.1, n))
    gs += [(none, none, 3), (*G.complete(40), 40), _messy_er(1500, 0.06, 9)]
    return gs


CASES = {
    "small": _small,
    "deep_out_degrees": lambda: _small() + [G.multipartite([520, 520, 520])],
    "sparse": lambda: [kc.gen_er(6000, 0.001, 3).arrays(), kc.gen_rmat(12, 8.0, seed=4).arrays()],
    # rows of 157 words (160 held), of 256 and one vertex past the most
    "wide_rows": lambda: [kc.gen_er(5000, 0.02, 6).arrays(), kc.gen_er(8192, 0.01, 7).arrays(),
                          kc.gen_er(8161, 0.012, 8).plant_cliques(3, 12, 20, 5).arrays()] + _small(),
    "past_wide_rows": lambda: [kc.gen_er(5000, 0.02, 6).arrays(), kc.gen_er(8193, 0.01, 7).arrays()] + _small(),
    "too_many_vertices": lambda: _small() + [kc.gen_er(16_385, 0.0002, 5).arrays()],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("orientation", ["degree", "degen"])
def test_batches_match_single_graphs(ctx, name, orientation):
    import torch

    gs = CASES[name]()
    s, d, off, nn = _batch(gs)
    # (k = 3 for the multipartite graph: listing 520^3 triangles for a larger k takes minutes)
    ks = np.array([3 if len(g[0]) > 500_000 else 3 + i % 4 for i, g in enumerate(gs)], np.uint32)
    want = []
    for (a, b, n), k in zip(gs, ks):
        if n == 0:
            want.append(0)
            continue
        with kc.Graph.from_edges(ctx, a, b, n) as g:
            want.append(g.orient("degen").count(int(k), mode="pivot"))
    dev = tuple(torch.from_numpy(x.view(np.int32)).cuda() for x in (s, d))
    torch.cuda.synchronize()
    ptrs = tuple(t.data_ptr() for t in dev)
    methods = [None] + [dict(mode=m, unit=u, part=8, encoding=e) for m in ("orient", "pivot", "auto")
                        for u in ("node", "edge") for e in ("bitmap", "list")]
    for fixed in methods:
        for device_ptrs in (None, ptrs):
            got = kc.batch_count(ctx, s, d, off, nn, ks, orientation=orientation, autotune=fixed is None, fixed=fixed,
                                 device_ptrs=device_ptrs)
            assert got == want, (fixed, device_ptrs is not None)
    assert np.array_equal(dev[0].cpu().numpy().view(np.uint32), s)  # the caller's edges are left alone


def test_endpoint_out_of_range(ctx):
    gs = _small()
    s, d, off, nn = _batch(gs)
    bad = next(i for i, g in enumerate(gs) if len(g[0]) > 40)
    d = d.copy()
    d[int(off[bad]) + 7] = nn[bad]
    with pytest.raises(kc.KCError, match=f"graph {bad} "):
        kc.batch_count(ctx, s, d, off, nn, np.full(len(gs), 3, np.uint32))
    assert kc.batch_count(ctx, *_batch(gs)[:4], np.full(len(gs), 3, np.uint32)) is not None


@pytest.mark.parametrize("orientation", ["degree", "degen"])
def test_out_of_memory_takes_the_general_way(ctx, orientation):
    """Every allocation of a batch built from bit rows fails in turn: the batch
    is then counted without them, and nothing is left allocated. Staging
    buffers of a pipeline, and batches that have no bit rows, still fail."""
    L = kc.lib()
    cases = [(_small() + [G.multipartite([520, 520, 520])], 0, True), (_small(), 2000, False),
             (CASES["too_many_vertices"](), 0, False)]
    for gs, chunk, always in cases:
        s, d, off, nn = _batch(gs)
        ks = np.full(len(gs), 3, np.uint32)
        ctx.set_batch_chunk_edges(chunk)
        try:
            want = kc.batch_count(ctx, s, d, off, nn, ks, orientation=orientation)
            L.kc_ctx_release_cached_memory(ctx.handle)
            base = L.kc_test_live_allocations()
            outcomes = []
            for i in range(200):
                L.kc_test_fail_alloc_after(i)
                try:
                    assert kc.batch_count(ctx, s, d, off, nn, ks, orientation=orientation) == want, i
                    outcomes.append("right")
                except kc.KCError as e:
                    assert e.name == "KC_ERR_OOM" and not always, (i, str(e))
                    outcomes.append("oom")
                finally:
                    L.kc_test_fail_alloc_after(-1)
                L.kc_ctx_release_cached_memory(ctx.handle)
                assert L.kc_test_live_allocations() == base, i
            assert ("oom" in outcomes) == (not always) and outcomes[-1] == "right"
        finally:
            ctx.set_batch_chunk_edges(0)


@pytest.mark.parametrize("device", [True, False])
def test_phases_hold_their_own_time(ctx, device):
    import torch

    gs = [kc.gen_er(1200, 0.2, i).arrays() for i in range(40)]
    s, d, off, nn = _batch(gs)
    dev = tuple(torch.from_numpy(x.view(np.int32)).cuda() for x in (s, d))
    torch.cuda.synchronize()
    ptrs = tuple(t.data_ptr() for t in dev) if device else None
    ks = np.full(len(gs), 3, np.uint32)
    kc.batch_count(ctx, s, d, off, nn, ks, device_ptrs=ptrs)
    _, st = kc.batch_count(ctx, s, d, off, nn, ks, device_ptrs=ptrs, return_stats=True)
    host = st["host_ms"]
    assert all(x >= 0 for x in host) and abs(sum(host) - st["ms_total"]) < 0.1 + 0.01 * st["ms_total"]
    assert host[0] >= 0.9 * st["ms_h2d"] and host[1] >= 0.9 * st["ms_build"], (host, st["ms_h2d"], st["ms_build"])
