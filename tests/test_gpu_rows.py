"""Row sorting, orientation and truss support at the edges of the row lengths
their kernels are chosen by: 256/257, 512/513, 1024/1025 entries, rows past
32,768, hubs whose rows one warp walks, a vertex range above and below the
bitmaps' 2^20, duplicate entries in every kind of row, and the edge counts,
degrees and vertex counts that the support kernels are chosen by."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import kcgpu_b200 as kc
from oracle.oracle import OracleGraph
from tests import graphs as G

pytestmark = pytest.mark.gpu


def _hubs(degrees, n: int, seed: int, noise: int):
    """Vertex i of the first len(degrees) gets degrees[i] random neighbours
    (with repeats on top), the rest a few random edges."""
    rng = np.random.default_rng(seed)
    s, d = [], []
    for i, deg in enumerate(degrees):
        nb = rng.choice(np.arange(len(degrees), n), size=deg, replace=False)
        s += [np.full(deg, i), nb[: deg // 3]]
        d += [nb, np.full(deg // 3, i)]
    s.append(rng.integers(0, n, noise))
    d.append(rng.integers(0, n, noise))
    s, d = np.concatenate(s).astype(np.uint32), np.concatenate(d).astype(np.uint32)
    order = rng.permutation(s.size)
    return s[order], d[order], n


def _star(leaves: int):
    return np.zeros(leaves, np.uint32), np.arange(1, leaves + 1, dtype=np.uint32), leaves + 1


def _matching_and_core(m: int):
    """A complete graph of 300 vertices and single edges, m edges in all."""
    s, d = G.complete(300)
    k = m - s.size
    return G.disjoint_union([(s, d, 300), (np.arange(k), np.arange(k, 2 * k), 2 * k)])


CASES = {
    "edges_of_ranges": lambda: _hubs([1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047,
                                      2048, 2049], 6000, 1, 3000),
    "longest_rows": lambda: _hubs([16_384, 16_385, 32_768, 32_769, 40_000], 60_000, 2, 60_000),
    "at_the_bitmap_limit": lambda: _hubs([1500, 3000, 33_000], 1 << 20, 3, 40_000),
    "past_the_bitmap_limit": lambda: _hubs([300, 1500, 3000, 17_000, 33_000], (1 << 20) + 1, 4, 40_000),
    # more long rows than CTAs sort them
    "many_long_rows": lambda: _hubs([1025 + 7 * (i % 147) for i in range(700)], 120_000, 5, 10_000),
    "many_long_rows_wide": lambda: _hubs([1100] * 320, 1 << 20, 6, 10_000),
    # supports from bitmaps (49,152 edges and more): vertices around a warp's share
    # with a small and with a wide bitmap, hubs cut into few and into many tasks,
    # most of a bitmap set by one vertex
    "support_shares": lambda: _hubs([31, 32, 33, 34, 127, 128, 129, 130, 255, 256, 257, 513], 30_000, 8, 80_000),
    "support_shares_wide": lambda: _hubs([31, 32, 33, 34, 127, 128, 129, 130, 255, 256, 257, 1025] * 8, 400_000, 9, 80_000),
    "support_stars": lambda: G.disjoint_union([_star(70_000), _star(17_000), G.multipartite([30, 40, 50])]),
    "support_edges_below": lambda: _matching_and_core(49_151),
    "support_edges_at": lambda: _matching_and_core(49_152),
    # one scan tile and the one-CTA key sort end at 4,096 vertices
    "small_4095": lambda: kc.gen_er(4095, 0.004, 11).arrays(),
    "small_4096": lambda: kc.gen_er(4096, 0.004, 12).arrays(),
    "small_4097": lambda: kc.gen_er(4097, 0.004, 13).arrays(),
    "two_vertices": lambda: (np.array([1], np.uint32), np.array([0], np.uint32), 2),
    "dense_core": lambda: kc.gen_rmat(13, 16.0, seed=7).arrays(),
}


def _check(ctx, s, d, n):
    og = OracleGraph(s, d, n)
    want_rp, want_ci = og.csr()
    want_sup = og.truss_support()
    with kc.Graph.from_edges(ctx, s, d, n) as g:
        rp, ci = g.csr()
        assert np.array_equal(rp, want_rp) and np.array_equal(ci, want_ci)
        assert np.array_equal(g.truss_support(), want_sup)
        for orientation in ("degree", "degen"):
            og.orient(orientation)
            want = og.dag()
            got = g.orient(orientation).dag()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), orientation


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_match_oracle(ctx, name):
    _check(ctx, *CASES[name]())


# Vertex counts whose bitmaps end just below, at and above 48 KB, with and
# without the kernels' static shared memory.
AROUND_48K = (392_192, 392_193, 393_088, 393_089, 393_100, 393_200, 393_216, 393_217)


def check_around_48k():
    ctx = kc.Context(0)
    for n in AROUND_48K:
        _check(ctx, *_hubs([1500, 3000], n, n, 70_000))
    ctx.close()


def test_bitmaps_around_48k_in_a_fresh_process():
    """(A larger graph in the same process would raise the launch limit first.)"""
    r = subprocess.run([sys.executable, "-c", "from tests.test_gpu_rows import check_around_48k; check_around_48k()"],
                       cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-1000:] + r.stderr[-3000:]
