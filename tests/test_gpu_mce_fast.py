"""Maximal cliques of roots around the limits of the register walk
(csrc/g2_mce_fast.cuh): |P0| of 32, 64 and 96, 128 live back rows, branches that
are renumbered, hand-off on and off; counts, histogram and per-root search-tree
nodes equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(g2, sizes, keep, backs, seed):
    """Random cores of the given sizes (edge probability keep) on the last ids, and
    `backs` earlier vertices per core, each adjacent to a random third of it."""
    rng = np.random.default_rng(seed)
    edges, n = [], sum(backs for _ in sizes)
    base, x = n, 0
    for p in sizes:
        a, b = np.triu_indices(p, 1)
        on = rng.random(a.size) < keep
        edges += [(base + int(i), base + int(j)) for i, j in zip(a[on], b[on])]
        for _ in range(backs):
            nb = np.flatnonzero(rng.random(p) < 0.33)
            edges += [(x, base + int(j)) for j in nb]
            x += 1
        base += p
    return g2.Graph.from_edges(base, edges)


@pytest.mark.parametrize("keep,backs", [(0.3, 3), (0.3, 200), (0.6, 40)])
def test_root_sizes(g2, orc, ctx, keep, backs):
    sizes = [5, 32, 33, 64, 65] + ([96, 97, 130] if keep < 0.5 else [])
    g = _layers(g2, sizes, keep, backs, 7)
    want = orc.mce(g, threads=8, per_root=True)
    ctx.load(g)
    for kw in ({}, {"schedule": "heuristic"}, {"spill_kcycles": 1}, {"flags": 16}, {"chunk": 3}):
        c, h, rn = ctx.mce(root_nodes=True, **kw)
        assert c == want["count"], (keep, backs, kw)
        assert np.array_equal(h, want["hist"][:h.size]) and np.array_equal(rn, want["root_nodes"]), (keep, backs, kw)


def test_sources_and_small_slab(g2, orc):
    """A subset of the roots, and slabs too small for the register walk's frames."""
    from g2aimd.context import Context
    g = g2.Graph.rmat(10, 16, seed=4).degeneracy_recoded()
    src = np.arange(g.n - 1, -1, -3, dtype=np.uint32)
    want = orc.mce(g, roots=src, threads=8)
    for scratch in (0, 148 * 24 * 1024 * 4):
        with Context(0, scratch_bytes=scratch) as c:
            c.load(g)
            cnt, h = c.mce(sources=src)
            assert cnt == want["count"] and np.array_equal(h, want["hist"][:h.size]), scratch


@pytest.mark.parametrize("fold", [0, 1, 4])
def test_size_counters_are_emptied_when_full(g2, orc, ctx, monkeypatch, fold):
    """The warps' 32-bit size counters live for all roots of a warp and are emptied
    every 2^fold inner nodes: with fold cut from 24 to a few, both those of whole roots
    and those of branches are emptied many times, and the histogram stays the oracle's."""
    monkeypatch.setenv("G2_HIST_FOLD", str(fold))
    for g in (g2.Graph.rmat(11, 16, seed=2).degeneracy_recoded(), _layers(g2, [97, 130], 0.3, 200, 7)):
        want = orc.mce(g, threads=8)
        ctx.load(g)
        for kw in ({}, {"schedule": "heuristic"}, {"flags": 16}):
            c, h = ctx.mce(**kw)
            assert c == want["count"] and int(h.sum()) == c, (fold, kw)
            assert np.array_equal(h, want["hist"][:h.size]), (fold, kw)


def test_branches_deep_in_a_root(g2, orc, ctx):
    """Cliques of 60 to 140 vertices with a few holes each, one of them over a core
    with many back neighbours: branches enter the register walk at depths from which
    their sizes exceed its shared counters."""
    rng = np.random.default_rng(11)
    edges, base = [], 0
    for p in (60, 110, 125, 140):
        a, b = np.triu_indices(p, 1)
        hole = set(int(x) for x in rng.choice(a.size, 9, replace=False))
        edges += [(base + int(i), base + int(j)) for t, (i, j) in enumerate(zip(a, b)) if t not in hole]
        base += p
    g = g2.Graph.from_edges(base, edges)
    want = orc.mce(g, threads=8, per_root=True)
    ctx.load(g)
    for kw in ({}, {"schedule": "heuristic"}, {"spill_kcycles": 1}, {"flags": 16}):
        c, h, rn = ctx.mce(root_nodes=True, **kw)
        assert c == want["count"], kw
        assert np.array_equal(h, want["hist"][:h.size]) and np.array_equal(rn, want["root_nodes"]), kw


def test_levels_above_a_small_branch_are_handed_off(g2, orc, ctx):
    """A few roots of more than 96 vertices whose depth-1 nodes all enter the register
    walk: idle warps get the root's own branches, not only those inside a walk."""
    g = g2.Graph.er(300, 0.4, seed=5).degeneracy_recoded()
    fwd = np.array([int((g.neighbors(v) > v).sum()) for v in range(g.n)])
    src = np.flatnonzero(fwd > 96).astype(np.uint32)[-4:]
    assert src.size == 4
    want = orc.mce(g, roots=src, threads=8, per_root=True)
    ctx.load(g)
    for kw in ({"spill_kcycles": 1}, {}, {"schedule": "heuristic", "spill_kcycles": 1}):
        c, h, rn = ctx.mce(sources=src, root_nodes=True, **kw)
        assert c == want["count"] and np.array_equal(h, want["hist"][:h.size]), kw
        assert np.array_equal(rn, want["root_nodes"]), kw
        assert ctx.spill_stats()[0] > 200, kw  # the roots were shared out


@pytest.mark.parametrize("take", [1, 5, 600, 5000])
def test_lists_of_few_roots_are_dealt_out_one_by_one(g2, orc, ctx, take):
    """The caller's roots, heaviest first, from one to two per resident warp: no warp
    takes several while others have none, and results follow the caller's order."""
    g = g2.Graph.er(5000, 0.02, seed=8).degeneracy_recoded()
    src = np.argsort(-g.degrees(), kind="stable").astype(np.uint32)[:take]
    want = orc.mce(g, roots=src, threads=8, per_root=True)
    ctx.load(g)
    for kw in ({}, {"schedule": "heuristic"}, {"flags": 16}, {"chunk": 3}):
        c, h, rn = ctx.mce(sources=src, root_nodes=True, **kw)
        assert c == want["count"] and np.array_equal(h, want["hist"][:h.size]), (take, kw)
        assert np.array_equal(rn, want["root_nodes"]), (take, kw)
    if take == 5000:  # one root a grab: no walk waits behind others (a chunk of 8 fills 630 of 3,552 warps)
        import time
        def best(**kw):
            t = []
            for _ in range(5):
                t0 = time.perf_counter()
                ctx.mce(sources=src, **kw)
                t.append(time.perf_counter() - t0)
            return min(t)
        assert best(schedule="heuristic", flags=16) < 1.25 * best(schedule="heuristic", flags=16, chunk=1)
