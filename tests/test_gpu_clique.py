"""3-, 4- and 5-clique counts on core bit rows (csrc/clique.cu) against the CPU
oracle, at the sizes where a root's walk changes: |P0| of 32, 128 and the
shared-memory limit, ids with and without a bit row, batches, split roots and
slabs too small for a root's rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nested(g2, n, keep, seed):
    """n vertices in a path of windows: vertex v is adjacent to each of the next
    `p` ids with probability `keep`, p running over the edges of the walks."""
    rng = np.random.default_rng(seed)
    sizes = [2, 3, 4, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160]
    edges = []
    for v in range(n):
        p = min(sizes[v % len(sizes)], n - 1 - v)
        on = np.flatnonzero(rng.random(p) < keep) + v + 1
        edges += [(v, int(u)) for u in on]
    return g2.Graph.from_edges(n, edges)


@pytest.mark.parametrize("q", [0, 24, 25])
def test_root_sizes(g2, orc, ctx, q):
    from g2aimd.context import Plan
    plan = Plan.preset(q)
    for g in (_nested(g2, 700, 1.0, 1), _nested(g2, 700, 0.3, 2)):
        if q == 25 and g.m > 60000:
            g = _nested(g2, 300, 1.0, 3)  # every subset of a window is a clique: keep the oracle short
        want = orc.match(g, plan, threads=8, per_root=True)
        ctx.load(g)
        for kw in ({}, {"schedule": "heuristic"}, {"schedule": "heuristic", "split": True, "granularity": 256},
                   {"schedule": "heuristic", "warps_per_block": 1}, {"chunk": 7, "warps_per_block": 4}):
            rc = np.zeros(g.n, np.uint64)
            assert ctx.match(plan, root_counts=rc, **kw) == want["count"], (q, kw)
            assert np.array_equal(rc, want["root_counts"]), (q, kw)


@pytest.mark.parametrize("q", [0, 24, 25])
def test_ids_without_bit_rows(g2, orc, ctx, q):
    """60,000 vertices with planted cliques on generator ids: the core's bit rows
    (about 1 MB here, 2,900 ids) hold few of the cliques' vertices."""
    from g2aimd.context import Plan
    plan = Plan.preset(q)
    g = g2.Graph.er(60000, 1e-5, planted=60, planted_size=40, seed=3)
    want = orc.match(g, plan, threads=8, per_root=True)
    src = np.arange(g.n - 1, -1, -2, dtype=np.uint32)
    ctx.load(g)
    for kw in ({}, {"schedule": "heuristic"}):
        rc = np.zeros(g.n, np.uint64)
        assert ctx.match(plan, root_counts=rc, **kw) == want["count"]
        assert np.array_equal(rc, want["root_counts"])
        assert ctx.match(plan, sources=src, **kw) == int(want["root_counts"][src].sum())


@pytest.mark.parametrize("take", [1, 7, 300])
def test_few_roots_get_a_small_matrix(g2, orc, ctx, take):
    """A run's bit rows are sized by its roots (8 KB each, 1 MB at least): of these
    60,000 vertices 2,900, 2,900 and 4,400 get one, 7,600 in the run over all of them."""
    from g2aimd.context import Plan
    g = g2.Graph.er(60000, 5e-4, planted=60, planted_size=30, seed=3).degeneracy_recoded()
    rng = np.random.default_rng(take)
    src = rng.choice(np.arange(g.n - 3000, g.n - 20), take, replace=False).astype(np.uint32)
    ctx.load(g)
    for q in (0, 24):
        plan = Plan.preset(q)
        want = orc.match(g, plan, roots=src, threads=8)["count"]
        for kw in ({}, {"schedule": "heuristic"}):
            assert ctx.match(plan, **kw) > 0
            assert ctx.match(plan, sources=src, **kw) == want, (q, kw)
    want = orc.mce(g, roots=src, threads=8)
    c, h = ctx.mce(sources=src)
    assert c == want["count"] and np.array_equal(h, want["hist"][:h.size])


@pytest.mark.parametrize("words", [0, 64 * 37])
def test_wide_5_clique_roots(g2, orc, words):
    """A root of 640 vertices one of which is adjacent to 420 earlier ones (more than are
    compressed into rows of their own), beside roots up to 130 wide: rows in shared
    memory, in slabs and, with small scratch, beyond them."""
    from g2aimd.context import Context, Plan
    plan = Plan.preset(25)
    rng = np.random.default_rng(12)
    n = 641
    e = [np.stack([np.zeros(640, int), np.arange(1, n)], 1)]
    a, b = np.triu_indices(520, 1)
    on = rng.random(a.size) < 0.06
    e.append(np.stack([a[on] + 1, b[on] + 1], 1))
    e.append(np.stack([rng.choice(np.arange(1, 521), 420, replace=False), np.full(420, 600)], 1))
    g = _csr(g2, n, np.concatenate(e))
    fwd = g.neighbors(0)
    assert fwd.size == 640 and int((g.neighbors(600) < 600).sum()) > 256
    want = orc.match(g, plan, threads=8, per_root=True)
    launch = dict(blocks=148, warps_per_block=8) if words else {}
    with Context(0, scratch_bytes=148 * 8 * words * 4) as c:
        c.load(g)
        for kw in ({}, {"schedule": "heuristic"}, {"schedule": "heuristic", "split": True, "granularity": 256}):
            rc = np.zeros(g.n, np.uint64)
            assert c.match(plan, root_counts=rc, **dict(launch, **kw)) == want["count"] > 0, (words, kw)
            assert np.array_equal(rc, want["root_counts"]), (words, kw)


@pytest.mark.parametrize("q", [0, 24, 25])
def test_rows_in_slabs_and_beyond(g2, orc, q):
    """Dense cores of 700 vertices (3- and 4-cliques: rows in shared memory and, with small
    scratch, beyond the slabs, the rest list) and of 420 (5-cliques, up to 97 wide)."""
    from g2aimd.context import Context, Plan
    plan = Plan.preset(q)
    rng = np.random.default_rng(5)
    n = 700 if q < 25 else 420
    a, b = np.triu_indices(n, 1)
    keep = rng.random(a.size) < (0.5 if q < 25 else 0.2)
    g = g2.Graph.from_edges(n, np.stack([a[keep], b[keep]], 1))
    want = orc.match(g, plan, threads=8, per_root=True)
    for words in (0, 64 * 37):
        launch = dict(blocks=148, warps_per_block=8) if words else {}
        with Context(0, scratch_bytes=148 * 8 * words * 4) as c:
            c.load(g)
            for kw in ({}, {"schedule": "heuristic"}, {"schedule": "heuristic", "warps_per_block": 2}):
                rc = np.zeros(g.n, np.uint64)
                assert c.match(plan, root_counts=rc, **dict(launch, **kw)) == want["count"], (words, kw)
                assert np.array_equal(rc, want["root_counts"]), (words, kw)


def test_batch_blocks(g2, orc, ctx):
    """Each graph of a batch has its own bit rows; empty and edgeless graphs among them."""
    from g2aimd.context import Plan
    gs = [g2.Graph.from_edges(3, []), g2.Graph.rmat(9, 8, seed=1).degeneracy_recoded(),
          g2.Graph.er(5000, 0.001, planted=10, planted_size=20, seed=2), g2.Graph.from_edges(0, []),
          _nested(g2, 300, 0.4, 4), g2.Graph.from_edges(3, [(0, 1), (1, 2), (0, 2)])]
    ctx.batch_load(gs)
    for q in (0, 24, 25):
        plan = Plan.preset(q)
        want = [orc.match(g, plan, threads=4)["count"] if g.n else 0 for g in gs]
        for kw in ({}, {"schedule": "heuristic"}):
            assert ctx.batch_match(plan, **kw).tolist() == want, (q, kw)


def _csr(g2, n, e):
    e = np.asarray(e, np.int64)
    e = e[e[:, 0] != e[:, 1]]
    key = np.unique(np.concatenate([e[:, 0] * n + e[:, 1], e[:, 1] * n + e[:, 0]]))
    rp = np.zeros(n + 1, np.uint64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return g2.Graph(rp, (key % n).astype(np.uint32))


def _sparse(g2, which):
    """Graphs whose roots are cheaper by their forward lists than by tiles."""
    rng = np.random.default_rng(4)
    if which == "far":  # small roots whose heads have no bit row
        return _csr(g2, 60000, np.stack([rng.integers(0, 60000, 900000), rng.integers(0, 60000, 900000)], 1))
    if which == "many":  # 1,300 roots of 65 to 300 vertices with hardly an edge among them
        d = np.tile([65, 66, 100, 129, 300], 260)
        e = np.stack([np.repeat(np.arange(1300), d), 1300 + rng.integers(0, 600, d.sum())], 1)
        return _csr(g2, 1900, np.concatenate([e, np.stack([1300 + rng.integers(0, 600, 500),
                                                           1300 + rng.integers(0, 600, 500)], 1)]))
    hub = np.stack([np.zeros(11999, int), np.arange(1, 12000)], 1)  # one wide root, a few triangles
    return _csr(g2, 12000, np.concatenate([hub, rng.integers(1, 12000, (3000, 2))]))


@pytest.mark.parametrize("which", ["far", "many", "hub"])
@pytest.mark.parametrize("q", [0, 24, 25])
def test_sparse_roots_by_their_lists(g2, orc, ctx, q, which):
    from g2aimd.context import Plan
    plan = Plan.preset(q)
    g = _sparse(g2, which)
    want = orc.match(g, plan, threads=8, per_root=True)
    src = np.arange(g.n - 1, -1, -3, dtype=np.uint32)
    ctx.load(g)
    for kw in ({}, {"schedule": "heuristic"}, {"schedule": "heuristic", "split": True, "granularity": 64},
               {"chunk": 5, "warps_per_block": 2}, {"schedule": "heuristic", "deadline_ms": 600000}):
        rc = np.zeros(g.n, np.uint64)
        assert ctx.match(plan, root_counts=rc, **kw) == want["count"], kw
        assert np.array_equal(rc, want["root_counts"]), kw
        assert ctx.match(plan, sources=src, **kw) == int(want["root_counts"][src].sum()), kw


@pytest.mark.parametrize("q,which", [(0, "hub"), (24, "many"), (25, "many")])
def test_sparse_roots_cost_what_they_hold(g2, ctx, q, which):
    """Roots with next to no cliques: the many take no longer than three plan walks, the
    hub (whose dense tiles took one warp 130 ms) no longer than 60 ms."""
    import time
    from g2aimd.context import Plan
    plan = Plan.preset(q)
    ctx.load(_sparse(g2, which))

    def best(**kw):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            ctx.match(plan, **kw)
            t.append(time.perf_counter() - t0)
        return min(t)

    for schedule in ("given", "heuristic"):
        limit = 0.06 if which == "hub" else 3 * best(schedule=schedule, intersect_mode=1)
        assert best(schedule=schedule) < limit, schedule
