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


@pytest.mark.parametrize("q", [0, 24, 25])
def test_rows_in_slabs_and_beyond(g2, orc, q):
    """A complete-ish core of 420 vertices: its rows exceed the shared memory of a
    CTA of one warp and, with small scratch, the slabs too (the rest list)."""
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
