"""Degeneracy order and recode on the device where the peel and the row sort
change their ways: vertices wider than a piece, shells that collapse at once,
gaps between levels, rows around the bitmap sort's threshold, isolated ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases(g2):
    rng = np.random.default_rng(3)
    star = [(0, i) for i in range(1, 5000)]
    rows = []  # hubs of 254 .. 258 neighbours (the threshold is 256 here)
    for h, d in enumerate((254, 255, 256, 257, 258, 1023, 1024)):
        rows += [(h, int(x)) for x in rng.choice(np.arange(10, 3000), d, replace=False)]
    full = [(i, j) for i in range(300) for j in range(i)]  # one shell, every level below it empty
    mixed = full + [(300 + i, i % 300) for i in range(2000)]
    return [g2.Graph.from_edges(5000, star), g2.Graph.from_edges(3000, rows), g2.Graph.from_edges(300, full),
            g2.Graph.from_edges(2400, mixed), g2.Graph.from_edges(70000, [(1, 69999)]),
            g2.Graph.rmat(15, 16, seed=9)]


def test_order_and_recode_equal_the_host(g2):
    from g2aimd.context import Context
    with Context(0) as c:
        for g in _cases(g2):
            perm_h, core_h = g.degeneracy_order()
            want = g.recode(perm_h)
            c.load(g)
            perm, core = c.degeneracy_order()
            assert np.array_equal(core, core_h) and np.array_equal(perm, perm_h), (g.n, g.m)
            perm, core = c.degeneracy_recode()
            got = c.copy_csr(g.m)
            assert np.array_equal(perm, perm_h) and np.array_equal(core, core_h), (g.n, g.m)
            assert np.array_equal(got.row_ptrs, want.row_ptrs) and np.array_equal(got.cols, want.cols), (g.n, g.m)


def test_repeated_neighbours_stay(g2):
    """Rows that name neighbours twice (lists are to be deduplicated, but such a graph
    was taken as it is): long rows, which are sorted by a bitmap of distinct ids, keep
    them like short ones, and no entry is left unwritten."""
    from g2aimd.context import Context
    rng = np.random.default_rng(6)
    hub = np.stack([np.zeros(900, int), rng.permutation(np.arange(1, 3000))[:900]], 1)
    e = np.concatenate([hub, hub[:37], np.stack([rng.integers(0, 3000, 4000), rng.integers(0, 3000, 4000)], 1)])
    e = e[e[:, 0] != e[:, 1]]
    both = np.concatenate([e, e[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    rp = np.zeros(3001, np.uint64)
    rp[1:] = np.cumsum(np.bincount(both[:, 0], minlength=3000))
    g = g2.Graph(rp, both[:, 1].astype(np.uint32))
    perm_h, core_h = g.degeneracy_order()
    want = g.recode(perm_h)
    with Context(0) as c:
        c.load(g)
        perm, core = c.degeneracy_recode()
        got = c.copy_csr(g.m)
    assert np.array_equal(perm, perm_h) and np.array_equal(core, core_h)
    assert np.array_equal(got.row_ptrs, want.row_ptrs) and np.array_equal(got.cols, want.cols)


def test_rows_over_several_spans_of_ids(g2):
    """2.5 million vertices: a row's new ids lie in three spans of the bitmap (2^20 ids
    each), rows around the threshold of n >> 10 among them."""
    from g2aimd.context import Context
    rng = np.random.default_rng(9)
    n = 2500000
    rows = []
    for h, d in enumerate((2440, 2441, 2442, 5000, 60000)):
        rows.append(np.stack([np.full(d, h * 500000), rng.choice(np.arange(1, n, 2), d, replace=False)], 1))
    rows.append(np.stack([rng.integers(0, n, 3000000), rng.integers(0, n, 3000000)], 1))
    e = np.concatenate(rows)
    e = e[e[:, 0] != e[:, 1]]
    key = np.unique(np.concatenate([e[:, 0] * n + e[:, 1], e[:, 1] * n + e[:, 0]]))
    rp = np.zeros(n + 1, np.uint64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    g = g2.Graph(rp, (key % n).astype(np.uint32))
    perm_h, core_h = g.degeneracy_order()
    want = g.recode(perm_h)
    long_rows = np.flatnonzero(np.diff(want.row_ptrs).astype(np.int64) >= n >> 10)
    spans = [set((want.neighbors(v) >> 20).tolist()) for v in long_rows]
    assert len(long_rows) >= 3 and any(s == {0, 1, 2} for s in spans)
    with Context(0) as c:
        c.load(g)
        perm, core = c.degeneracy_recode()
        got = c.copy_csr(g.m)
    assert np.array_equal(perm, perm_h) and np.array_equal(core, core_h)
    assert np.array_equal(got.row_ptrs, want.row_ptrs) and np.array_equal(got.cols, want.cols)


@pytest.mark.parametrize("blocks", [1, 2, 37])
def test_order_with_fewer_resident_ctas(g2, monkeypatch, blocks):
    """A context that may not keep a CTA on every SM peels with fewer."""
    from g2aimd.context import Context
    monkeypatch.setenv("G2_PEEL_BLOCKS", str(blocks))
    g = g2.Graph.rmat(14, 12, seed=4)
    perm_h, core_h = g.degeneracy_order()
    with Context(0) as c:
        c.load(g)
        perm, core = c.degeneracy_order()
    assert np.array_equal(core, core_h) and np.array_equal(perm, perm_h)
