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
