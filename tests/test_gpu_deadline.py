"""MCE with a time budget (g2_opts.deadline_ms): past the budget warps start no
new root and drop the root they walk, so the run ends soon after and returns
G2_ERR_DEADLINE with the results of the roots that finished.  Those results are
exact: the count and histogram equal the oracle's over exactly the roots whose
search-tree node count is non-zero.  The limit is a device clock read, not a
fault: the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_generous_budget_changes_nothing(orc, c1_graph):
    from g2aimd.context import Context
    g = c1_graph
    want = orc.mce(g, hist_len=64)
    with Context(0) as c:
        c.load(g)
        count, hist, _rn = c.mce(hist_len=64, root_nodes=True, deadline_ms=60000)
        assert not c.expired
        assert count == want["count"] and np.array_equal(hist, want["hist"])


def test_budget_run_out_keeps_finished_roots_exact(g2, orc):
    from g2aimd.context import Context
    g = g2.Graph.rmat(14, 16, seed=1).degeneracy_recoded()
    with Context(0) as c:
        c.load(g)
        count, hist, rn = c.mce(hist_len=128, root_nodes=True, deadline_ms=5)
        assert c.expired
        done = np.flatnonzero(rn > 0).astype(np.uint32)
        assert 0 < done.size < g.n
        want = orc.mce(g, roots=done, hist_len=128, threads=8)
        assert count == want["count"] and np.array_equal(hist, want["hist"])
        # the context runs normally afterwards
        c2, _h2 = c.mce(sources=done[:256], hist_len=128)
        assert c2 == orc.mce(g, roots=done[:256], hist_len=128)["count"] and not c.expired


@pytest.mark.parametrize("q,budget", [(24, 1), (25, 2), (1, 5), (2, 5)])
def test_match_budget_keeps_finished_roots_exact(g2, orc, q, budget):
    """Plan-driven counts with a time budget: clique plans (bitmap path) and
    plan walks (4-cycles, diamonds).  Finished roots are the ones with a
    recorded cost; the count equals the oracle's over exactly those roots."""
    from g2aimd.context import Context, Plan
    g = g2.Graph.rmat(16, 16, seed=3).degeneracy_recoded()
    plan = Plan.preset(q)
    with Context(0) as c:
        c.load(g)
        c.load_core(g.core)
        full = c.match(plan, schedule="heuristic", flags=1)
        cost = np.zeros(g.n, np.uint64)
        got = c.match(plan, root_cost=cost, schedule="heuristic", flags=1, deadline_ms=budget)
        done = np.flatnonzero(cost > 0).astype(np.uint32)
        if c.expired:
            assert done.size < g.n and got <= full
        else:
            assert got == full
        want = orc.match(g, plan, roots=done, threads=8)["count"]
        assert got == want
        # generous budget: everything finishes
        assert c.match(plan, schedule="heuristic", flags=1, deadline_ms=600000) == full and not c.expired


def test_device_stream_status_reports_the_budget(g2):
    """g2_run_status gives a device-stream run's outcome: G2_ERR_DEADLINE when
    its budget ran out before every root finished (a run that takes more than
    ten times the budget), 0 for a run without one."""
    import torch
    from g2aimd.context import Context, Plan
    g = g2.Graph.rmat(16, 16, seed=3).degeneracy_recoded()
    dev = torch.device("cuda", 0)
    st = torch.cuda.Stream(dev)
    out = torch.zeros(1, dtype=torch.int64, device=dev)
    with Context(0) as c:
        c.load(g)
        c.load_core(g.core)
        c.set_plan(Plan.preset(1))  # 4-cycles: the plan walk
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        c.match_device(out.data_ptr(), stream=st.cuda_stream, schedule="heuristic", flags=1)
        e1.record(st)
        assert c.run_status(st.cuda_stream) == 0
        full, full_ms = int(out[0].item()), e0.elapsed_time(e1)
        c.match_device(out.data_ptr(), stream=st.cuda_stream, schedule="heuristic", flags=1, deadline_ms=1)
        code = c.run_status(st.cuda_stream)
        if full_ms > 10.0:
            assert code == -11 and int(out[0].item()) < full  # G2_ERR_DEADLINE
        else:
            assert code in (0, -11)


def test_budgeted_run_takes_roots_in_exact_cost_order(g2):
    """One warp under a time budget finishes a prefix of the schedule's order:
    descending heuristic cost, whole numbers below 2^24 here and many of them within
    a percent of each other, ties in the caller's order (a shuffled one here)."""
    from g2aimd.context import Context
    g = g2.Graph.er(5000, 0.02, seed=8).degeneracy_recoded()
    d = g.degrees().astype(np.float32)
    p = np.array([int((g.neighbors(v) > v).sum()) for v in range(g.n)], np.float32)
    src = np.random.default_rng(2).permutation(g.n).astype(np.uint32)
    order = np.argsort(-(p * (p + d) + np.float32(1))[src], kind="stable")
    with Context(0) as c:
        c.load(g)
        _n, _h, rn = c.mce(sources=src, root_nodes=True, schedule="heuristic", blocks=1, warps_per_block=1, chunk=1,
                           deadline_ms=20)
        assert c.expired
    done = rn[order] > 0
    k = int(done.sum())
    assert 20 < k < g.n and done[:k].all()


@pytest.mark.parametrize("schedule", ["given", "heuristic"])
@pytest.mark.parametrize("q,n,keep", [(0, 8000, 1.0), (24, 2500, 1.0), (25, 1100, 0.7)])
def test_clique_budget_runs_out_inside_a_root(g2, q, n, keep, schedule):
    """Counting the cliques over one root of n - 1 vertices takes many times the budget of
    1 ms: the run ends soon after it, drops the root and says so; the finished roots of
    a full run afterwards are unharmed."""
    import time
    from g2aimd.context import Context, Plan
    plan = Plan.preset(q)
    rng = np.random.default_rng(3)
    a, b = np.triu_indices(n - 1, 1)
    on = rng.random(a.size) < keep * (0.25 if n > 2000 else 1.0)
    row = np.concatenate([np.zeros(n - 1, np.int64), a[on] + 1])
    col = np.concatenate([np.arange(1, n), b[on] + 1])
    key = np.sort(np.concatenate([row * n + col, col * n + row]))
    rp = np.zeros(n + 1, np.uint64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    g = g2.Graph(rp, (key % n).astype(np.uint32))
    src = np.zeros(1, np.uint32)
    with Context(0) as c:
        c.load(g)
        full = c.match(plan, sources=src, schedule=schedule)
        t0 = time.perf_counter()
        assert c.match(plan, sources=src, schedule=schedule) == full
        full_ms = 1e3 * (time.perf_counter() - t0)
        cost = np.zeros(1, np.uint64)
        got = c.match(plan, sources=src, schedule=schedule, deadline_ms=1, root_cost=cost)  # loads the kernels
        t0 = time.perf_counter()
        got = c.match(plan, sources=src, schedule=schedule, deadline_ms=1, root_cost=cost)
        ms = 1e3 * (time.perf_counter() - t0)
        assert full_ms > 6, full_ms
        assert c.expired and got == 0 and cost[0] == 0, (full_ms, ms)
        # (5-cliques look at the clock once per highest vertex of the root)
        assert ms < (0.9 if q == 25 else 0.5) * full_ms, (full_ms, ms)
        assert c.match(plan, sources=src, schedule=schedule, deadline_ms=600000) == full and not c.expired
