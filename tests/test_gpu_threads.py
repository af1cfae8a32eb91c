"""Contexts in several threads of one process: launches of the same kernels with
different CTA sizes must not take the shared-memory limit from one another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_threads_with_different_cta_sizes(g2, orc):
    """6-cliques over a hub of 1,500 forward neighbours (rows of two words per lane:
    67 KB of shared memory per CTA of 8 warps, 17 KB per CTA of 2) and maximal
    cliques, each thread with a context and CTA size of its own."""
    from g2aimd.context import Context, Plan
    a, b = np.triu_indices(12, 1)
    g = g2.Graph.from_edges(1501, np.concatenate([np.stack([np.zeros(1500, int), np.arange(1, 1501)], 1),
                                                  np.stack([a + 1000, b + 1000], 1)]))
    plan = Plan.preset(26)
    want = orc.match(g, plan, threads=4)["count"]
    want_mce = orc.mce(g, threads=4)["count"]
    assert plan.k == 6 and want > 0
    bad = []

    def run(warps):
        try:
            with Context(0, scratch_bytes=256 << 20) as c:
                c.load(g)
                for _ in range(200):
                    got = c.match(plan, warps_per_block=warps), c.mce(warps_per_block=warps)[0]
                    if got != (want, want_mce):
                        bad.append((warps, got))
        except Exception as e:
            bad.append((warps, repr(e)))

    threads = [threading.Thread(target=run, args=(w,)) for w in (8, 2, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
