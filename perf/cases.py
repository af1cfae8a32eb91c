"""Performance cases of the framework: maximal cliques, plan-driven counts,
batches, end-to-end loads and degeneracy recoding, each through the public
Python entry points (g2aimd.Graph, g2aimd.context.Context) on seeded synthetic
graphs of the shapes that bench.py and the tests use.

A case is a dict: `kind` picks the entry points, `graph` the generator
("rmat": 2^scale vertices and `ef` edges per vertex; "cl": Chung-Lu with `n`,
`gamma`, `deg`; "er": G(n, p) with planted cliques), the other keys are sizes
and options.  The seed passed to prepare() is the generator's seed.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "g2-aimd_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import g2aimd  # noqa: E402
from g2aimd.context import FLAG_NO_SPLIT, Context, CostModel, Plan  # noqa: E402

HIST = 256
CLIQUE_PRESET = {3: 0, 4: 24, 5: 25}  # triangle, 4-clique, 5-clique
# the launch parameters the benchmark's autotuner settles on for its 4-clique workload (bench.py --fixed)
TUNED = {"flags": FLAG_NO_SPLIT, "granularity": 64, "warps_per_block": 4, "chunk": 1, "ctas_per_sm": 6}


def listed():
    return [
        # the smallest calls, where latency and launches count: the test suite's G(2000, 0.01) with five planted K12
        {"name": "mce_er2000", "kind": "mce", "graph": "er", "n": 2000, "p": 0.01, "schedule": "given"},
        {"name": "k4_er2000", "kind": "clique", "graph": "er", "n": 2000, "p": 0.01, "k": 4, "schedule": "given",
         "tuned": False},
        # triangles of a mid-sized graph, every option at its default
        {"name": "tri_rmat18", "kind": "clique", "graph": "rmat", "scale": 18, "ef": 16, "k": 3,
         "schedule": "given", "tuned": False},
        # the benchmark's headline: 4-cliques of R-MAT scale 20, edge factor 16, learned schedule, tuned launch
        {"name": "k4_rmat20", "kind": "clique", "graph": "rmat", "scale": 20, "ef": 16, "k": 4,
         "schedule": "learned", "tuned": True},
        # 5-cliques, the deepest counts of the clique path: R-MAT scale 16
        {"name": "k5_rmat16", "kind": "clique", "graph": "rmat", "scale": 16, "ef": 16, "k": 5,
         "schedule": "heuristic", "tuned": False},
        # plan walks over a power-law graph with hubs: 4-cycles and diamonds (bench.py --leg walk)
        {"name": "cycle4_cl200k", "kind": "walk", "graph": "cl", "n": 200000, "gamma": 2.2, "deg": 20.0,
         "preset": 1, "schedule": "heuristic"},
        {"name": "diamond_cl200k", "kind": "walk", "graph": "cl", "n": 200000, "gamma": 2.2, "deg": 20.0,
         "preset": 2, "schedule": "heuristic"},
        # maximal cliques of a power-law graph (bench.py --leg mce) and of a dense core with planted cliques (--leg c3)
        {"name": "mce_cl262k", "kind": "mce", "graph": "cl", "n": 1 << 18, "gamma": 2.3, "deg": 16.0,
         "schedule": "heuristic"},
        {"name": "mce_rmat13_planted", "kind": "mce", "graph": "rmat", "scale": 13, "ef": 16, "planted": 50,
         "schedule": "heuristic"},
        # many small graphs in one call (bench.py --leg c4): maximal cliques and triangles of each
        {"name": "batch24_cl", "kind": "batch", "graph": "cl", "count": 24, "n_lo": 1000, "n_hi": 60000,
         "gamma": 2.4, "deg": 16.0},
        # a new graph with every call, from pinned host memory to the count (bench.py's end-to-end leg)
        {"name": "load_k4_rmat17", "kind": "load", "graph": "rmat", "scale": 17, "ef": 16, "k": 4},
        # a raw graph on the device to its degeneracy order, recoded CSR and triangle count
        {"name": "recode_rmat18", "kind": "recode", "graph": "rmat", "scale": 18, "ef": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mce", "clique", "clique", "walk", "batch", "load", "recode"])
    sched = rng.choice(["given", "heuristic", "learned"])
    if kind == "clique":
        k = rng.choice([3, 4, 5])
        if rng.random() < 0.5:
            return {"kind": "clique", "graph": "rmat", "scale": rng.randint(11, {3: 19, 4: 19, 5: 15}[k]),
                    "ef": rng.randint(6, 16), "k": k, "schedule": sched, "tuned": rng.random() < 0.5}
        return {"kind": "clique", "graph": "cl", "n": _log(rng, 2000, 300000), "gamma": round(rng.uniform(2.2, 2.8), 2),
                "deg": round(rng.uniform(8.0, 24.0), 1), "k": k, "schedule": sched, "tuned": rng.random() < 0.5}
    if kind == "walk":
        return {"kind": "walk", "graph": "cl", "n": _log(rng, 2000, 190000), "gamma": round(rng.uniform(2.25, 2.8), 2),
                "deg": round(rng.uniform(6.0, 19.0), 1), "preset": rng.choice([1, 2]),
                "schedule": rng.choice(["given", "heuristic"])}
    if kind == "mce":
        g = rng.choice(["er", "cl", "cl", "rmat"])
        if g == "er":
            n = _log(rng, 500, 8000)
            return {"kind": "mce", "graph": "er", "n": n, "p": round(rng.uniform(10.0, 40.0) / n, 5), "schedule": sched}
        if g == "cl":
            return {"kind": "mce", "graph": "cl", "n": _log(rng, 2000, 250000), "gamma": round(rng.uniform(2.35, 2.8), 2),
                    "deg": round(rng.uniform(6.0, 16.0), 1), "schedule": sched}
        return {"kind": "mce", "graph": "rmat", "scale": rng.randint(8, 12), "ef": rng.randint(8, 16),
                "planted": rng.randint(0, 20), "schedule": sched}
    if kind == "batch":
        lo = _log(rng, 500, 5000)
        return {"kind": "batch", "graph": "cl", "count": rng.randint(3, 24), "n_lo": lo, "n_hi": lo * rng.randint(2, 8),
                "gamma": round(rng.uniform(2.4, 2.8), 2), "deg": round(rng.uniform(6.0, 16.0), 1)}
    if kind == "load":
        return {"kind": "load", "graph": "rmat", "scale": rng.randint(11, 16), "ef": rng.randint(6, 16),
                "k": rng.choice([3, 4])}
    if rng.random() < 0.5:
        return {"kind": "recode", "graph": "rmat", "scale": rng.randint(11, 17), "ef": rng.randint(6, 16)}
    return {"kind": "recode", "graph": "cl", "n": _log(rng, 2000, 300000), "gamma": round(rng.uniform(2.2, 2.8), 2),
            "deg": round(rng.uniform(6.0, 20.0), 1)}


def _into(ctx, case, seed):
    """The case's raw graph (generator's ids) as the context's graph."""
    if case["graph"] == "rmat":
        ctx.gen_rmat(case["scale"], case["ef"], planted=case.get("planted", 0), pmin=20, pmax=60, seed=seed)
    elif case["graph"] == "er":
        ctx.load(g2aimd.Graph.er(case["n"], case["p"], planted=5, planted_size=12, seed=seed))
    else:
        ctx.load(g2aimd.Graph.chung_lu(case["n"], case["gamma"], case["deg"], seed=seed))


def _model(name):
    return CostModel.load(os.path.join(_PKG, "models", name + ".npz"))


class _Pinned:
    """A recoded host graph and its core numbers in pinned memory."""

    def __init__(self, g):
        self.keep = [torch.from_numpy(g.row_ptrs.view(np.int64)).pin_memory(),
                     torch.from_numpy(g.cols.view(np.int32)).pin_memory(),
                     torch.from_numpy(g.core.view(np.int32)).pin_memory()]
        rp, ci, core = (t.numpy() for t in self.keep)
        self.graph = g2aimd.Graph(rp.view(np.uint64), ci.view(np.uint32))
        self.core = core.view(np.uint32)


def prepare(case, seed):
    kind = case["kind"]
    ctx = Context(0)
    state = {"case": case, "ctx": ctx}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        sizes = np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"])).round().astype(int)
        ctx.batch_load([g2aimd.Graph.chung_lu(int(n), case["gamma"], case["deg"],
                                              seed=int(rng.integers(1, 1 << 31))).degeneracy_recoded() for n in sizes])
        ctx.set_model(_model("mce"))
        state["plan"] = Plan.preset(0)
    elif kind == "load":
        g = g2aimd.Graph.rmat(case["scale"], case["ef"], seed=seed).degeneracy_recoded()
        state["pinned"] = _Pinned(g)
        ctx.set_model(_model("k4"))
        ctx.load(state["pinned"].graph)
        state["plan"] = Plan.preset(CLIQUE_PRESET[case["k"]])
    elif kind == "recode":
        if case["graph"] == "rmat":
            m = ctx.gen_rmat(case["scale"], case["ef"], seed=seed)
            g = ctx.copy_csr(m)
        else:
            g = g2aimd.Graph.chung_lu(case["n"], case["gamma"], case["deg"], seed=seed)
        state["rp"] = torch.from_numpy(g.row_ptrs.view(np.int64)).cuda()
        state["ci"] = torch.from_numpy(g.cols.view(np.int32)).cuda()
        state["n"], state["m"] = g.n, g.m
        ctx.load_device(state["rp"].data_ptr(), state["ci"].data_ptr(), g.n, g.m)
        state["plan"] = Plan.preset(0)
    else:
        _into(ctx, case, seed)
        ctx.degeneracy_recode()  # the context keeps the recoded CSR and its core numbers
        if case["schedule"] == "learned":
            ctx.set_model(_model("mce" if kind == "mce" else "k4"))
        if kind == "clique":
            state["plan"] = Plan.preset(CLIQUE_PRESET[case["k"]])
        elif kind == "walk":
            state["plan"] = Plan.preset(case["preset"])
    ctx.reserve()
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "mce":
        count, hist = ctx.mce(hist_len=HIST, schedule=case["schedule"])
        return count, hist
    if kind == "clique":
        return ctx.match(state["plan"], schedule=case["schedule"], **(TUNED if case["tuned"] else {}))
    if kind == "walk":
        return ctx.match(state["plan"], schedule=case["schedule"])
    if kind == "batch":
        counts, hist = ctx.batch_mce(hist_len=HIST, schedule="learned")
        return counts, hist, ctx.batch_match(state["plan"], schedule="heuristic")
    if kind == "load":
        p = state["pinned"]
        ctx.load(p.graph)
        ctx.load_core(p.core)
        return ctx.match(state["plan"], schedule="learned", **TUNED)
    ctx.load_device(state["rp"].data_ptr(), state["ci"].data_ptr(), state["n"], state["m"])
    perm, core = ctx.degeneracy_recode()
    return perm, core, ctx.match(state["plan"], schedule="heuristic")


def _size(case):
    """(vertices, directed entries) the generator aims at (before duplicate edges drop out)."""
    if case["kind"] == "batch":
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)  # mean of a log-uniform size
        return n, n * case["deg"]
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, 2.0 * case["ef"] * n
    if case["graph"] == "er":
        return case["n"], case["n"] * case["n"] * case["p"] + 5 * 12 * 11
    return case["n"], case["n"] * case["deg"]


def work(case):
    """The CSR read once (per job of a batch), and what a pass writes: counts
    and histogram, or the permutation, core numbers and recoded CSR."""
    n, m = _size(case)
    csr = 8.0 * (n + 1) + 4.0 * m
    b = csr + 8.0
    if case["kind"] == "mce":
        b += 8.0 * HIST
    elif case["kind"] == "batch":
        b = 2.0 * csr + 16.0 * case["count"] + 8.0 * HIST
    elif case["kind"] == "load":
        b = csr + 4.0 * n + 8.0
    elif case["kind"] == "recode":
        b = 2.0 * csr + 8.0 * n + 8.0
    return {"bytes": b, "flops": 0.0}


def exact(case, seed):
    """Counts and orders are whole numbers and are compared as such: no output has a rounding error."""
    return None
