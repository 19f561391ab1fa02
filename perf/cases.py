"""The work that is timed: what a user of this framework has it do, through the
calls of ``usap_b200.api``.

Graphs are seeded degree-corrected SBM graphs (``usap_b200.generator``) with the
shapes of the repository's own workloads: N from 1000 (plain solve on a small
graph) to 50000 (the headline graph), round(N^0.35) or the named number of
planted blocks, within-block fraction 0.5 to 0.8, Dirichlet alpha 1 or 10, and
nodal batches of a quarter (the default) or a tenth of the vertices.
"""
import math

import numpy as np
import torch

from usap_b200 import api, generator
from usap_b200 import native as nat

# Edges of a generated graph per vertex (out-degrees 5..100, mean about 15.8).
_DEG = 15.6
# Edges per vertex of an ingested file: that many of the graph's edges, so that every seed has as many.
_TSV_DEG = 13


def listed():
    return [
        # a small graph solved on a resident context: the smallest whole solve, where launches and host work count
        {"name": "solve_n1000", "kind": "solve", "n": 1000, "blocks": 11, "within": 0.8, "alpha": 10.0,
         "batches": 10, "precision": 3, "init_mode": 0},
        # an ordinary graph with overlapping blocks of uneven size, the default batch count
        {"name": "solve_n5000_hard", "kind": "solve", "n": 5000, "blocks": 19, "within": 0.5, "alpha": 1.0,
         "batches": 4, "precision": 3, "init_mode": 0},
        # started from one block per vertex: large B, an odd size
        {"name": "solve_n4999_singletons", "kind": "solve", "n": 4999, "blocks": 19, "within": 0.8, "alpha": 1.0,
         "batches": 10, "precision": 3, "init_mode": 1},
        # the one-shot call from host edge arrays: adjacency build, copies, solve, result copied back
        {"name": "oneshot_n20000", "kind": "oneshot", "n": 20000, "blocks": 32, "within": 0.5, "alpha": 1.0,
         "batches": 10, "precision": 3, "init_mode": 0},
        # the headline graph, graph resident
        {"name": "solve_n50000", "kind": "solve", "n": 50000, "blocks": 44, "within": 0.5, "alpha": 1.0,
         "batches": 10, "precision": 3, "init_mode": 0},
        # the same in exact FP64
        {"name": "solve_n50000_fp64", "kind": "solve", "n": 50000, "blocks": 44, "within": 0.5, "alpha": 1.0,
         "batches": 10, "precision": 0, "init_mode": 0},
        # many graphs, several chains each, in one call
        {"name": "batch_12x4", "kind": "batch", "graphs": 12, "chains": 4, "lo": 1000, "hi": 20000, "batches": 10,
         "precision": 3},
        # requests submitted together to a running service, all waited for
        {"name": "serve_24", "kind": "serve", "graphs": 24, "lo": 1000, "hi": 30000, "batches": 10, "precision": 3},
        # a stream: a weighted graph loaded and solved, new edges and vertices added, the solve continued
        {"name": "stream_n3001", "kind": "stream", "n": 3001, "blocks": 16, "within": 0.8, "alpha": 10.0,
         "batches": 10, "precision": 3},
        # ingest of the text of an edge list file
        {"name": "tsv_n50000", "kind": "tsv", "n": 50000, "blocks": 44, "within": 0.5, "alpha": 1.0},
        # a partition scored where it lies on the device
        {"name": "evaluate_n50000", "kind": "evaluate", "n": 50000, "b1": 44, "b2": 57},
        # the description length of a partition from device arrays, without allocation
        {"name": "entropy_n5000", "kind": "entropy", "n": 5000, "e": 79000, "b": 19},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "oneshot", "batch", "serve", "stream", "tsv", "evaluate", "entropy"])
    within, alpha = round(rng.uniform(0.5, 0.8), 3), rng.choice([1.0, 10.0])
    batches = rng.choice([4, 10])
    if kind in ("solve", "oneshot"):
        init = rng.choice([0, 0, 1, 2])
        n = _log_uniform(rng, 1000, 4999 if init == 1 else 50000)
        return {"kind": kind, "n": n, "blocks": max(1, round(n ** 0.35)), "within": within, "alpha": alpha,
                "batches": batches, "precision": rng.choice([3, 3, 0]), "init_mode": init}
    if kind == "batch":
        return {"kind": kind, "graphs": rng.randint(3, 11), "chains": rng.randint(1, 4), "lo": 1000,
                "hi": _log_uniform(rng, 4000, 20000), "batches": 10, "precision": rng.choice([3, 3, 0])}
    if kind == "serve":
        return {"kind": kind, "graphs": rng.randint(4, 20), "lo": 1000, "hi": _log_uniform(rng, 4000, 30000),
                "batches": 10, "precision": rng.choice([3, 3, 0])}
    if kind == "stream":
        n = _log_uniform(rng, 1000, 5000)
        return {"kind": kind, "n": n, "blocks": max(1, round(n ** 0.35)), "within": within, "alpha": alpha,
                "batches": 10, "precision": 3}
    if kind == "tsv":
        n = _log_uniform(rng, 1000, 50000)
        return {"kind": kind, "n": n, "blocks": max(1, round(n ** 0.35)), "within": within, "alpha": alpha}
    if kind == "evaluate":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 200000), "b1": rng.randint(5, 75), "b2": rng.randint(5, 90)}
    return {"kind": "entropy", "n": _log_uniform(rng, 1000, 60000), "e": _log_uniform(rng, 16000, 1000000),
            "b": _log_uniform(rng, 2, 1024)}


def _graph(case, seed):
    return generator.generate(generator.SBMConfig(n=case["n"], blocks=case["blocks"], within=case["within"],
                                                  alpha=case["alpha"], seed=seed))


def _graphs(case, seed):
    """Graphs of the batched and served workloads: sizes spread log-uniformly, other parameters drawn."""
    rng = np.random.default_rng(seed)
    k = case["graphs"]
    out = []
    for i in range(k):
        # sizes at equal steps of the log range, the same ones for every seed
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / k)))
        out.append(generator.generate(generator.SBMConfig(
            n=n, blocks=max(1, int(round(n ** 0.35))), within=float(rng.uniform(0.5, 0.8)),
            alpha=float(rng.choice([1.0, 10.0])), seed=int(rng.integers(0, 2**31 - 1)))))
    return [out[i] for i in np.random.default_rng(k).permutation(k)]


def _params(case, seed):
    return nat.default_params(num_batch_nodal_update=case["batches"], seed=seed, precision=case["precision"],
                              init_mode=case.get("init_mode", 0))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "oneshot"):
        g = _graph(case, seed)
        st = {"kind": kind, "graph": g, "params": _params(case, seed)}
        if kind == "solve":
            st["ctx"] = api.Context(0)
            st["ctx"].load(g.src, g.dst, None, g.n)
        return st
    if kind == "batch":
        return {"kind": kind, "graphs": _graphs(case, seed), "params": _params(case, seed),
                "seeds": [list(range(100 * i + seed % 97, 100 * i + seed % 97 + case["chains"]))
                          for i in range(case["graphs"])]}
    if kind == "serve":
        return {"kind": kind, "graphs": _graphs(case, seed), "params": _params(case, seed), "server": api.Server(0)}
    if kind == "stream":
        g = _graph(case, seed)
        rng = np.random.default_rng([seed, 1])
        w = rng.integers(1, 6, g.num_edges).astype(np.int32)
        n1 = (4 * g.n) // 5
        early = (g.src < n1) & (g.dst < n1) & (rng.random(g.num_edges) < 0.9)
        early |= (g.src < n1) & (g.dst < n1) & np.r_[True, g.src[1:] != g.src[:-1]]   # keep a first out-edge
        return {"kind": kind, "ctx": api.Context(0), "n": g.n, "n1": n1, "params": _params(case, seed),
                "a": (g.src[early], g.dst[early], w[early]), "b": (g.src[~early], g.dst[~early], w[~early])}
    if kind == "tsv":
        g = _graph(case, seed)
        rng = np.random.default_rng([seed, 4])
        keep = np.sort(rng.permutation(g.num_edges)[:_TSV_DEG * g.n])
        text = "".join(["%d\t%d\t1\n" % p for p in zip((g.src[keep] + 1).tolist(), (g.dst[keep] + 1).tolist())])
        return {"kind": kind, "ctx": api.Context(0), "text": text.encode(), "n": g.n}
    if kind == "evaluate":
        truth, given = _labels(case, seed)
        return {"kind": kind, "n": case["n"], "truth": torch.from_numpy(truth).cuda(),
                "given": torch.from_numpy(given).cuda()}
    src, dst, part = _edges(case, seed)
    return {"kind": kind, "n": case["n"], "b": case["b"], "src": torch.from_numpy(src).cuda(),
            "dst": torch.from_numpy(dst).cuda(), "part": torch.from_numpy(part).cuda(),
            "S_q": torch.zeros(1, dtype=torch.int64, device="cuda")}


def _labels(case, seed):
    """A planted partition and a found one: most vertices follow a block to block map, the rest are off."""
    rng = np.random.default_rng([seed, 2])
    n, b1, b2 = case["n"], case["b1"], case["b2"]
    truth = rng.choice(b1, size=n, p=rng.dirichlet(np.full(b1, 3.0))).astype(np.int32)
    given = rng.integers(0, b2, size=b1)[truth]
    off = rng.random(n) < 0.25
    given[off] = rng.integers(0, b2, size=int(off.sum()))
    truth[rng.random(n) < 0.01] = -1     # vertices whose truth is unknown
    return truth, given.astype(np.int32)


def _edges(case, seed):
    rng = np.random.default_rng([seed, 3])
    n, e, b = case["n"], case["e"], case["b"]
    part = rng.integers(0, b, n)
    src = rng.integers(0, n, e)
    dst = rng.integers(0, n, e)
    order = np.argsort(part, kind="stable")
    lo, hi = np.searchsorted(part[order], part[src]), np.searchsorted(part[order], part[src], side="right")
    own = rng.random(e) < 0.6            # that share of the edges stays in its block
    dst[own] = order[(lo + rng.integers(0, 1 << 30, e) % (hi - lo))[own]]
    k = np.sort(src * n + dst)
    return (k // n).astype(np.int32), (k % n).astype(np.int32), part.astype(np.int32)


def _solved(assign, res):
    return {"assign": assign, "B": res["B"], "S": res["S"], "S_q": res["S_q"], "stages": res["stages"],
            "sweeps": res["sweeps"], "moves": res["nodal_moves"], "proposals": res["nodal_proposals"]}


def run(st):
    kind = st["kind"]
    if kind == "solve":
        return _solved(*st["ctx"].partition(st["params"]))
    if kind == "oneshot":
        g = st["graph"]
        return _solved(*api.partition(g.src, g.dst, None, g.n, params=st["params"]))
    if kind == "batch":
        jobs, _ = api.batch_partition(st["graphs"], st["seeds"], st["params"])
        return {"assign": np.concatenate([j["assign"] for j in jobs]), "B": np.array([j["result"]["B"] for j in jobs]),
                "S": np.array([j["result"]["S"] for j in jobs]),
                "moves": np.array([j["result"]["nodal_moves"] for j in jobs])}
    if kind == "serve":
        tickets = [st["server"].submit(g.src, g.dst, None, g.n, params=st["params"]) for g in st["graphs"]]
        got = [st["server"].wait(t) for t in tickets]
        return {"assign": np.concatenate([a for a, _, _ in got]), "B": np.array([r["B"] for _, r, _ in got]),
                "S": np.array([r["S"] for _, r, _ in got]), "moves": np.array([r["nodal_moves"] for _, r, _ in got])}
    if kind == "stream":
        ctx, n, n1 = st["ctx"], st["n"], st["n1"]
        ctx.load(*st["a"], n1)
        p1, r1 = ctx.partition(st["params"])
        ctx.add_edges(*st["b"], n=n)
        init = np.concatenate([p1, r1["B"] + np.arange(n - n1, dtype=np.int32)])
        return {"first": _solved(p1, r1), "second": _solved(*ctx.partition_from(init, st["params"]))}
    if kind == "tsv":
        st["ctx"].load_tsv(st["text"], st["n"])
        return st["ctx"].adjacency()
    if kind == "evaluate":
        return api.evaluate_device(st["truth"].data_ptr(), st["given"].data_ptr(), st["n"])
    nat.check(nat.lib().usap_entropy_static(
        st["src"].data_ptr(), st["dst"].data_ptr(), None, st["src"].numel(), st["n"], st["part"].data_ptr(), st["b"],
        st["S_q"].data_ptr(), torch.cuda.current_stream().cuda_stream))
    return st["S_q"]


def _solve_work(n, batches, precision, init_mode=0):
    """One solve at its least: each stage halves B down to about N^0.35 and searches on for three stages more,
    each stage takes the three sweeps before the convergence test can end it, and a sweep reads every vertex's
    neighbours and their blocks in both directions and, for each proposal, its terms: 8 of every block in the
    float form, 8 of every edge in the exact one."""
    e = _DEG * n
    b = n / 2 if init_mode == 1 else n / 16
    sizes = []
    while b > n ** 0.35:
        sizes.append(b)
        b /= 2
    sizes += [1.5 * n ** 0.35] * 3
    terms = sum(3 * n * (8 * x if precision == 3 else 8 * _DEG * 2) for x in sizes)
    return {"bytes": len(sizes) * 3 * (16 * e + 12 * n), "flops": 2 * terms}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "oneshot"):
        w = _solve_work(case["n"], case["batches"], case["precision"], case["init_mode"])
        if kind == "oneshot":
            w["bytes"] += 8 * _DEG * case["n"] + 4 * case["n"]
        return w
    if kind in ("batch", "serve"):
        k = case["graphs"]
        all_ = [_solve_work(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / k), case["batches"],
                            case["precision"]) for i in range(k)]
        return {f: case.get("chains", 1) * sum(w[f] for w in all_) for f in ("bytes", "flops")}
    if kind == "stream":
        one, two = (_solve_work(x, case["batches"], case["precision"]) for x in (0.8 * case["n"], case["n"]))
        return {f: one[f] + two[f] for f in one}
    if kind == "tsv":
        n, e = case["n"], _TSV_DEG * case["n"]
        return {"bytes": e * (2 * len(str(n)) + 4) + 16 * e + 16 * n, "flops": 0}
    if kind == "evaluate":
        return {"bytes": 8 * case["n"] + 12 * case["b1"] * case["b2"], "flops": 15 * case["b1"] * case["b2"]}
    return {"bytes": 8 * case["e"] + 4 * case["n"] + 8, "flops": 4 * min(case["e"], case["b"] ** 2)}


def exact(case, seed):
    """The scores and the description length in 64 bits; a solve's outputs depend on its own draws and have no
    such value."""
    if case["kind"] == "evaluate":
        truth, given = (x.astype(np.int64) for x in _labels(case, seed))
        known = truth >= 0
        truth, given = truth[known], given[known]
        n = truth.size
        c = np.zeros((case["b1"], case["b2"]), np.int64)
        np.add.at(c, (truth, given), 1)
        r, s = c.sum(1), c.sum(0)
        plogp = lambda x: float((x[x > 0] / n * np.log(x[x > 0] / n)).sum())  # noqa: E731
        h1, h2, h12 = -plogp(r), -plogp(s), -plogp(c.reshape(-1))
        mi = h1 + h2 - h12
        pairs = lambda x: int((x * (x - 1) // 2).sum())  # noqa: E731
        same, p1, p2, every = pairs(c), pairs(r), pairs(s), n * (n - 1) // 2
        expected = p1 * p2 / every
        return {"accuracy": None, "rand_index": (every + 2 * same - p1 - p2) / every,
                "adjusted_rand_index": (same - p1 * p2 // every) / (0.5 * (p1 + p2) - p1 * p2 // every),
                "adjusted_rand_index_exact": (same - expected) / (0.5 * (p1 + p2) - expected),
                "pairwise_recall": same / p1, "pairwise_precision": same / p2, "h_truth": h1, "h_given": h2,
                "h_truth_given": h12 - h2, "h_given_truth": h12 - h1, "mi": mi, "nmi": 2 * mi / (h1 + h2),
                "nmi_sqrt": mi / math.sqrt(h1 * h2), "missed_info": (h12 - h2) / h1,
                "erroneous_info": (h12 - h1) / h2, "n": None, "b_truth": None, "b_given": None}
    return None
