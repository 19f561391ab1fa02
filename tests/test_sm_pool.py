"""The SMs handed out to concurrent solves' nodal phases: one pool per device
for every context, batch and server, never more CTAs than are resident
together (a phase's CTAs wait for one another)."""
import os
import subprocess
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sm_pool_accounting(tmp_path):
    csrc = os.path.join(ROOT, "usap_b200", "csrc")
    exe = str(tmp_path / "sm_pool_main")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", csrc,
                    os.path.join(ROOT, "tests", "sm_pool", "sm_pool_main.cpp"), os.path.join(csrc, "smpool.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


@pytest.mark.gpu
def test_server_batch_and_contexts_at_once():
    """A server, a batch and contexts on two threads solve at the same time:
    every result equals the one solved alone."""
    from usap_b200 import api, generator as gen, native as nat
    graphs = [gen.generate(gen.SBMConfig(n=n, blocks=max(1, round(n ** 0.35)), within=0.6, alpha=2.0, seed=n))
              for n in (150, 1201, 3000, 9001)]
    params = lambda s: nat.default_params(num_batch_nodal_update=10, seed=s)  # noqa: E731
    alone = {(i, s): api.partition(g.src, g.dst, None, g.n, params=params(s))
             for i, g in enumerate(graphs) for s in (1, 2)}

    def same(got, key):
        return np.array_equal(got[0], alone[key][0]) and got[1]["S_q"] == alone[key][1]["S_q"]

    bad = []

    def context(i):
        g = graphs[i]
        ctx = api.Context(0)
        ctx.load(g.src, g.dst, None, g.n)
        for s in (1, 2):
            if not same(ctx.partition(params(s)), (i, s)):
                bad.append(("context", i, s))
        ctx.close()

    def batch():
        jobs, _ = api.batch_partition(graphs, [[1, 2]] * len(graphs), params(0))
        bad.extend(("batch", j["graph"], j["seed"]) for j in jobs
                   if not same((j["assign"], j["result"]), (j["graph"], j["seed"])))

    def run(fn, *a):
        def f():
            try:
                fn(*a)
            except Exception as e:  # a thread's failure is the test's
                bad.append(repr(e))
        return threading.Thread(target=f)

    srv = api.Server(0)
    tickets = [(srv.submit(g.src, g.dst, None, g.n, params=params(s)), (i, s))
               for i, g in enumerate(graphs) for s in (1, 2)]
    threads = [run(context, 3), run(context, 1), run(batch)]
    for t in threads:
        t.start()
    for t, key in tickets:
        got = srv.wait(t)
        if not same(got[:2], key):
            bad.append(("server",) + key)
    for t in threads:
        t.join()
    srv.close()
    assert not bad, bad


@pytest.mark.gpu
def test_concurrent_forms_without_cooperative_launches():
    """persistent = 0 holds in the batched and served forms too: launches per
    batch, the same results."""
    from usap_b200 import api, generator as gen, native as nat
    graphs = [gen.generate(gen.SBMConfig(n=n, blocks=5, within=0.7, alpha=2.0, seed=n)) for n in (300, 900)]
    alone = [api.partition(g.src, g.dst, None, g.n, params=nat.default_params(seed=1)) for g in graphs]
    jobs, stats = api.batch_partition(graphs, [[1], [1]], nat.default_params(persistent=0))
    assert stats["gang_launches"] == 0
    srv = api.Server(0)
    for g, (part, res), j in zip(graphs, alone, jobs):
        p, r, _ = srv.wait(srv.submit(g.src, g.dst, None, g.n, params=nat.default_params(seed=1, persistent=0)))
        assert np.array_equal(j["assign"], part) and j["result"]["S_q"] == res["S_q"]
        assert np.array_equal(p, part) and r["S_q"] == res["S_q"]
    srv.close()
    assert api.batch_partition(graphs, [[1], [1]], nat.default_params())[1]["gang_launches"] > 0


@pytest.mark.gpu
def test_workers_are_those_that_solve():
    from usap_b200 import api, generator as gen, native as nat
    g = gen.generate(gen.SBMConfig(n=200, blocks=4, within=0.8, alpha=5.0, seed=1))
    for asked in (0, 3, 32):
        srv = api.Server(0, workers=asked)
        want = srv.stats()["workers"]
        assert want == 3 if asked == 3 else 1 <= want <= 8
        tickets = [srv.submit(g.src, g.dst, None, g.n) for _ in range(20)]
        for t in tickets:
            srv.wait(t)
        assert 1 <= srv.stats()["peak_running"] <= want
        srv.close()
        _, stats = api.batch_partition([g], [list(range(12))], nat.default_params(), workers=asked)
        assert stats["workers"] == (3 if asked == 3 else 8)
