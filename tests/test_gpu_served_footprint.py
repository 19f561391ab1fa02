"""The served form's estimate of a request's device memory: an upper bound of
what the solve holds, without term tables that the float nodal dS never has
(a tile that it packs has none), so that a request which fits is not refused."""
import numpy as np
import pytest

from usap_b200 import generator as gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("init_mode", [0, 1])
def test_request_within_its_own_memory_is_admitted(init_mode):
    from cuda.bindings import driver as cu, runtime as rt

    from usap_b200 import api, native as nat
    n = 6000
    G = gen.generate(gen.SBMConfig(n=n, blocks=8, within=0.8, alpha=5, seed=3))
    e = G.num_edges
    params = nat.default_params(num_batch_nodal_update=10, seed=1, init_mode=init_mode)
    want, wres = api.partition(G.src, G.dst, None, n, params=params)
    # the tile pair at B = n and its chunk sums; the graph and the state are
    # bounded by 200 e + 400 n bytes, and 16 MiB is for the rest.  Term tables
    # up to 4096 blocks would add 128 MiB.
    budget = 8 * (n + 4) ** 2 + 4 * n * (n // 128 + 2) + 200 * e + 400 * n + (16 << 20)
    srv = api.Server(workers=1, memory_budget=budget)
    pool = rt.cudaDeviceGetDefaultMemPool(0)[1]
    attr = rt.cudaMemPoolAttr
    before = int(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)[1])
    rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, cu.cuuint64_t(0))
    part, res, _ = srv.wait(srv.submit(G.src, G.dst, None, n, params=params))
    peak = int(rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh)[1]) - before
    admitted = srv.stats()["peak_admitted_bytes"]
    srv.close()
    assert np.array_equal(part, want) and res["S_q"] == wres["S_q"]
    assert 0 < peak <= admitted <= budget
