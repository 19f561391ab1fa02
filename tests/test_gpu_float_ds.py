"""The float nodal dS of the persistent kernels at the edges of its variants,
whole solves against the oracle bit for bit.

A solve from one block per vertex (init_mode 1) has its first nodal phase at
N / 2 blocks and halves from there, so each graph passes through several of
the variants: the tile copied to shared memory (B <= 88), full tiles, sparse
tiles (under a fifth as many edges as cells), neighbour weights in 2 or 4
bytes a block (B <= 1536 and 768, half as much for two vertices a warp) or
hashed, and hubs proposed by a warp (up to 2048 neighbours and 768 blocks) or
by a CTA with its table in shared or global memory.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, e, hub=0, heavy=0, isolated=0, seed=1):
    """Random edges with a planted half, `hub` more at vertex 3 each way, one
    vertex of weight `heavy`, `isolated` vertices without edges."""
    rng = np.random.default_rng(seed)
    src, dst = rng.integers(0, n, e), rng.integers(0, n, e)
    near = rng.random(e) < 0.6
    dst[near] = (src[near] // 40 * 40 + rng.integers(0, 40, int(near.sum()))) % n
    if hub:
        other = rng.permutation(n)[:hub] if hub <= n else rng.integers(0, n, hub)
        src, dst = np.concatenate([src, np.full(hub, 3), other]), np.concatenate([dst, other, np.full(hub, 3)])
    w = None
    if heavy:
        w = rng.integers(1, 4, src.size)
        w[np.nonzero(src == 5)[0][0]] = heavy
    return n + isolated, src.astype(np.int32), dst.astype(np.int32), None if w is None else w.astype(np.int32)


CASES = {
    # the limits of the array forms of the neighbour weights, on sparse and on full tiles
    "sparse_768": (dict(n=1536, e=20000), {}),
    "sparse_769": (dict(n=1538, e=20000), {}),
    "sparse_1537": (dict(n=3074, e=40000, isolated=3), {}),
    "full_769": (dict(n=1538, e=130000), {}),
    "full_1537": (dict(n=3074, e=480000), {}),
    # odd sizes down to a few blocks; few vertices a batch, and more than one
    # wave of one CTA
    "small_odd": (dict(n=179, e=3001), {"num_batch_nodal_update": 7}),
    "one_cta": (dict(n=700, e=9001), {"num_batch_nodal_update": 2, "persistent_ctas": 1}),
    # hubs: 2 bytes a block, 4 bytes, by a CTA with its table in shared and in global memory
    "hub_110": (dict(n=900, e=9000, hub=110), {}),
    "hub_400": (dict(n=900, e=9000, hub=400), {}),
    "hub_1500": (dict(n=900, e=9000, hub=1500), {}),
    "hub_2000_B2600": (dict(n=5200, e=20000, hub=2000), {"max_num_nodal_itr": 1}),
    # weights, and a weighted degree beyond 16 bits
    "weighted": (dict(n=400, e=6000, heavy=9), {}),
    "heavy": (dict(n=400, e=6000, heavy=70000), {}),
    # the exact value evaluated beside it
    "shadow": (dict(n=500, e=9000, hub=150), {"fp64_shadow": 1}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_float_ds_solve_exact(oracle, name):
    from usap_b200 import api, native as nat
    spec, extra = CASES[name]
    n, src, dst, w = _graph(**spec)
    params = {"num_batch_nodal_update": 10, "seed": 5, "init_mode": 1, "max_num_nodal_itr": 2, **extra}
    ctx = api.Context(0)
    ctx.load(src, dst, w, n)
    part, res = ctx.partition(nat.default_params(**params))
    ctx.close()
    opar = {k: v for k, v in params.items() if k not in ("persistent_ctas", "fp64_shadow")}
    opart, ores, _ = oracle.OracleGraph(n, src, dst, w).partition(opar)
    assert np.array_equal(part, opart)
    assert (res["B"], res["S_q"], res["sweeps"], res["nodal_moves"]) == (
        ores["B"], ores["S_q"], ores["sweeps"], ores["nodal_moves"])


def test_float_ds_batch_exact(oracle):
    """The same through the batched form, jobs of several variants at once."""
    import types
    from usap_b200 import api, native as nat
    graphs = [types.SimpleNamespace(n=g[0], src=g[1], dst=g[2], weight=g[3])
              for g in (_graph(**CASES[k][0]) for k in ("sparse_769", "small_odd", "hub_400", "hub_1500", "heavy"))]
    params = {"num_batch_nodal_update": 10, "init_mode": 1, "max_num_nodal_itr": 2}
    jobs, _ = api.batch_partition(graphs, [[1, 2]] * len(graphs), nat.default_params(**params))
    for j in jobs:
        g = graphs[j["graph"]]
        opart, ores, _ = oracle.OracleGraph(g.n, g.src, g.dst, g.weight).partition(dict(params, seed=j["seed"]))
        assert np.array_equal(j["assign"], opart), (j["graph"], j["seed"])
        assert j["result"]["S_q"] == ores["S_q"]
