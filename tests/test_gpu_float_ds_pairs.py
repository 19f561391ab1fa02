"""The float nodal dS where two vertices share a warp, whole solves against the
oracle bit for bit.

A batch gets two vertices a warp when it has more than 24 vertices per CTA, so
these solves run on one or two CTAs.  From one block per vertex the first
nodal phase has N / 2 blocks, on both sides of the limits up to which a
half-warp keeps its neighbour weights in arrays (768 blocks with unit weights,
384 with others), hashed beyond; on sparse tiles and on full ones, whose
old-state terms come from tables there, and once on every SM.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, e, weighted=False, seed=3):
    """Edges of which a quarter of the vertices hold most, so that the others'
    degrees stay below the 64 of a half-warp."""
    rng = np.random.default_rng(seed)
    src, dst = rng.integers(0, n, e), rng.integers(0, n, e)
    full = rng.random(e) < 0.8
    src[full] = src[full] // 4 * 4
    dst[full] = dst[full] // 4 * 4
    near = rng.random(e) < 0.5
    dst[near] = (src[near] // 40 * 40 + rng.integers(0, 40, int(near.sum()))) % n
    w = rng.integers(1, 4, e).astype(np.int32) if weighted else None
    return src.astype(np.int32), dst.astype(np.int32), w


CASES = {
    "sparse_384_w": (768, 8000, True, {}),
    "sparse_385_w": (770, 8000, True, {}),
    "sparse_768": (1536, 20000, False, {}),
    "sparse_769": (1538, 20000, False, {}),
    "sparse_769_w_two_ctas": (1538, 20000, True, {"persistent_ctas": 2}),
    "full_384": (768, 30000, False, {}),
    "full_384_w": (768, 30000, True, {}),
    "full_385_w": (770, 30000, True, {}),
    "full_768": (1536, 118500, False, {}),
    "full_769": (1538, 118500, False, {}),
    "full_769_w": (1538, 118500, True, {}),
    "full_769_tables_on_every_sm": (1538, 118500, False, {"persistent_ctas": 0}),
    "odd": (331, 5003, False, {"num_batch_nodal_update": 3}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_float_ds_pairs_exact(oracle, name):
    from usap_b200 import api, native as nat
    n, e, weighted, extra = CASES[name]
    src, dst, w = _graph(n, e, weighted)
    params = {"num_batch_nodal_update": 2, "seed": 5, "init_mode": 1, "max_num_nodal_itr": 2, "persistent_ctas": 1,
              **extra}
    ctx = api.Context(0)
    ctx.load(src, dst, w, n)
    part, res = ctx.partition(nat.default_params(**params))
    ctx.close()
    params.pop("persistent_ctas")
    opart, ores, _ = oracle.OracleGraph(n, src, dst, w).partition(params)
    assert np.array_equal(part, opart)
    assert (res["B"], res["S_q"], res["sweeps"], res["nodal_moves"]) == (
        ores["B"], ores["S_q"], ores["sweeps"], ores["nodal_moves"])
