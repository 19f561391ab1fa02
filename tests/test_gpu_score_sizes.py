"""Scores, description length and TSV ingest at the sizes where their kernels
change path or have a remainder: the block count up to which a CTA counts the
whole matrix, the largest table counted in shared memory, vertices and edges
around a CTA's share, text lengths around a thread's 16 bytes.  Everything is
compared exactly (integer sums of identically rounded terms).
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()


@pytest.mark.parametrize("b,e", [(1, 1), (2, 4095), (19, 4097), (103, 30001), (104, 30001), (105, 30001), (333, 8192),
                                 (1024, 50000)])
@pytest.mark.parametrize("weighted", [False, True])
def test_entropy_static_sizes(b, e, weighted):
    import torch
    from usap_b200 import api, native
    rng = np.random.default_rng(b + e)
    n = 2000
    src = np.sort(rng.integers(0, n, e)).astype(np.int32)
    dst = rng.integers(0, n, e).astype(np.int32)
    w = rng.integers(1, 6, e).astype(np.int32) if weighted else None
    part = np.where(rng.random(n) < 0.5, 0, rng.integers(0, b, n)).astype(np.int32)
    ctx = api.Context(0)
    ctx.load(src, dst, w, n)
    want = ctx.op_entropy(part, b)
    ctx.close()
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    d = [_dev(x) for x in (src, dst, part)]
    dw = _dev(w) if weighted else None
    native.check(native.lib().usap_entropy_static(
        C.c_void_p(d[0].data_ptr()), C.c_void_p(d[1].data_ptr()), C.c_void_p(dw.data_ptr()) if weighted else None, e, n,
        C.c_void_p(d[2].data_ptr()), b, C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert int(out.item()) == want


@pytest.mark.parametrize("n,b1,b2", [(2, 1, 1), (4095, 1, 8192), (4096, 8192, 1), (4097, 64, 128), (30011, 64, 129),
                                     (30011, 2, 4096), (30011, 2049, 4)])
def test_evaluate_sizes(n, b1, b2):
    from usap_b200 import api
    rng = np.random.default_rng(n + b1)
    truth = rng.integers(0, b1, n).astype(np.int32)
    given = rng.integers(0, b2, n).astype(np.int32)
    truth[0], given[0] = b1 - 1, b2 - 1
    if n > 100:
        truth[rng.random(n) < 0.1] = -1
        truth[0] = b1 - 1
    t, g = _dev(truth), _dev(given)
    got, want = api.evaluate_device(t.data_ptr(), g.data_ptr(), n), api.evaluate(truth, given)
    assert got.keys() == want.keys()
    for k in want:
        assert got[k] == want[k] or (np.isnan(got[k]) and np.isnan(want[k])), k


@pytest.mark.parametrize("bad", [(0, -1), (-2, 0), (2**31 - 1, 0), (0, 2**31 - 1)])
def test_evaluate_refuses(bad):
    from usap_b200 import api, native
    truth = np.zeros(5000, np.int32)
    given = np.zeros(5000, np.int32)
    truth[4321], given[4321] = bad
    t, g = _dev(truth), _dev(given)
    with pytest.raises(native.UsapError):
        api.evaluate_device(t.data_ptr(), g.data_ptr(), 5000)


@pytest.mark.parametrize("edges,pad", [(1, 0), (1, 4), (3, 1), (1023, 0), (1024, 7), (5000, 9)])
@pytest.mark.parametrize("last", ["\n", ""])
def test_tsv_sizes(edges, pad, last):
    from usap_b200 import api
    rng = np.random.default_rng(edges + pad)
    n = 700
    src, dst = rng.integers(0, n, edges), rng.integers(0, n, edges)
    src[0] = n - 1
    # zeros in front shift where the lines end within a thread's bytes
    lines = ["%0*d\t%d\t1" % (1 + (pad + i) % 5, a + 1, b + 1) for i, (a, b) in enumerate(zip(src, dst))]
    text = ("\n".join(lines) + last).encode()
    one, two = api.Context(0), api.Context(0)
    one.load_tsv(text)
    two.load(src.astype(np.int32), dst.astype(np.int32), None, n)
    got, want = one.adjacency(), two.adjacency()
    assert one.n == n and one.e == edges
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    one.close()
    two.close()
