"""The kernels that small and mid-size MSMs take, at the edges of their ranges,
against the CPU oracle (bit-exact: integer work, tolerance zero)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def M():
    from impeller_b200 import build
    build.build()
    from impeller_b200 import msm
    msm._lib.load()
    return msm


def check(M, curve, n, c, tables, scalars=None, seed=6):
    pts = O.gen_points(n, seed=seed, curve=curve)
    sc = O.gen_scalars(n, seed=seed, stream=3, curve=curve) if scalars is None else scalars
    ctx = M.MsmContext(pts, curve=curve)
    if tables:
        ctx.precompute(c)
    first = M.to_host(ctx.msm_device(M.to_device(sc), c=c))
    again = M.to_host(ctx.msm_device(M.to_device(sc), c=c))  # the kept table image
    ctx.close()
    want = O.msm(pts, sc, curve=curve)
    assert np.array_equal(first, want) and np.array_equal(again, want)


# One-block sort: 96 K digits (32 a scalar at window 8) and one scalar more,
# one and two rounds of the block, one scalar.
@pytest.mark.parametrize("n", [1, 1024, 1025, 3072, 3073])
@pytest.mark.parametrize("tables", [False, True])
def test_one_block_sort_edges(M, n, tables):
    check(M, O.BN254, n, 8, tables)


# its limit of 8192 buckets: 13 sets of 2^9, then 12 of 2^10
@pytest.mark.parametrize("c", [10, 11])
def test_one_block_sort_buckets(M, c):
    check(M, O.BN254, 700, c, False)


# Bucket reduction by lane pairs up to 2^17 buckets (window 18 with one shared
# set), one bucket to eight per pair, and past it; the windows' partials make
# tree groups of 1, 2, 8, 16, 17 to 32 and several levels.
@pytest.mark.parametrize("c", [5, 6, 7, 9, 11, 13, 14, 15, 16, 18, 19])
def test_reduction_by_buckets(M, c):
    check(M, O.BN254, 1500, c, True)


@pytest.mark.parametrize("c", [6, 12, 18])
def test_reduction_by_buckets_bls12381(M, c):
    check(M, O.BLS12381, 600, c, True)


# One heavy bucket over tens of thousands of slices: its pieces merge in parts
# by several blocks, and the parts' sums (more than a warp's worth) by the last.
@pytest.mark.parametrize("n", [1 << 18, 77777])
def test_heavy_bucket_in_parts(M, n):
    one = O.gen_scalars(1, seed=2, stream=2)
    check(M, O.BN254, n, 16, False, scalars=np.repeat(one, n, axis=0))


# Equal and opposite points in one bucket: the lane pairs' additions meet
# doublings and the identity.
def test_equal_and_opposite_buckets(M):
    n = 640
    pts = O.gen_points(1, seed=9)
    pts = np.repeat(pts, n, axis=0)
    sc = O.gen_scalars(n // 2, seed=9, stream=5)
    r = O.R_MOD
    neg = np.zeros_like(sc)
    for i, row in enumerate(sc):
        v = (r - sum(int(x) << (32 * k) for k, x in enumerate(row))) % r
        neg[i] = [(v >> (32 * k)) & 0xFFFFFFFF for k in range(8)]
    for scalars in (np.concatenate([sc, neg]), np.repeat(sc[:1], n, axis=0)):
        for c in (8, 13):
            ctx = M.MsmContext(pts)
            got = M.to_host(ctx.msm_device(M.to_device(scalars), c=c))
            ctx.close()
            assert np.array_equal(got, O.msm(pts, scalars))


# A batch whose windows differ by 2^12 in size, with and without a graph.
@pytest.mark.parametrize("graph", [False, True])
def test_batch_of_uneven_windows(M, graph):
    sizes, windows = [3000, 70, 1, 20000, 999], [16, 8, 4, 16, 13]
    pts = O.gen_points(max(sizes), seed=12)
    ctx = M.MsmContext(pts)
    scs = [O.gen_scalars(s, seed=12, stream=i) for i, s in enumerate(sizes)]
    b = ctx.batch(sizes, windows=windows, graph=graph)
    for _ in range(2):
        got = M.to_host(b.run([M.to_device(s) for s in scs]))
        torch.cuda.synchronize()
    for i, s in enumerate(scs):
        assert np.array_equal(got[i], O.msm(pts[:sizes[i]], s))
    b.close()
    ctx.close()
