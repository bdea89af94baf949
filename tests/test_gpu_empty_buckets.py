"""MSMs that leave most buckets or whole windows empty: zero scalars, ones, small
values and few points, against the CPU oracle (bit-exact: integer work, tolerance
zero).  The lane pairs of the tails leave early where all of them add the
identity, and must not where one does not."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MODULUS = {O.BN254: O.R_MOD, O.BLS12381: O.R_BLS}


@pytest.fixture(scope="module")
def M():
    from impeller_b200 import build
    build.build()
    from impeller_b200 import msm
    msm._lib.load()
    return msm


def mont(values, curve):
    r = MODULUS[curve]
    return np.array([[((int(v) << 256) % r >> (32 * k)) & 0xFFFFFFFF for k in range(8)] for v in values], np.uint32)


def columns(n, curve):
    rng = np.random.RandomState(n)
    last = np.zeros(n, np.int64)
    last[-1] = 1
    r = MODULUS[curve]
    return {"zeros": np.zeros(n, np.int64), "ones": np.ones(n, np.int64), "last": last,
            "bytes": rng.randint(0, 256, n), "signs": [(0, 1, r - 1)[i] for i in rng.randint(0, 3, n)],
            "top": [1 << 250 if i % 97 == 0 else 0 for i in range(n)]}


@pytest.mark.parametrize("curve", [O.BN254, O.BLS12381])
@pytest.mark.parametrize("n,c,tables", [(1, 8, False), (33, 8, True), (700, 13, False), (700, 16, True), (2000, 19, True)])
def test_empty_buckets_and_windows(M, curve, n, c, tables):
    pts = O.gen_points(n, seed=61, curve=curve)
    ctx = M.MsmContext(pts, curve=curve)
    if tables:
        ctx.precompute(c)
    cols = {k: mont(v, curve) for k, v in columns(n, curve).items()}
    want = {k: O.msm(pts, v, curve=curve) for k, v in cols.items()}
    for k, v in cols.items():
        assert np.array_equal(M.to_host(ctx.msm_device(M.to_device(v), c=c)), want[k]), k
    names = sorted(cols)
    b = ctx.batch([n] * len(names), windows=[c] * len(names))
    got = M.to_host(b.run([M.to_device(cols[k]) for k in names]))
    for i, k in enumerate(names):
        assert np.array_equal(got[i], want[k]), k
    b.close()
    ctx.close()
