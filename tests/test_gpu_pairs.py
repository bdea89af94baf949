"""MSMs whose buckets are added pairwise in affine form before the
accumulation, against the CPU oracle (bit-exact: integer work, tolerance
zero).

The levels run only on millions of entries, so the cases take small windows
over a few hundred thousand points: several levels, odd and even bucket
lengths, the last tile partly filled, unused slots, and the pairs the
additions treat apart -- equal points (a doubling), opposite points (the
identity) and identity inputs.
"""
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


P = {O.BN254: 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47,
     O.BLS12381: 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB}


def special_points(n, curve):
    """n points drawn from 8 points, their negatives and the identity, so that
    nearly every bucket holds equal, opposite and identity neighbours."""
    base = O.gen_points(8, seed=5, curve=curve)
    words = base.shape[1]
    neg = base.copy()
    for i in range(8):
        y = sum(int(v) << (32 * k) for k, v in enumerate(base[i, words // 2:]))
        y = P[curve] - y
        neg[i, words // 2:] = [(y >> (32 * k)) & 0xFFFFFFFF for k in range(words // 2)]
    pool = np.concatenate([base, neg, np.zeros((1, words), np.uint32)])
    return np.ascontiguousarray(pool[np.random.RandomState(3).randint(0, len(pool), n)])


# name: curve, points, window, resident table set, which points.  At 64, 32
# and 20 digits a scalar: 3 levels of plain windows, 1 level of one shared
# set, 2 levels with 8 bucket sets' worth of odd remainders.
CASES = {
    "bn254_plain_c4": ("bn254", (1 << 19) + 3, 4, False, "random"),
    "bn254_tables_c8": ("bn254", (1 << 18) + 77, 8, True, "random"),
    "bn254_plain_c13": ("bn254", 1_000_001, 13, False, "random"),
    "bn254_special_c4": ("bn254", (1 << 18) - 1, 4, False, "special"),
    "bls12381_plain_c4": ("bls12381", (1 << 17) + 9, 4, False, "random"),
    "bls12381_special_c8": ("bls12381", (1 << 17) + 1, 8, False, "special"),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_pairwise_levels_match_oracle(M, name):
    curve_name, n, c, tables, which = CASES[name]
    curve = {"bn254": O.BN254, "bls12381": O.BLS12381}[curve_name]
    pts = O.gen_points(n, seed=2, curve=curve) if which == "random" else special_points(n, curve)
    sc = O.gen_scalars(n, seed=2, stream=9, curve=curve)
    ctx = M.MsmContext(pts, curve=curve)
    launches = ctx.launches(n, c)
    if tables:
        ctx.precompute(c)
    got = M.to_host(ctx.msm_device(M.to_device(sc), c=c))
    # the same context and window on few points runs no levels: fewer launches
    assert launches > ctx.launches(1000, c)
    ctx.close()
    assert np.array_equal(got, O.msm(pts, sc, curve=curve))


def test_skewed_scalars_choose_levels_on_the_device(M):
    """Scalars of one small digit: the plan lays out levels, the entries are
    too few for them, and the accumulation takes the sorted entries."""
    n = 1 << 19
    pts = M.gen_points_device(n, seed=4)
    ctx = M.MsmContext(pts)
    sc = np.zeros((n, 8), np.uint32)
    one = O.gen_scalars(1, seed=1, stream=1)  # any scalar: 500 copies, the rest zero
    sc[::1049] = one
    got = M.to_host(ctx.msm_device(M.to_device(sc), c=4))
    want = O.msm(M.to_host(pts).reshape(n, -1), sc)
    ctx.close()
    assert np.array_equal(got, want)
