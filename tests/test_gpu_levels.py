"""The pairwise affine levels and the parts of heavy buckets: that they run where
the plan says, with every number of levels the device can choose, against the
CPU oracle (bit-exact: integer work, tolerance zero)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SCRATCH = 1
MODULUS = {O.BN254: O.R_MOD, O.BLS12381: 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001}


@pytest.fixture(scope="module")
def M():
    from impeller_b200 import build
    build.build()
    from impeller_b200 import msm
    msm._lib.load()
    return msm


def expected_levels(entries, buckets, curve):
    """The engine's rule: buckets of 8 points and more on average, and enough
    slots left after the level."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    slots_min = sms * (10240 if curve == O.BLS12381 else 20480)
    k = 0
    while entries >= (8 * buckets << k) and (entries + (2 * (1 << k) - 1) * buckets) >> (k + 1) >= slots_min:
        k += 1
    return k


# curve, points, window, resident tables, digits and buckets of a plan
CASES = {
    "bn254_plain_c4": (O.BN254, (1 << 18) + 3, 4, False, 64, 32 * 8),
    "bn254_tables_c8": (O.BN254, (1 << 18) + 77, 8, True, 32, 128),
    "bn254_plain_c13": (O.BN254, 700_001, 13, False, 20, 10 * 4096),
    "bls12381_plain_c4": (O.BLS12381, (1 << 17) + 9, 4, False, 64, 64 * 8),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_levels_of_a_plan(M, name):
    curve, n, c, tables, digits, buckets = CASES[name]
    levels = expected_levels(n * digits, buckets, curve)
    assert levels >= 1
    pts, sc = O.gen_points(n, seed=51, curve=curve), O.gen_scalars(n, seed=51, stream=1, curve=curve)
    ctx, d_sc = M.MsmContext(pts, curve=curve), M.to_device(sc)
    if tables:
        ctx.precompute(c)
    full = ctx.launches(n, c)
    # the same plan without its levels, as where there is no room for them
    M._lib.check(M._lib.load().impeller_fail_scratch_step(SCRATCH), "impeller_fail_scratch_step")
    without = M.to_host(ctx.msm_device(d_sc, c=c))
    # one kernel a level, the one that decides how many run, and the accumulation of the last level's points
    assert full - ctx.launches(n, c) == levels + 2
    ctx.close()
    ctx = M.MsmContext(pts, curve=curve)
    if tables:
        ctx.precompute(c)
    got = M.to_host(ctx.msm_device(d_sc, c=c))
    assert ctx.launches(n, c) == full
    ctx.close()
    want = O.msm(pts, sc, curve=curve)
    assert np.array_equal(got, want) and np.array_equal(without, want)


# Zero scalars leave the device fewer levels than the plan has: all three, two
# (the last in the buffer of even levels), one, none; two and one on BLS12-381.
@pytest.mark.parametrize("curve,n,share,laid_out,chosen", [
    (O.BN254, 1 << 19, 1.0, 3, 3), (O.BN254, 1 << 19, 0.5, 3, 2), (O.BN254, 1 << 19, 0.25, 3, 1),
    (O.BN254, 1 << 19, 0.1, 3, 0), (O.BLS12381, 1 << 17, 1.0, 2, 2), (O.BLS12381, 1 << 17, 0.5, 2, 1)])
def test_levels_chosen_by_the_device(M, curve, n, share, laid_out, chosen):
    c, digits, buckets = 4, 64, (32 if curve == O.BN254 else 64) * 8
    assert expected_levels(n * digits, buckets, curve) == laid_out
    # 15 of 16 digits of a random scalar are not zero (1 % covers the spread and the top digits)
    for f in (0.99, 1.01):
        assert expected_levels(int(n * share * digits * 15 / 16 * f), buckets, curve) == chosen
    pts = M.to_host(M.gen_points_device(n, seed=52, curve=curve)).reshape(n, -1)
    sc = O.gen_scalars(n, seed=52, stream=2, curve=curve)
    sc[np.random.RandomState(5).permutation(n)[int(n * share):]] = 0
    ctx = M.MsmContext(pts, curve=curve)
    got = M.to_host(ctx.msm_device(M.to_device(sc), c=c))
    ctx.close()
    assert np.array_equal(got, O.msm(pts, sc, curve=curve))


# Every scalar one: a single bucket holds all points, in more parts than a warp
# has lanes (52 and 38 of them; 37 and more on BLS12-381).
@pytest.mark.parametrize("curve,n", [(O.BN254, 1 << 18), (O.BN254, 77777), (O.BLS12381, 1 << 18)])
def test_one_bucket_of_all_points(M, curve, n):
    one = (1 << 256) % MODULUS[curve]
    row = np.array([(one >> (32 * i)) & 0xFFFFFFFF for i in range(8)], np.uint32)
    pts = M.to_host(M.gen_points_device(n, seed=53, curve=curve)).reshape(n, -1)
    sc = np.repeat(row[None], n, axis=0)
    ctx = M.MsmContext(pts, curve=curve)
    got = M.to_host(ctx.msm_device(M.to_device(sc), c=16))
    ctx.close()
    assert np.array_equal(got, O.msm(pts, sc, curve=curve))
