"""Transforms at the edges of the pass plans: the cluster of blocks up to 2^11,
two even passes up to 2^20, three passes above, with a twiddle table and with
recomputed twiddles, on straight and wrapping views.  Bit-exact against the
CPU oracle (integer work, tolerance zero); past 2^20 the two kinds against
each other and the table's through an inverse round trip."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FIELDS = {"bn254_fr": O.FR, "bls12381_fr": O.BLS_FR}


@pytest.fixture(scope="module")
def N():
    from impeller_b200 import build
    build.build()
    from impeller_b200 import ntt
    ntt._lib.load()
    return ntt


def field_id(N, field):
    return {O.FR: N.BN254_FR, O.BLS_FR: N.BLS12381_FR}[field]


def scalars(log_n, field, seed):
    curve = O.BLS12381 if field == O.BLS_FR else O.BN254
    return O.gen_scalars(1 << log_n, seed=seed, stream=4, curve=curve)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy().view(np.uint32).reshape(-1, 8)


def unit(log_n, field):
    return O.mont_limbs(O.root_of_unity(log_n, field), field)


def transform(N, field, log_n, w, d, recompute, **view):
    f = field_id(N, field)
    if recompute:
        g = N.GenPqOmegas(f)
        pq, om = np.zeros((g.get_pq_len(log_n), 8), np.uint32), np.zeros((32, 8), np.uint32)
        g.get_fn()(pq, om, 1 << log_n, w)
        N.RecomputeNtt(f).get_fn()(d, dev(pq), dev(om), **view)
    else:
        tw = np.zeros((max(1, (1 << log_n) // 2), 8), np.uint32)
        N.SsipPrecompute(f).get_fn()(tw, w)
        N.SsipNtt(f).get_fn()(d, dev(tw), **view)


@pytest.mark.parametrize("name", sorted(FIELDS))
@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("log_n", [7, 9, 10, 11, 12, 14, 17, 18, 19])
def test_pass_plans_match_oracle(N, log_n, recompute, name):
    field = FIELDS[name]
    x = scalars(log_n, field, log_n)
    w = unit(log_n, field)
    d = dev(x)
    transform(N, field, log_n, w, d, recompute)
    assert np.array_equal(host(d), O.ntt(x, w, field))


@pytest.mark.parametrize("log_n", [9, 11, 14])
def test_wrapping_views(N, log_n):
    n, whole, off = 1 << log_n, (1 << log_n) + 123, 100 + (1 << (log_n - 1))
    big = scalars(log_n + 1, O.FR, 3)[:whole]
    w = unit(log_n, O.FR)
    idx = (off + np.arange(n)) % whole
    want = big.copy()
    want[idx] = O.ntt(big[idx], w)
    for recompute in (False, True):
        d = dev(big)
        transform(N, O.FR, log_n, w, d, recompute, offset=off, whole_len=whole, length=n)
        assert np.array_equal(host(d), want)


@pytest.mark.parametrize("log_n", [21, 22])
def test_three_passes(N, log_n):
    x = scalars(log_n, O.FR, 5)
    w = unit(log_n, O.FR)
    a, b = dev(x), dev(x)
    transform(N, O.FR, log_n, w, a, False)
    transform(N, O.FR, log_n, w, b, True)
    got = host(a)
    assert np.array_equal(got, host(b))
    # the transform with w^-1 gives n x
    inverse = O.mont_limbs(pow(O.root_of_unity(log_n, O.FR), -1, O.R_MOD), O.FR)
    transform(N, O.FR, log_n, inverse, a, False)
    back = host(a)
    n = 1 << log_n
    for i in (0, 1, 2, 3, n // 2, n - 1, 12345, 999983):
        v = sum(int(t) << (32 * k) for k, t in enumerate(x[i]))
        assert sum(int(t) << (32 * k) for k, t in enumerate(back[i])) == v * n % O.R_MOD
