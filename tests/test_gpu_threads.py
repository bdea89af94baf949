"""Two host threads on one card, one in the drop-in MSM and one building window
tables: they share the card's streams.  Bit-exact, tolerance zero."""
import threading

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


def test_msm_beside_a_table_build(M):
    n, m = 60000, 40000
    pts, sc = O.gen_points(n, seed=71), O.gen_scalars(n, seed=71, stream=1)
    want = O.msm(pts, sc)
    op = M.MSM(M.MsmConfig())
    buf, keep = M.alloc_gpu_buffer(op.get_buffer_size(n)[0])
    cfg = M.MsmConfig(window_size=13, target_window=4)
    build = M.MSMPrecompute(cfg).get_fn()

    def tables():
        t = [pts[:m].copy()] + [np.zeros((m, 16), np.uint32) for _ in range(cfg.get_precompute() - 1)]
        build(t, m, 1)
        return np.stack(t)

    alone = tables()
    sums, built, errors = [], [], []

    def loop(f, out, times):
        try:
            for _ in range(times):
                out.append(f())
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(lambda: op.run([pts], [sc], [buf])[0], sums, 40)),
               threading.Thread(target=loop, args=(tables, built, 15))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and len(sums) == 40 and len(built) == 15
    assert all(np.array_equal(s, want) for s in sums)
    assert all(np.array_equal(t, alone) for t in built)
    # the tables give the same MSM
    op2 = M.MSM(M.MsmConfig(window_size=13, target_window=4))
    buf2, keep2 = M.alloc_gpu_buffer(op2.get_buffer_size(m)[0])
    assert np.array_equal(op2.run(list(alone), [sc[:m]], [buf2])[0], O.msm(pts[:m], sc[:m]))
