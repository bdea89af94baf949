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


def test_contexts_closed_beside_a_batch_graph_being_made(M):
    # closing a context and adding tables wait for the device, which fails, and
    # ends the capture, while a graph is captured on it
    sizes = [3000, 70, 1500]
    pts = O.gen_points(max(sizes), seed=72)
    scs = [O.gen_scalars(n, seed=72, stream=i) for i, n in enumerate(sizes)]
    want = [O.msm(pts[:n], s) for n, s in zip(sizes, scs)]
    d_pts, d_scs = M.to_device(pts), [M.to_device(s) for s in scs]
    errors, wrong = [], []

    def batches():
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                ctx = M.MsmContext(d_pts)
                for _ in range(60):
                    b = ctx.batch(sizes, graph=True)
                    got = M.to_host(b.run(d_scs, stream=st))
                    wrong.extend(i for i in range(len(sizes)) if not np.array_equal(got[i], want[i]))
                    b.close()
                ctx.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def contexts():
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for k in range(60):
                    ctx = M.MsmContext(d_pts)
                    if k % 3 == 0:
                        ctx.precompute(8)
                    if not np.array_equal(M.to_host(ctx.msm_device(d_scs[0], stream=st)), want[0]):
                        wrong.append(k)
                    ctx.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=f) for f in (batches, contexts, contexts)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and not wrong
