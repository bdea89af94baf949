"""Scratch of resident contexts and batches when memory is short.  The failures
are made on the host (the step returns an error instead of running); results are
compared with the CPU oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SCRATCH, UPLOAD = 1, 2


@pytest.fixture(scope="module")
def M():
    from impeller_b200 import build
    build.build()
    from impeller_b200 import msm
    msm._lib.load()
    return msm


def fail_next(M, step):
    M._lib.check(M._lib.load().impeller_fail_scratch_step(step), "impeller_fail_scratch_step")


def test_run_after_a_failed_upload_of_the_tables(M):
    # the tables' memory is not taken for uploaded ones by the next call
    n = 3000
    pts, sc = O.gen_points(n, seed=21), O.gen_scalars(n, seed=21, stream=1)
    d_sc, ctx = M.to_device(sc), M.MsmContext(pts)
    fail_next(M, UPLOAD)
    with pytest.raises(M._lib.ImpellerError, match="upload of a plan's tables"):
        ctx.msm_device(d_sc)
    got = M.to_host(ctx.msm_device(d_sc))
    ctx.close()
    assert np.array_equal(got, O.msm(pts, sc))


# 2^18 + 5 points at 64 digits lay out two levels of pairwise additions
N, C = (1 << 18) + 5, 4


@pytest.fixture(scope="module")
def leveled():
    pts, sc = O.gen_points(N, seed=22), O.gen_scalars(N, seed=22, stream=1)
    small = O.gen_scalars(900, seed=22, stream=2)
    return pts, sc, O.msm(pts, sc), small, O.msm(pts[:900], small)


def test_plan_without_levels_takes_over_until_the_scratch_grows(M, leveled):
    pts, sc, want, small, want_small = leveled
    d_sc, d_small, ctx = M.to_device(sc), M.to_device(small), M.MsmContext(pts)
    full = ctx.launches(N, C)
    assert np.array_equal(M.to_host(ctx.msm_device(d_small, c=8)), want_small)  # some scratch is there
    fail_next(M, SCRATCH)
    assert np.array_equal(M.to_host(ctx.msm_device(d_sc, c=C)), want)
    reduced = ctx.launches(N, C)
    assert reduced < full
    # other sizes leave it in place, and it them
    assert np.array_equal(M.to_host(ctx.msm_device(d_small, c=8)), want_small)
    assert ctx.launches(N, C) == reduced
    # a plan that needs more scratch: room again, and the levels are back
    assert np.array_equal(M.to_host(ctx.msm_device(d_sc, c=3)), want)
    assert ctx.launches(N, C) == full
    assert np.array_equal(M.to_host(ctx.msm_device(d_sc, c=C)), want)
    ctx.close()


def test_levels_take_a_quarter_of_the_free_memory_at_most(M, leveled):
    pts, sc, want, small, want_small = leveled
    ctx, room = M.MsmContext(pts), M.MsmContext(pts)
    full = room.launches(N, C)
    # the levels take 0.75 points of 64 bytes a digit: 0.8 GB
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (5 << 29), dtype=torch.uint8, device="cuda")
    d_sc = M.to_device(sc)
    assert np.array_equal(M.to_host(ctx.msm_device(d_sc, c=C)), want)
    assert ctx.launches(N, C) < full
    b = ctx.batch([N, 900], windows=[C, 8], graph=False)
    got = M.to_host(b.run([d_sc, M.to_device(small)]))
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want_small)
    less = b.launches
    b.close()
    del hold
    torch.cuda.empty_cache()
    b = ctx.batch([N, 900], windows=[C, 8], graph=False)
    assert b.launches > less
    b.close()
    assert np.array_equal(M.to_host(room.msm_device(d_sc, c=C)), want)
    assert room.launches(N, C) == full
    room.close()
    ctx.close()


def test_batch_without_room_for_levels(M, leveled):
    pts, sc, want, small, want_small = leveled
    ctx = M.MsmContext(pts)
    full = ctx.batch([N, 900], windows=[C, 8])
    fail_next(M, SCRATCH)
    b = ctx.batch([N, 900], windows=[C, 8])
    assert b.launches < full.launches
    for batch in (b, full):
        got = M.to_host(batch.run([M.to_device(sc), M.to_device(small)]))
        assert np.array_equal(got[0], want) and np.array_equal(got[1], want_small)
        batch.close()
    ctx.close()



def test_whole_scalars_where_the_images_find_no_room(M):
    n = 5000
    pts, sc = O.gen_points(n, seed=23), O.gen_scalars(n, seed=23, stream=1)
    want = O.msm(pts, sc)
    ctx = M.MsmContext(pts)
    full, d_sc = ctx.launches(n, 13), M.to_device(sc)
    fail_next(M, SCRATCH)
    for c in (13, 0):
        assert np.array_equal(M.to_host(ctx.msm_device(d_sc, c=c)), want)
    assert ctx.launches(n, 13) == full - 1  # no kernel for the images
    fail_next(M, SCRATCH)
    b = ctx.batch([n, 777, 1])
    for _ in range(2):
        got = M.to_host(b.run([d_sc, d_sc[:777], d_sc[:1]]))
    for i, k in enumerate((n, 777, 1)):
        assert np.array_equal(got[i], O.msm(pts[:k], sc[:k]))
    b.close()
    ctx.close()


def test_last_run_of_a_drop_in_call_with_fewer_msms(M):
    # five MSMs a run sort entry by entry, the four that there are in two
    # levels, which takes more scratch: all within the buffer
    n, guard = 1_000_000, 1 << 20
    op = M.MSM(M.MsmConfig(window_size=18, target_window=15, batch_per_run=5))
    size = op.get_buffer_size(n)[0]
    buf, keep = M.alloc_gpu_buffer(size + guard)
    keep[size:] = 0xA5
    pts = M.to_host(M.gen_points_device(n, seed=24)).reshape(n, -1)
    sc = [M.to_host(M.gen_scalars_device(n, seed=24, stream_id=i)).reshape(n, 8) for i in (1, 2)]
    got = op.run([pts], [sc[0], sc[1], sc[1], sc[0]], [buf])
    assert bool((keep[size:] == 0xA5).all())
    want = [O.msm(pts, s) for s in sc]
    for g, k in zip(got, (0, 1, 1, 0)):
        assert np.array_equal(g, want[k])


def test_server_budget_counts_freed_scratch(M):
    # scratch that a closed context left in the pool is free for a server
    n = 1 << 21
    keep = M.MsmContext(O.gen_points(100, seed=25))  # the pool lives
    ctx = M.MsmContext(M.gen_points_device(n, seed=25))
    sc = M.gen_scalars_device(n, seed=25)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.msm_device(sc)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    assert used > 1 << 28
    ctx.close()
    srv = M.MsmServer(keep, max_batch=2, max_inflight=1)
    budget = srv.stats()["budget_bytes"]
    srv.close()
    keep.close()
    assert budget > free - (1 << 30) - used // 4
