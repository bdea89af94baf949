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
