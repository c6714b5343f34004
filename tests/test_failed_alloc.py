"""An allocation that fails in a re-plan or a load (GPU; made to fail on the
host by a hook) leaves no shot loaded: later calls return QP3D_ERR_STATE instead
of stepping a shot whose lists are gone, and the next load works."""
import numpy as np
import pytest

import qp3d
import synthetic
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.fixture
def fctx():
    with qp3d.Context(0) as c:
        yield c


def _not_loaded(ctx):
    for call in (lambda: ctx.advance(1), ctx.reset, lambda: ctx.record(0, 1)):
        with pytest.raises(qp3d.QP3DError, match="-5"):
            call()


def _works(ctx, shot, want):
    ctx.tune(test_fail_alloc=0)
    ctx.load(shot)
    ctx.advance(shot.nt)
    assert bits_equal(ctx.record(), want)


def test_replan_of_a_loaded_shot(fctx):
    shot = synthetic.small_case(nt=12, seed=75)
    with qp3d.Context(0) as c:          # fctx has no larger lists from before
        want = c.forward(shot)
    fctx.tune(chunks=1)
    fctx.load(shot)
    fctx.advance(4)
    fctx.tune(test_fail_alloc=1)
    with pytest.raises(qp3d.QP3DError, match="-3"):
        fctx.tune(chunks=6)             # a segment for each of six times as many columns
    _not_loaded(fctx)
    _works(fctx, shot, want)


@pytest.mark.parametrize("nsrc", [4, 100])   # fused into the steps, and on their own
def test_reload_with_more_sources(fctx, nsrc):
    shot = synthetic.small_case(nt=12, seed=76)
    want = fctx.forward(shot)
    more = synthetic.small_case(nt=12, seed=76)
    v = more.src.reshape(shot.nz, shot.nx, shot.ny)
    v[12:22, 12:22, 15] = 1.0 if nsrc == 100 else 0.0
    v[12, 12, 15:19] = 1.0
    fctx.load(shot)
    fctx.tune(test_fail_alloc=1)
    with pytest.raises(qp3d.QP3DError, match="-3"):
        fctx.load(more)
    _not_loaded(fctx)
    _works(fctx, shot, want)
