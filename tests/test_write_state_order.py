"""Steps that are enqueued right after qp3d_shot_write_state see the whole state
(GPU): its copies go to the steps' own stream.  The second run waits for the
device in between."""
import pytest

import qp3d
import synthetic
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def test_steps_after_a_written_state():
    torch = pytest.importorskip("torch")
    shot = synthetic.small_case(hx=90, hy=70, nz0=80, pml=10, nt=3, seed=74)
    state = synthetic.random_state(shot, seed=74)
    out = []
    with qp3d.Context(0) as ctx:
        for wait in (False, True):
            ctx.load(shot)
            ctx.write_state(0, *state)
            if wait:
                torch.cuda.synchronize()
            ctx.advance(shot.nt)
            out.append((ctx.record(),) + tuple(ctx.read_state()))
    for a, b in zip(*out):
        assert bits_equal(a, b)
