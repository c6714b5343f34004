"""The first gradient of a context equals the next ones bit for bit (GPU): the
kept wavefields and decisions are zeroed, once, on the steps' own stream, so a
forward pass that starts right after finds them zero and is not zeroed itself.
Kept wavefields that take long to zero beside a step: 852 MB (every u^k) or
85 MB and 80 MB of decisions, against microseconds."""
import numpy as np
import pytest

import qp3d
import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", [0, 1])
def test_first_gradient_equals_the_second(keep):
    nt = 300 if keep else 900
    shot = synthetic.small_case(hx=70, hy=50, nz0=70, pml=8, nt=nt, seed=72, fm=30.0)
    with qp3d.Context(0) as ctx:
        d_obs = ctx.forward(shot) * np.float32(1.1)
    with qp3d.Context(0) as ctx:
        ctx.tune(adj_keep_all=keep)
        _, first = ctx.adjoint(shot, d_obs)
        _, again = ctx.adjoint(shot, d_obs)
    for a, b in zip(first, again):
        assert np.any(a) and np.array_equal(a.view(np.uint64), b.view(np.uint64))
