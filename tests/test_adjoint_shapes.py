"""qp3d_adjoint of one shape after another on one context (GPU): the state
buffers a context keeps belong to the shape they were made for, so the second
gradient equals, bit for bit, that of a context that has seen no other shape.
Pairs of equal padded volume: x and z exchanged (the planes that no step writes
lie elsewhere), a longer row in the same pitch and a thinner shell (a larger
record)."""
import numpy as np
import pytest

import qp3d
import synthetic

pytestmark = pytest.mark.gpu


def _shot(hx, hy, nz0, pml):
    return synthetic.small_case(hx=hx, hy=hy, nz0=nz0, pml=pml, nt=160, seed=71, fm=30.0)


@pytest.mark.parametrize("keep", [0, 1])
@pytest.mark.parametrize("first,second", [
    ((44, 20, 20, 6), (20, 20, 44, 6)),    # 56 x 32 x 32 and 32 x 32 x 56
    ((20, 24, 18, 6), (20, 50, 18, 6)),    # ny 36 and 62, both in rows of 64
    ((18, 20, 18, 8), (22, 24, 22, 6))])   # 34 x 36 x 34, shells of 8 and 6
def test_shapes_of_equal_volume_share_nothing(first, second, keep):
    a, b = _shot(*first), _shot(*second)
    rng = np.random.default_rng(71)
    with qp3d.Context(0) as fresh:
        fresh.tune(adj_keep_all=keep)
        obs = {}
        for s in (a, b):
            r = fresh.forward(s)
            obs[id(s)] = (r * (1 + 0.1 * rng.standard_normal(r.shape))).astype(np.float32)
        _, want = fresh.adjoint(b, obs[id(b)])
    with qp3d.Context(0) as ctx:
        ctx.tune(adj_keep_all=keep)
        ctx.adjoint(a, obs[id(a)])
        _, got = ctx.adjoint(b, obs[id(b)])
    for g, w in zip(got, want):
        assert np.any(w) and np.array_equal(g.view(np.uint64), w.view(np.uint64))
