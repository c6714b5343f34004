"""Segments of deferred cells that overflow (GPU; a hook leaves them room for
one cell): the steps are re-run, shots of a batch by the queue of its
resolution, and every result equals, bit for bit, that of a run with room.  The
re-run of a gradient's checkpointed forward records its decisions again."""
import numpy as np
import pytest

import qp3d
import synthetic as S
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [1, 0])
@pytest.mark.parametrize("graph,candidate", [(1, 0), (0, 3)])
def test_batch(graph, candidate, arith):
    shots = [S.small_case(hx=22, hy=26, nz0=18, pml=8, nt=50, seed=81),
             S.small_case(hx=47, hy=33, nz0=24, pml=6, nt=44, seed=82),
             S.small_case(hx=15, hy=70, nz0=30, pml=10, nt=50, seed=83)]
    out, redo = [], []
    for cap in (0, 1):
        with qp3d.Context(0) as ctx:
            ctx.tune(arith=arith, batch_tune=0, batch_candidate=candidate, batch_graph=graph,
                     test_defer_cap=cap)
            out.append(ctx.batch(shots))
            redo.append(ctx.batch_stats()["redo_steps"])
    assert redo[1] > redo[0] + len(shots)
    for a, b in zip(*out):
        assert np.any(a) and bits_equal(a, b)


@pytest.mark.parametrize("keep", [0, 1])
def test_gradient(keep):
    shot = S.small_case(hx=40, hy=30, nz0=26, pml=8, nt=90, seed=84, fm=30.0)
    out = []
    for cap in (0, 1):
        with qp3d.Context(0) as ctx:
            d_obs = ctx.forward(shot) * np.float32(1.1)
            ctx.tune(adj_keep_all=keep, test_defer_cap=cap)
            out.append(ctx.adjoint(shot, d_obs)[1])
            redo = ctx.stats()[0]
    assert redo.sum() > 3
    for a, b in zip(*out):
        assert np.any(a) and np.array_equal(a.view(np.uint64), b.view(np.uint64))
