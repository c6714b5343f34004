"""A batch of many small shots, each with a PML width and profiles of its own
(GPU): every shot takes its own layer table, work items and tensor maps, on the
first call and on one with other sizes through the same buffers."""
import pytest

import qp3d
import synthetic as S
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def _shots(n, seed):
    return [S.small_case(hx=12 + (7 * i + seed) % 23, hy=12 + (11 * i + seed) % 29,
                         nz0=11 + (5 * i) % 13, pml=5 + (i + seed) % 9, nt=24, seed=seed + i)
            for i in range(n)]


def test_many_shots_of_two_calls():
    with qp3d.Context(0) as ctx, qp3d.Context(0) as one:
        for n, seed in ((40, 3), (25, 90)):
            shots = _shots(n, seed)
            for s, r in zip(shots, ctx.batch(shots)):
                assert bits_equal(r, one.forward(s))
