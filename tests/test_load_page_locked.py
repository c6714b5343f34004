"""qp3d_shot_load from page-locked volumes has read them when it returns (GPU):
a caller that writes its next model into the same buffers right after the call
must not change the loaded one.  The volumes are large, so that their copies
take longer than the rest of a load; the second load of a geometry allocates
nothing, and so waits for nothing on the way."""
import numpy as np
import pytest

import qp3d
import synthetic
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def test_buffers_may_be_overwritten_after_the_load():
    n, nt = 320, 3
    small = synthetic.small_case(hx=20, hy=20, nz0=20, pml=8, nt=nt, seed=73)
    held = [qp3d.PinnedArray((n * n * n,)) for _ in range(3)]
    vp, eps, delta = (h.array for h in held)
    shot = qp3d.Shot(n, n, n, 8, 8, 10.0, 10.0, 10.0, 5e-4, vp, eps, delta, None, small.wavelet,
                     small.prof, small.c, small.c2)
    assert shot.vp.ctypes.data == vp.ctypes.data    # the page-locked memory itself
    u = np.zeros((n, n, n), np.float32)
    u[n // 2, n // 2, ::8] = 1.0

    def model():
        vp[:] = 3000.0
        eps[:] = 0.2
        delta[:] = 0.1

    def run(ctx):
        ctx.write_state(0, u_cur=u)
        ctx.advance(nt)
        return ctx.read_state()[1]

    with qp3d.Context(0) as ctx:
        model()
        ctx.load(shot)
        ctx.sync()
        want = run(ctx)
        ctx.load(shot)
        for a in (delta, eps, vp):      # the last copied first
            a[:] = 0.0
        got = run(ctx)
    assert np.any(want[:n * n * (n // 2 - 1)]) and bits_equal(got, want)
    for h in held:
        h.free()
