"""A load that does not fit the device reports QP3D_ERR_NOMEM, and the next one
works (GPU): a record of 470 GB against 288."""
import numpy as np
import pytest

import qp3d
import synthetic
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def test_load_after_one_that_does_not_fit():
    shot = synthetic.small_case(hx=70, hy=70, nz0=18, pml=6, nt=12, seed=77)
    big = synthetic.small_case(hx=70, hy=70, nz0=18, pml=6, nt=12, seed=77)
    big.wavelet = np.zeros(24_000_000, np.float32)
    with qp3d.Context(0) as ctx:
        want = ctx.forward(shot)
        with pytest.raises(qp3d.QP3DError, match="-3"):
            ctx.load(big)
        assert bits_equal(ctx.forward(shot), want)
