"""The packing of a narrow last y tile, on both sides of its rule, bit for bit
against the oracle (GPU): four quads, the last one whole or of one cell (eight
rows a warp), five (four rows), two (sixteen) and three.  A last tile holds at
least six cells."""
import pytest

import synthetic
from test_step_forms import _check, sctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [1, 0])
@pytest.mark.parametrize("ny,hx", [(48, 20), (45, 31), (49, 24), (40, 27), (38, 43), (41, 22)])
def test_last_y_tile(sctx, ny, hx, arith):  # noqa: F811
    pml = 6
    shot = synthetic.small_case(hx=hx, hy=ny - 2 * pml, nz0=15, pml=pml, nt=8, seed=65)
    assert shot.ny == ny
    _check(sctx, shot, *synthetic.random_state(shot, seed=65), arith)
