"""qp3d_gradmax_noalloc at its documented limit in x (GPU): 65535 tiles of 32
rows in one column of y tiles.  The kernel's own tiles are of 24 rows, so their
number passes the 65535 of a launch grid's second dimension.  The maximum is
at the last updated cell along x, beside a spike in the outer band: a launch
that left out its last tile would miss it."""
import numpy as np
import pytest

import qp3d

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx", [65535 * 24 + 11, 65535 * 32 + 10])
def test_longest_accepted_grid(nx):
    ny, nz, ldy = 11, 11, 12
    u = torch.zeros((nz, nx, ldy), device="cuda")
    u[5, nx - 5, 5] = 1.0
    u[5, 7, 5] = 0.5
    c = np.zeros(36, np.float32)
    c[31] = 0.5
    out = torch.zeros(1, device="cuda")
    rc = qp3d.load().qp3d_gradmax_noalloc(u.data_ptr(), nx, ny, nz, ldy, 1.0, 1.0, 1.0,
                                          c.ctypes.data, out.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream, None, 0)
    assert rc == 0
    # 0.5 * (1 - 0), exact; the other spike gives 0.25
    assert float(out.item()) == 0.5
