"""qp3d_gradmax_noalloc's two kernels (through L1 up to 24 Mi pitched cells, from
staged planes above) at the sizes where they can go wrong: the smallest grid,
remainders of the 32-cell tiles, pitches with garbage in the padding, a row
that ends a block, and a volume on either side of the line.  Reference: the
same differences in FP64 (plain torch); tolerance: seven roundings of the
largest sum of magnitudes a derivative is made of."""
import numpy as np
import pytest

import qp3d

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W = [0.833, -0.2381, 0.059, -0.0099, 0.00079]


@pytest.mark.parametrize("nx,ny,nz,ldy", [(11, 11, 11, 12), (12, 43, 33, 64), (27, 36, 38, 36),
                                          (26, 37, 16, 40), (75, 133, 29, 160),
                                          (300, 290, 262, 320), (300, 300, 273, 320)])
def test_maximum_equals_fp64(nx, ny, nz, ldy):
    g = torch.Generator(device="cuda").manual_seed(nx * ny)
    u = torch.full((nz, nx, ldy), float("nan"), device="cuda")
    u[:, :, :ny] = torch.randn((nz, nx, ny), generator=g, device="cuda")
    c = np.zeros(36, np.float32)
    c[31:36] = W
    out = torch.zeros(1, device="cuda")
    rc = qp3d.load().qp3d_gradmax_noalloc(u.data_ptr(), nx, ny, nz, ldy, 10.0, 12.5, 8.0,
                                          c.ctypes.data, out.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream, None, 0)
    assert rc == 0
    v, want, bound = u[:, :, :ny].double(), 0.0, 0.0
    box = (slice(5, -5),) * 3
    for ax, h in ((1, 10.0), (2, 12.5), (0, 8.0)):
        t = torch.zeros_like(v[box])
        for m in range(5):
            a, b, n = list(box), list(box), v.shape[ax]
            a[ax], b[ax] = slice(6 + m, n - 4 + m), slice(4 - m, n - 6 - m)
            t += (v[tuple(a)] - v[tuple(b)]) * (float(c[31 + m]) / h)
        want = max(want, float(t.abs().max()))
        bound = max(bound, 2 * float(v.abs().max()) * float(np.abs(c).sum()) / h)
    assert abs(float(out.item()) - want) <= 7 * 2.0 ** -24 * bound
