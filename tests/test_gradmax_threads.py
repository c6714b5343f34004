"""qp3d_gradmax_noalloc from several host threads at once (GPU), each on its own
stream with grids of its own (other numbers of CTAs, both kernels): every call
delivers the maximum that the same call delivers alone, with more threads than
the device has scratch entries, and so does a call after them."""
import threading

import numpy as np
import pytest

import qp3d

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GRIDS = [(11, 11, 11), (40, 50, 30), (75, 133, 29), (130, 64, 90), (300, 300, 290)]


class _Call:
    def __init__(self, i):
        self.nx, self.ny, self.nz = GRIDS[i % len(GRIDS)]
        self.ldy = (self.ny + 31) // 32 * 32
        g = torch.Generator(device="cuda").manual_seed(i)
        self.u = torch.randn((self.nz, self.nx, self.ldy), generator=g, device="cuda")
        self.u *= 1.0 + 0.1 * i
        self.out = torch.zeros(1, device="cuda")
        self.c = np.zeros(36, np.float32)
        self.c[31:36] = (0.833, -0.2381, 0.059, -0.0099, 0.00079)
        self.stream = torch.cuda.Stream()

    def __call__(self):
        rc = qp3d.load().qp3d_gradmax_noalloc(
            self.u.data_ptr(), self.nx, self.ny, self.nz, self.ldy, 10.0, 10.0, 10.0,
            self.c.ctypes.data, self.out.data_ptr(), self.stream.cuda_stream, None, 0)
        return rc

    def value(self):
        with torch.cuda.stream(self.stream):
            return float(self.out.item())


@pytest.mark.parametrize("threads,rounds", [(8, 40), (40, 10)])
def test_calls_at_the_same_time(threads, rounds):
    calls = [_Call(i) for i in range(threads)]
    torch.cuda.synchronize()
    want = []
    for c in calls:
        assert c() == 0
        want.append(c.value())
    assert min(want) > 0 and len(set(want)) == threads
    wrong, start = [], threading.Barrier(threads)

    def work(i):
        start.wait()
        for r in range(rounds):
            if calls[i]() != 0 or calls[i].value() != want[i]:
                wrong.append((i, r))

    th = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not wrong
    for c, w in zip(calls, want):
        c.out.fill_(-1.0)
        torch.cuda.synchronize()
        assert c() == 0 and c.value() == w
