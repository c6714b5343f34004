"""qp3d_gradmax_noalloc as the first CUDA call of a host thread (GPU): the
thread has no current context yet, which the driver's tensor-map encoding
needs."""
import ctypes
import threading

import numpy as np
import pytest

import qp3d

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [32, 300])    # through L1; from staged planes
def test_first_call_of_a_thread(n):
    u = torch.zeros((n, n, n), device="cuda")
    u[16, 16, 16] = 2.0
    c = np.zeros(36, np.float32)
    c[31] = 0.5
    out = torch.zeros(1, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    err = ctypes.create_string_buffer(256)
    got = []

    def call():
        got.append(qp3d.load().qp3d_gradmax_noalloc(
            u.data_ptr(), n, n, n, n, 1.0, 1.0, 1.0, c.ctypes.data, out.data_ptr(),
            stream.cuda_stream, err, len(err)))

    t = threading.Thread(target=call)
    t.start()
    t.join()
    assert got == [0], err.value
    assert float(out.item()) == 1.0
