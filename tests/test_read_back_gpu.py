"""Copies to the host: through the staging buffer and past it, into pages that are not there yet, off their boundaries."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from inferi_b200.ops import Backend

pytestmark = pytest.mark.gpu
LEAST, MOST, STAGED = 16384, 1 << 20, 640 << 10   # (beyond STAGED bytes a copy goes past the staging buffer)


def d2h(b, dst_ptr, src, nbytes, stream=None):
    assert b.lib.ib_memcpy_d2h(b.handle, stream, dst_ptr, src.data_ptr(), nbytes) == 0


@pytest.mark.parametrize("nbytes", [4, LEAST - 4, LEAST, LEAST + 4, 513024, MOST - 4, MOST, MOST + 4, 5 * MOST, 262140, 262144, 393220, STAGED - 4, STAGED, STAGED + 4])
@pytest.mark.parametrize("offset", [0, 4, 4092])
def test_bytes_arrive(backend, nbytes, offset):
    src = torch.randint(-2**31, 2**31 - 1, (nbytes // 4,), dtype=torch.int32, device="cuda")
    for make in (lambda n: np.empty(n, np.uint8), lambda n: torch.empty(n, dtype=torch.uint8).pin_memory().numpy()):
        out = make(nbytes + 2 * 4096)
        out[:offset], out[offset + nbytes:] = 7, 9
        d2h(backend, out.ctypes.data + offset, src, nbytes)
        torch.cuda.synchronize()
        assert np.array_equal(out[offset:offset + nbytes].view(np.int32), src.cpu().numpy())
        assert (out[:offset] == 7).all() and (out[offset + nbytes:] == 9).all()


def test_a_copy_follows_its_stream(backend):
    """Into ordinary memory the copy is complete when the call returns, behind what the stream holds."""
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        x = torch.zeros(100000, device="cuda")
        for _ in range(50):
            x += torch.matmul(torch.ones(100000, 8, device="cuda"), torch.full((8,), 0.125, device="cuda"))
    out = np.empty(100000, np.float32)
    d2h(backend, out.ctypes.data, x, out.nbytes, s.cuda_stream)
    assert (out == 50.0).all()


def test_threads_share_one_context():
    """A thread that finds the staging buffer taken copies past it."""
    b = Backend(0)
    wrong = []

    def work(k):
        src = torch.full((120000,), float(k), device="cuda")
        torch.cuda.synchronize()
        for _ in range(60):
            out = np.empty(120000, np.float32)
            d2h(b, out.ctypes.data, src, out.nbytes)
            torch.cuda.synchronize()
            if not (out == k).all():
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(1, 5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    b.close()
    assert not wrong


@pytest.mark.parametrize("threaded", [False, True])
def test_a_copy_beside_a_capture(threaded):
    """A context's first copy, while another stream of the process is being captured: it arrives, and the capture goes on."""
    b = Backend(0)
    src, x = torch.arange(130000, dtype=torch.float32, device="cuda"), torch.zeros(8, device="cuda")
    out, other, graph = np.zeros(130000, np.float32), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()

    def copy():
        d2h(b, out.ctypes.data, src, out.nbytes, other.cuda_stream)

    with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="global"):
        x += 1
        if threaded:
            t = threading.Thread(target=copy)
            t.start()
            t.join()
        else:
            copy()
        x += 1
    assert np.array_equal(out, src.cpu().numpy())
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()
    b.close()
