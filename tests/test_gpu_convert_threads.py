"""A thread that has converted a matrix ends while another captures a graph: what
the library keeps per thread is given back without disturbing the capture."""
import threading

import pytest

import matrixmultiplicationcuda_gb300 as m

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_thread_ends_during_a_capture(dev):
    A = torch.zeros(64, 64, dtype=torch.float16, device=dev)
    A[3, 40] = 1
    converted, leave, out = threading.Event(), threading.Event(), []

    def work():
        out.append(m.dense_to_bcsr(A)[1])
        converted.set()
        leave.wait()

    x = torch.zeros(4, device=dev)
    x.add_(1)
    t = threading.Thread(target=work)
    t.start()
    converted.wait(60)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g):     # (the mode that no thread may disturb)
            x.add_(1)
            leave.set()
            t.join()
            x.add_(1)
    finally:
        leave.set()
    g.replay()
    torch.cuda.synchronize()
    assert x[0].item() == 3 and out[0].tolist() == [2]


def test_threads_keep_their_counts(dev):
    """Conversions at the same time, more at a time than there are pinned words for."""
    start, wrong = threading.Barrier(80), []

    def work(n):
        A = torch.zeros(1024, 64, dtype=torch.float16, device=dev)
        A.view(64, 16, 4, 16)[torch.arange(n) // 4, 0, torch.arange(n) % 4, 5] = 1
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            start.wait()
            for _ in range(10):
                rp, ci, vals = m.dense_to_bcsr(A)
                if ci.numel() != n or vals.numel() != 256 * n or rp[-1].item() != n:
                    wrong.append(n)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(1, 81)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
