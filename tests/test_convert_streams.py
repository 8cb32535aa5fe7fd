"""dense_to_bcsr on a stream of the caller's: its workspace and results come from
the current stream's memory pool, so whatever is still queued on the current
stream may use that memory. The order of waits and launches, with a recording
library in place of the real one. No GPU needed."""
import torch

import matrixmultiplicationcuda_gb300 as m
from matrixmultiplicationcuda_gb300 import bcsr


class Stream:
    def __init__(self, log, handle):
        self.log, self.cuda_stream = log, handle

    def wait_stream(self, other):
        self.log.append("wait")


class Library:
    def __init__(self, log):
        self.log = log

    def spmm_dense_to_bcsr_mask_words(self, M, K, bR, bC):
        return 4

    def spmm_dense_to_bcsr_count_masks(self, A, M, K, lda, bR, bC, rp, masks, nnzb, s):
        nnzb._obj.value = 3
        self.log.append("count")
        return 0

    def spmm_dense_to_bcsr_fill_masks(self, *args):
        self.log.append("fill")
        return 0


def convert(monkeypatch, use_current):
    log, recorded = [], []
    stream, current = Stream(log, 1), Stream(log, 2)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda handle: stream)
    monkeypatch.setattr(bcsr, "lib", lambda: Library(log))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: current)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: recorded.append(t.numel()))
    A = torch.zeros(32, 64, dtype=torch.float16)
    monkeypatch.setattr(bcsr, "stream_handle", lambda s=None: 0)
    m.dense_to_bcsr(A, 16, 16, stream=current if use_current else stream)
    return log, recorded


def test_another_stream_waits_for_the_pool_it_takes_memory_from(monkeypatch):
    log, recorded = convert(monkeypatch, use_current=False)
    assert log == ["wait", "count", "wait", "fill"]
    assert sorted(recorded) == [3, 3, 4, 768]   # row_ptr, col_idx, masks, vals


def test_the_current_stream_waits_for_nothing(monkeypatch):
    log, recorded = convert(monkeypatch, use_current=True)
    assert log == ["count", "fill"] and not recorded
