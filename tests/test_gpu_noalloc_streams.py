"""The allocation-free transpose shares one scratch array: calls on several streams, from several threads
and from a replayed graph, enqueued with nothing between them that waits."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

from cuda_als_gb300._lib import CsrView, lib
from test_gpu_index_edges import _csr

pytestmark = pytest.mark.gpu

# one, two and three passes; counters and words of very different sizes
SHAPES = [(7139, 16458, 369125), (300, 200, 40960), (5000, 70000, 200000), (60000, 300, 590000)]


class _State:
    def __init__(self, torch, k):
        self.m, self.n, self.nnz = SHAPES[k]
        row, ptr, col, val = _csr(np.random.default_rng(k), self.m, self.n, self.nnz)
        order = np.argsort(col, kind="stable")
        self.want = (np.concatenate([[0], np.bincount(col, minlength=self.n).cumsum()]), row[order], val[order])
        up = lambda a, t: torch.from_numpy(a.astype(t)).cuda()  # noqa: E731
        self.ins = up(ptr, np.int32), up(col, np.int32), up(val, np.float32)
        self.outs = (torch.zeros(self.n + 1, dtype=torch.int32, device="cuda"),
                     torch.zeros(self.nnz, dtype=torch.int32, device="cuda"),
                     torch.zeros(self.nnz, dtype=torch.float32, device="cuda"))
        self.stream = torch.cuda.Stream()

    def call(self, stream=None):
        view = CsrView(self.m, self.n, self.nnz, *[C.c_void_p(t.data_ptr()) for t in self.ins])
        st = (stream or self.stream).cuda_stream
        return lib().als_csr_to_csc_device_noalloc(C.byref(view), *[C.c_void_p(t.data_ptr()) for t in self.outs],
                                                   C.c_void_p(st))

    def check(self):
        for got, want in zip(self.outs, self.want):
            assert np.array_equal(got.cpu().numpy(), want)
            got.zero_()


def _states(torch):
    states = [_State(torch, k) for k in range(len(SHAPES))]
    torch.cuda.synchronize()
    return states


def test_calls_on_several_streams():
    torch = pytest.importorskip("torch")
    states = _states(torch)
    for _ in range(40):
        for s in states:
            assert s.call() == 0
    torch.cuda.synchronize()
    for s in states:
        s.check()


def test_calls_from_several_threads():
    torch = pytest.importorskip("torch")
    states = _states(torch)
    status = []

    def work(s):
        torch.cuda.set_device(0)
        status.extend(s.call() for _ in range(30))

    threads = [threading.Thread(target=work, args=(s,)) for s in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [0] * (30 * len(states))
    for s in states:
        s.check()


def test_a_captured_call():
    torch = pytest.importorskip("torch")
    states = _states(torch)
    for s in states:  # set up, and loaded
        assert s.call() == 0
    torch.cuda.synchronize()
    for s in states:
        s.check()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            assert s.call(torch.cuda.current_stream()) == 0
        for _ in range(2):
            g.replay()
            torch.cuda.synchronize()
            s.check()
            torch.cuda.synchronize()
