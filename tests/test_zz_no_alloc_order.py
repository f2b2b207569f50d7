"""bm3d_basic_noalloc from several streams and host threads: its calls share one device array, and run one after the
other whatever streams they come from.  Also a call captured into a CUDA graph."""
import ctypes as C
import threading

import numpy as np
import pytest

from bm3d_b200 import _capi, synth

pytestmark = pytest.mark.gpu

TOL = 1e-4       # float outputs, as in the other parity tests


class Call:
    def __init__(self, seed, h, w, profile, sigma):
        import torch
        nz, _ = synth.gray_frames(seed, 1, h, w, sigma)
        self.src = torch.from_numpy(nz[0, 0]).cuda()
        self.dst = torch.empty_like(self.src)
        self.args = (w, h, w * 4, profile, sigma)
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        self.enqueue()
        torch.cuda.synchronize()
        self.expected = self.dst.cpu().numpy()

    def enqueue(self, stream=None):
        w, h, stride, profile, sigma = self.args
        r = _capi.lib().bm3d_basic_noalloc(C.c_void_p(self.src.data_ptr()), C.c_void_p(self.dst.data_ptr()), w, h, stride,
                                           profile, sigma, C.c_void_p((stream or self.stream).cuda_stream))
        assert r == _capi.BM3D_OK, _capi.last_error()

    def check(self):
        assert float(np.abs(self.dst.cpu().numpy() - self.expected).max()) <= TOL


def calls():
    return [Call(41, 540, 960, b"np", 10.0), Call(42, 97, 131, b"lc", 25.0), Call(43, 288, 352, b"fast", 15.0)]


def test_streams():
    import torch
    cs = calls()
    for _ in range(8):
        for c in cs:
            c.dst.zero_()
        torch.cuda.synchronize()
        for c in cs:
            c.enqueue()
        torch.cuda.synchronize()
        for c in cs:
            c.check()


def test_threads():
    import torch
    cs = calls()
    errors = []

    def work(c):
        try:
            for _ in range(20):
                c.enqueue()
                c.stream.synchronize()
                c.check()
        except BaseException as e:  # noqa: BLE001 -- re-raised on the main thread
            errors.append(e)

    ts = [threading.Thread(target=work, args=(c,)) for c in cs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]
    torch.cuda.synchronize()


def test_graph():
    import torch
    a, b, _ = calls()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.enqueue(torch.cuda.current_stream())
    for _ in range(2):
        a.dst.zero_()
        g.replay()
        torch.cuda.synchronize()
        a.check()
        b.enqueue()
        torch.cuda.synchronize()
        b.check()
