"""A chain of mat-vecs of few tokens, each launched before the one ahead of it has ended: two buffers written in turn, so that a kernel that
reads early meets old numbers and one that writes early destroys what is still read.  The same bits with a synchronisation behind each, without
one, and replayed as a graph."""
import ctypes as C

import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, release, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


@pytest.mark.parametrize("dt,W,T", [(BF16, 2048, 1), (BF16, 200, 8), (BF16, 129, 3), (F32, 512, 1), (F32, 37, 5)])
def test_chain(gpu, dt, W, T):
    r = np.random.default_rng(W)
    lib, links = gpu.cuda_lib(), 12
    w, _ = as_dt(dt, r.standard_normal((links, W, W)) * (1.2 / W) ** 0.5)
    ws = [dev(gpu, as_dt(dt, w[i])[1]) for i in range(links)]
    x0 = as_dt(dt, r.standard_normal((T, W)))[1]
    bufs = [dev(gpu, x0), zeros(gpu, x0.nbytes)]

    def chain(sync):
        for i in range(links):
            gpu.check(lib.ggb_op_linear_act(dt, ws[i].ptr, W, W, bufs[i % 2].ptr, W, T, 4, bufs[(i + 1) % 2].ptr), "linear_act")
            if sync:
                gpu.sync()

    def start():
        bufs[0].upload(x0)
        gpu.sync()

    start()
    chain(True)
    want = bufs[0].download(x0.dtype)
    assert want.any()
    for _ in range(20):
        start()
        chain(False)
        assert (bufs[0].download(x0.dtype) == want).all()
    start()
    gpu.check(lib.ggb_capture_begin(), "capture_begin")
    chain(False)
    g = C.c_void_p()
    gpu.check(lib.ggb_capture_end(C.byref(g)), "capture_end")
    for _ in range(20):
        start()
        gpu.check(lib.ggb_graph_launch(g), "graph_launch")
        assert (bufs[0].download(x0.dtype) == want).all()
    gpu.check(lib.ggb_graph_free(g), "graph_free")
